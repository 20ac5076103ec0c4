"""Forms that need something the device may not have: without it, calls run as they do where the form was
never chosen, with the same results bit for bit.  GRZ_TUNE_WITHHOLD takes the thing away."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [8, 12])
def test_no_clusters(scale):
    """Without clusters of 16 blocks small PageRank graphs take the two kernels, and small CC/BFS iterations
    the engines' own; in between and afterwards the cluster forms run."""
    from grazelle import graphgen as gg, native
    from grazelle.engine import Graph
    g = gg.rmat(scale, 4, seed=scale)
    V, pull, push = g.num_vertices, g.pull_order().pairs(), g.push_order().pairs()
    L = O.layout(V, pull, push)
    with Graph(0) as G:
        G.load_pairs(V, pull, push)
        found = []
        for withhold in (native.WITHHOLD_CLUSTERS, 0, native.WITHHOLD_CLUSTERS):
            G.tune(withhold=withhold)
            assert G.tuning()["withhold"] == withhold
            before = G.launch_count()
            p = G.pr_init(0.85).pr_iterate(8).props()
            launches = G.launch_count() - before
            found.append([p] + [x for flags in (0, native.FORCE_PULL, native.FORCE_PUSH) for x in G.bfs(0, flags)]
                         + [G.connected_components()])
            assert launches >= 16 if withhold else launches < 10
        for other in found[1:]:
            for a, b in zip(found[0], other):
                np.testing.assert_array_equal(a, b)
        np.testing.assert_array_equal(found[0][1], O.bfs(L)[0])
        np.testing.assert_array_equal(found[0][-1], O.cc(L)[0])
        with pytest.raises(native.GrzError):
            G.tune(withhold=1 << 20)
