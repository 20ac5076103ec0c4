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


@pytest.mark.parametrize("seg", [1, 14])
def test_no_memory_for_faster_pagerank(seg):
    """Packed props, source segments and the list with hot sources are there to be faster.  Without the
    memory for any of them the graph still runs, also right after a run that had them, and CC over segments
    goes on."""
    from grazelle import graphgen as gg, native
    from grazelle.engine import Graph
    g = gg.rmat(18, 44, seed=81)
    V, pull, push = g.num_vertices, g.pull_order().pairs(), g.push_order().pairs()
    H, S, P = native.WITHHOLD_HOT_LIST, native.WITHHOLD_SEGMENTS, native.WITHHOLD_PACKED
    ref = None
    for first in (P, H, S, H | S, P | H | S, 0):
        with Graph(0) as G:
            G.tune(pr_segment_bits=seg, cc_pull_first=0)
            G.load_pairs(V, pull, push)
            for withhold in (first, 0, first):
                G.tune(withhold=withhold)
                p = G.pagerank(5, damping=0.85)
                ref = p if ref is None else ref
                np.testing.assert_array_equal(p, ref, err_msg="withheld %d after %d" % (withhold, first))
            G.tune(pr_props=1)
            np.testing.assert_array_equal(G.pagerank(5, damping=0.85), ref)
            if first in (H, 0):
                np.testing.assert_array_equal(G.connected_components(), O.cc(O.layout(V, pull, push))[0])
