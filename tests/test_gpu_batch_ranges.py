"""The batch's fused PPR iteration at the edges of its ranges: destinations cut by range starts (a hub
whose in-edges fill many), graphs smaller than a range, batches smaller than one step, seeds without
in-edges, unused instances, and props below 2^-60, which take the longer unpacking.

Against the serial FP64 oracle: relative L1 error below 1e-12 as in the other PPR tests.  Sums are exact
128-bit ones, so the ranks are the same bit for bit whatever the number of blocks.
"""
import numpy as np
import pytest

from oracle import ppr as P

pytestmark = pytest.mark.gpu


def edges(V, src, dst):
    from grazelle import graphgen as gg
    return gg.EdgeList(V, np.asarray(src, dtype=np.uint64), np.asarray(dst, dtype=np.uint64))


def in_star(n):
    """every vertex -> 1, and 1 -> 2: vertex 0 has no in-edges"""
    o = np.setdiff1d(np.arange(n), [1])
    return edges(n, np.concatenate([o, [1]]), np.concatenate([np.ones(n - 1, dtype=int), [2]]))


def hubs(n, fan):
    """hub i -> hub i + 1 and `fan` leaves: a hub's prop is about fan times smaller than the one before"""
    src, dst, V = [], [], n
    for i in range(n):
        if i + 1 < n:
            src.append(i), dst.append(i + 1)
        src += [i] * fan
        dst += range(V, V + fan)
        V += fan
    return edges(V, src, dst)


def rand(n, deg, seed):
    rng = np.random.RandomState(seed)
    return edges(n, rng.randint(0, n, n * deg), rng.randint(0, n, n * deg))


def batch_of(gs):
    from grazelle.batch import Batch
    B = Batch(0)
    for g in gs:
        B.add_graph(g.num_vertices, g.pull_order().pairs())
    B.build()
    return B


CASES = {
    "stars": lambda: [in_star(32), in_star(64), in_star(30001), in_star(1200)],
    "small": lambda: [rand(32 + i, 2, i) for i in range(40)],
    "tiny": lambda: [edges(33, [0, 1], [1, 2])],
    "mixed": lambda: [rand(5000, 9, 1), in_star(40), rand(33, 1, 2), rand(20011, 4, 3), hubs(7, 3000)],
}


@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("k", [1, 8])
def test_ranges(name, k):
    gs = CASES[name]()
    rng = np.random.RandomState(len(name) + k)
    seeds = [[0] + [int(x) for x in rng.randint(0, g.num_vertices, rng.randint(0, k))] for g in gs]
    B = batch_of(gs)
    try:
        first = None
        for blocks in (8, 1, 3):
            B.tune(ppr_blocks=blocks)
            for iterations in (1, 2, 7):
                ranks, _ = B.ppr(seeds, iterations=iterations, damping=0.85)
                if iterations == 7:
                    if first is None:
                        first = [r.copy() for r in ranks]
                    for a, b in zip(first, ranks):
                        np.testing.assert_array_equal(a, b)
                if blocks != 8:
                    continue
                for g, gr, sd in zip(gs, ranks, seeds):
                    pull = g.pull_order().pairs()
                    for i in range(gr.shape[1]):
                        if i >= len(sd):
                            assert not gr[:, i].any()
                            continue
                        ref = P.ppr(g.num_vertices, pull, sd[i], iterations, 0.85)
                        assert np.abs(gr[:, i] - ref).sum() / np.abs(ref).sum() < 1e-12
    finally:
        B.close()


def test_small_props():
    """each rank by itself: sums of at most two terms, so a few roundings, and bits below 2^-124 cut off"""
    g = hubs(7, 3000)
    B = batch_of([g])
    try:
        ranks, _ = B.ppr([[0]], iterations=9, damping=0.85)
    finally:
        B.close()
    ref = P.ppr(g.num_vertices, g.pull_order().pairs(), 0, 9, 0.85)
    assert 0 < ref[ref > 0].min() < 2.0 ** -60
    np.testing.assert_allclose(ranks[0][:, 0], ref, rtol=1e-12, atol=9 * 2.0 ** -124)


@pytest.mark.parametrize("n", [32767, 32768, 32769])
def test_ranges_around_32768_vectors(n):
    """From 2^15 vectors on a warp has at least 32: n vertices of one in-edge each, so n vectors."""
    rng = np.random.RandomState(n)
    g = edges(n, rng.randint(0, n, n), np.arange(n))
    seeds, found = [[0, n - 1, 77]], []
    with batch_of([g]) as B:
        assert B.info()["vectors"] == n
        for blocks in (8, 1):
            B.tune(ppr_blocks=blocks)
            found.append(B.ppr(seeds, 6, 0.85)[0][0])
    np.testing.assert_array_equal(found[0], found[1])
    for i, s in enumerate(seeds[0]):
        ref = P.ppr(n, g.pull_order().pairs(), s, 6, 0.85)
        assert np.abs(found[0][:, i] - ref).sum() < 1e-12 * np.abs(ref).sum()
