"""BFS passes at the edges of their forms, compared exactly.

The first-vector pull takes 128 destinations per warp, one per lane slot or, when at most 32 are wanted,
packed: against the pull without that pass (bfs_pull_first 0), for groups of 0 to 128 wanted
destinations.  The push appends up to 128 first touches per warp at once and stops when the visit will
sweep: a pushed vertex's parent is the smallest of its frontier sources, whatever the order.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

COUNTS = [0, 1, 2, 31, 32, 33, 64, 127, 128]


def groups(seed):
    """groups of 128 vertices, of which COUNTS[i] have in-edges: 1 to 12 of them, from anywhere"""
    from grazelle import graphgen as gg
    rng = np.random.RandomState(seed)
    V = 128 * len(COUNTS) * 4 + 37
    src, dst = [], []
    for i in range(V // 128):
        for v in 128 * i + rng.permutation(128)[:COUNTS[i % len(COUNTS)]]:
            n = rng.choice([1, 4, 5, 12])
            src += list(rng.randint(0, V, n))
            dst += [v] * n
    src += [0] * 50
    dst += list(rng.randint(0, V, 50))
    e = np.unique(np.stack([dst, src], 1), axis=0)
    return gg.EdgeList(V, e[:, 1].astype(np.uint64), e[:, 0].astype(np.uint64))


@pytest.mark.parametrize("hubs", [0, 16])
@pytest.mark.parametrize("first", [1, 2])
def test_pull_first_densities(first, hubs):
    from grazelle import native
    from grazelle.engine import Graph
    for seed in (1, 2):
        g = groups(seed)
        pull, push = g.pull_order().pairs(), g.push_order().pairs()
        with Graph(0) as A, Graph(0) as B:
            A.tune(bfs_pull_first=first, hubs=hubs)
            B.tune(bfs_pull_first=0)
            for G in (A, B):
                G.load_pairs(g.num_vertices, pull, push)
            for r in (0, int(g.src[5]), g.num_vertices - 1):
                for flags in (native.FORCE_PULL, native.FORCE_PULL | native.FLAG_HOST_LOOP, 0):
                    (pa, la), (pb, lb) = A.bfs(r, flags), B.bfs(r, flags)
                    np.testing.assert_array_equal(la, lb)
                    np.testing.assert_array_equal(pa, pb)
                np.testing.assert_array_equal(la, O.bfs_levels(push, g.num_vertices, r))


@pytest.mark.parametrize("n,mid,fan", [(300, 3, 40), (70000, 300, 300), (70000, 2, 60000), (1000000, 5000, 700)])
def test_push_parents(n, mid, fan):
    """0 -> `mid` vertices -> `fan` random vertices each (many of them shared, in one vector too) -> 0"""
    from grazelle import graphgen as gg, native
    from grazelle.engine import Graph
    rng = np.random.RandomState(n % 1000 + mid)
    m = 1 + np.arange(mid)
    src = np.concatenate([np.zeros(mid, dtype=np.int64), np.repeat(m, fan), np.arange(mid + 1, n)])
    dst = np.concatenate([m, rng.randint(0, n, mid * fan), np.zeros(n - mid - 1, dtype=np.int64)])
    e = np.unique(src * n + dst)
    src, dst = e // n, e % n
    g = gg.EdgeList(n, src.astype(np.uint64), dst.astype(np.uint64))
    with Graph(0) as G:
        G.load_pairs(n, g.pull_order().pairs(), g.push_order().pairs())
        for flags in (native.FORCE_PUSH, native.FORCE_PUSH | native.FLAG_HOST_LOOP):
            par, lv = G.bfs(0, flags)
            tree = lv[src] + 1 == lv[dst]
            tree &= lv[src] >= 0
            ref = np.full(n, n, dtype=np.int64)
            np.minimum.at(ref, dst[tree], src[tree])
            seen = lv > 0
            np.testing.assert_array_equal(par[seen].astype(np.int64), ref[seen])
            assert lv[0] == 0 and (lv[m] == 1).all() and seen.sum() == (ref < n).sum()
        lab = G.connected_components(native.FORCE_PUSH)
        np.testing.assert_array_equal(lab, G.connected_components(native.FORCE_PULL))


@pytest.mark.parametrize("n", [2, 3, 5, 1023, 1026, 300001])
def test_digest(n):
    """four vertices per thread, the last n % 4 by themselves; again after other sums"""
    from grazelle import graphgen as gg
    from grazelle.engine import Graph
    rng = np.random.RandomState(n)
    src, dst = rng.randint(0, n, 2 * n), rng.randint(0, n, 2 * n)
    src[0], dst[0] = 0, n - 1
    g = gg.EdgeList(n, src.astype(np.uint64), dst.astype(np.uint64))
    deg = g.out_degrees().astype(np.int64)
    odd = (np.arange(n, dtype=np.uint64) * np.uint64(0x9E3779B97F4A7C15)) | np.uint64(1)

    def ref(x, reached, degrees):
        h = int(np.sum((x.astype(np.uint64) + np.uint64(1)) * odd, dtype=np.uint64))
        return int(reached.sum()), int(degrees[reached].sum()), h

    with Graph(0) as G:
        G.load_pairs(n, g.pull_order().pairs(), g.push_order().pairs())
        for r in (0, n - 1, 0):
            lv = G.bfs(r)[1]
            for _ in range(2):
                assert G.digest() == ref(np.where(lv < 0, 0xffffffff, lv), lv >= 0, deg)
        lab = G.connected_components()
        assert G.digest() == ref(lab, lab == np.arange(n), 0 * deg)


@pytest.mark.parametrize("first_n", [1, 2, 5])
@pytest.mark.parametrize("hubs", [0, 64])
def test_first_pass_over_sources_in_any_order(first_n, hubs):
    """Lists need only be grouped by destination.  The parent is the largest frontier source of the first
    vector that holds one, wherever in the vector it stands: the early-exit pass, the compacted pull, the
    scan and a restatement of the rule agree."""
    from grazelle import graphgen as gg, native
    from grazelle.engine import Graph
    g = gg.rmat(12, 8, seed=12)
    V, pull = g.num_vertices, g.pull_order()
    o = np.lexsort((np.random.RandomState(2).rand(g.num_edges), pull.dst))
    src, dst = pull.src[o].astype(np.int64), pull.dst[o].astype(np.int64)
    start = np.searchsorted(dst, np.arange(V + 1))
    with Graph(0) as G:
        G.tune(hubs=hubs)
        G.load_pairs(V, gg.EdgeList(V, src.astype(np.uint64), dst.astype(np.uint64)).pairs(), g.push_order().pairs())
        for r in (0, 9):
            found = []
            for form in ({"bfs_pull_first": first_n}, {"bfs_pull_first": 0}, {"bfs_pull_scan": 1}):
                G.tune(bfs_pull_first=first_n, bfs_pull_scan=0).tune(**form)
                found.append(G.bfs(r, native.FORCE_PULL))
            levels = found[0][1]
            rule = np.full(V, -1.0)
            for v in np.flatnonzero(levels > 0):
                s = src[start[v]:start[v + 1]]
                hit = np.flatnonzero(levels[s] == levels[v] - 1)
                first = s[hit[0] // 4 * 4:hit[0] // 4 * 4 + 4]
                rule[v] = first[levels[first] == levels[v] - 1].max()
            for par, lv in found:
                np.testing.assert_array_equal(lv, levels)
                np.testing.assert_array_equal(par, rule)


@pytest.mark.parametrize("V", [(1 << 19) - 1, 1 << 19, (1 << 19) + 8191, 2200007])
def test_cc_push_compaction_in_two_parts(V):
    """From 2^19 vertices on a CC push lists the lowest 1/256 of them first: the labels under forced
    pushes, as one graph and step by step, whichever part a vertex is in."""
    from grazelle import graphgen as gg, native
    from grazelle.engine import Graph
    rng = np.random.RandomState(V & 0xffff)
    a, b = rng.randint(0, V, size=2 * V), rng.randint(0, V, size=2 * V)
    a[:4], b[:4] = [0, 8191, 8192, V - 1], [V - 1, 8192, 16384, V - 2]
    g = gg.EdgeList(V, np.concatenate([a, b]).astype(np.uint64), np.concatenate([b, a]).astype(np.uint64))
    pull = g.pull_order().pairs()
    ref = O.cc_min_labels(pull, V).astype(np.float64)
    with Graph(0) as G:
        G.load_pairs(V, pull, g.push_order().pairs())
        for flags in (native.FORCE_PUSH, native.FORCE_PUSH | native.FLAG_HOST_LOOP, 0):
            np.testing.assert_array_equal(G.connected_components(flags), ref, err_msg="flags %d" % flags)


@pytest.mark.parametrize("V", [2470001, 2540003])
def test_pulls_over_long_lists(V):
    """From 2 tiles of 1024 vectors for each of 1216 blocks on, the pulls over compacted destinations take
    such tiles instead of 256: a random tree, a vector per vertex, with a destination of 5000 vectors among
    them, on either side of that length; vertex 0 reaches everything."""
    from grazelle import graphgen as gg, native
    from grazelle.engine import Graph
    rng = np.random.RandomState(V & 0xffff)
    dst = np.arange(1, V)
    src = (rng.rand(V - 1) * dst).astype(np.int64)
    hub = np.unique(rng.randint(0, V, size=20000))
    hub = hub[hub != 1234567]
    g = gg.EdgeList(V, np.concatenate([src, hub]).astype(np.uint64), np.concatenate([dst, np.full(hub.shape[0], 1234567)]).astype(np.uint64))
    pull, push = g.pull_order().pairs(), g.push_order().pairs()
    with Graph(0) as G:
        G.load_pairs(V, pull, push)
        labels = O.cc_min_labels(pull, V).astype(np.float64)
        for flags in (native.FORCE_PULL, native.FORCE_PULL | native.FLAG_HOST_LOOP):
            np.testing.assert_array_equal(G.connected_components(flags), labels)
        G.tune(bfs_pull_scan=1)
        par, lv = G.bfs(0, native.FORCE_PULL)
        np.testing.assert_array_equal(lv, O.bfs_levels(push, V, 0))
        for form in ({"bfs_pull_scan": 0, "bfs_pull_first": 0}, {"bfs_pull_first": 1}):
            G.tune(**form)
            for flags in (native.FORCE_PULL, native.FORCE_PULL | native.FLAG_HOST_LOOP):
                par2, lv2 = G.bfs(0, flags)
                np.testing.assert_array_equal(par2, par)
                np.testing.assert_array_equal(lv2, lv)
