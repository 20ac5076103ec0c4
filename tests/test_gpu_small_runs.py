"""Small CC/BFS iterations run many at a time in one cluster: whole runs against the host loop (one
engine kernel chain per iteration) and the oracle.

Parents, levels, engines and iteration counts of BFS are those of single iterations whatever runs
them, and CC labels are unique, so everything is compared exactly.  The graphs put frontiers at the
edges: a path (one vertex per level), stars whose hub fills a list or outgrows it, meshes, power-law
graphs whose frontiers grow past the bound and shrink again, vertices without out-edges, and lists
whose sources do not ascend.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _edges(V, src, dst):
    from grazelle import graphgen as gg
    return gg.EdgeList(V, np.asarray(src, dtype=np.uint64), np.asarray(dst, dtype=np.uint64))


def path(n):
    return _edges(n, np.arange(n - 1), np.arange(1, n))


def star(n):
    """0 -> hub 1 -> every other vertex -> the last one"""
    o = np.arange(2, n - 1)
    return _edges(n, np.concatenate([[0], np.full(o.shape[0], 1), o]), np.concatenate([[1], o, np.full(o.shape[0], n - 1)]))


def mesh(n, seed):
    v = np.arange(n * n)
    r, d = v[v % n != n - 1], v[v + n < n * n]
    a, b = np.concatenate([r, d]), np.concatenate([r + 1, d + n])
    keep = np.random.RandomState(seed).rand(a.shape[0]) > 0.2
    return _edges(n * n, np.concatenate([a[keep], b[keep]]), np.concatenate([b[keep], a[keep]]))


def graphs():
    from grazelle import graphgen as gg
    return {"path2": path(2), "path700": path(700), "star70": star(70), "star9000": star(9000), "star70000": star(70000),
            "mesh40": mesh(40, 3), "mesh150": mesh(150, 4), "rmat11": gg.rmat(11, seed=5), "rmat15": gg.rmat(15, 8, seed=6),
            "rmat15sym": gg.rmat(15, 8, seed=7, symmetric=True), "er40k": gg.erdos_renyi(40000, 3, seed=8)}


@pytest.mark.parametrize("name", list(graphs()))
def test_bfs_equals_the_host_loop(name):
    from grazelle import native, switch
    from grazelle.engine import Graph
    g = graphs()[name]
    V = g.num_vertices
    pull, push = g.pull_order().pairs(), g.push_order().pairs()
    roots = sorted({0, 1, V // 2, V - 1, int(g.src[g.num_edges // 2])})
    with Graph(0) as G:
        G.load_pairs(V, pull, push)
        net = switch.pretrained(0)
        for learned in (False, True):
            G.set_policy(native.POLICY_LEARNED if learned else native.POLICY_THRESHOLD, net if learned else None)
            for flags in (0, native.FORCE_PULL, native.FORCE_PUSH):
                for r in roots:
                    what = "%s learned %s flags %d root %d" % (name, learned, flags, r)
                    par, lv, st = G.bfs(r, flags, stats=True)
                    par2, lv2, st2 = G.bfs(r, flags | native.FLAG_HOST_LOOP, stats=True)
                    np.testing.assert_array_equal(lv, lv2, err_msg=what)
                    np.testing.assert_array_equal(par, par2, err_msg=what)
                    assert (st.iterations, st.pull_iterations, st.push_iterations) == (st2.iterations, st2.pull_iterations, st2.push_iterations), what
        for r in roots:
            np.testing.assert_array_equal(G.bfs(r)[1], O.bfs_levels(push, V, r), err_msg="%s root %d" % (name, r))


@pytest.mark.parametrize("name", list(graphs()))
def test_cc_equals_the_oracle(name):
    from grazelle import native
    from grazelle.engine import Graph
    g = graphs()[name]
    pull, push = g.pull_order().pairs(), g.push_order().pairs()
    ref = O.cc_min_labels(pull, g.num_vertices).astype(np.float64)
    with Graph(0) as G:
        G.load_pairs(g.num_vertices, pull, push)
        for flags in (0, native.FORCE_PUSH, native.FORCE_PULL, 0, native.FORCE_PUSH):
            lab, st = G.connected_components(flags, stats=True)
            np.testing.assert_array_equal(lab, ref, err_msg="%s flags %d" % (name, flags))
            assert st.iterations == st.pull_iterations + st.push_iterations
        G.bfs(0)  # the scratch arrays serve both applications
        np.testing.assert_array_equal(G.connected_components(), ref)


@pytest.mark.parametrize("hubs", [0, 64])
def test_hub_encoded_pull_list(hubs):
    """The pull's parents are looked up in the pull list, hub-encoded or not."""
    from grazelle import graphgen as gg, native
    from grazelle.engine import Graph
    g = gg.rmat(14, 6, seed=9)
    with Graph(0) as G:
        G.tune(hubs=hubs)
        G.load_pairs(g.num_vertices, g.pull_order().pairs(), g.push_order().pairs())
        for r in (0, 77, 5000):
            par, lv = G.bfs(r, native.FORCE_PULL)
            par2, lv2 = G.bfs(r, native.FORCE_PULL | native.FLAG_HOST_LOOP)
            np.testing.assert_array_equal(par, par2)
            np.testing.assert_array_equal(lv, lv2)


@pytest.mark.parametrize("derive", [False, True])
def test_lists_grouped_but_not_ascending(derive):
    """Lists need only be grouped by their shared vertex.  With sources in another order the small pulls
    go to the pull kernels and PageRank is not segmented: the results are those of the host loop and of
    the ascending lists (levels, labels, PageRank props bit for bit)."""
    from grazelle import graphgen as gg, native
    from grazelle.engine import Graph
    g = gg.rmat(13, 8, seed=10)
    V, rng = g.num_vertices, np.random.RandomState(1)
    pull, push = g.pull_order(), g.push_order()
    o = np.lexsort((rng.rand(g.num_edges), pull.dst))
    mixed = gg.EdgeList(V, pull.src[o], pull.dst[o]).pairs()
    with Graph(0) as A, Graph(0) as B:
        A.load_pairs(V, pull.pairs(), push.pairs())
        for G in (A, B):
            G.tune(pr_segment_bits=10)
        if derive:
            B.load_pull_derive_push(V, g.num_edges, mixed.ctypes.data)
        else:
            B.load_pairs(V, mixed, push.pairs())
        for r in (0, 100):
            for flags in (0, native.FORCE_PULL):
                par, lv = B.bfs(r, flags)
                par2, lv2 = B.bfs(r, flags | native.FLAG_HOST_LOOP)
                np.testing.assert_array_equal(par, par2)
                np.testing.assert_array_equal(lv, lv2)
                np.testing.assert_array_equal(lv, A.bfs(r, flags)[1])
        np.testing.assert_array_equal(B.connected_components(), A.connected_components())
        np.testing.assert_array_equal(B.pagerank(5), A.pagerank(5))


def _repeated(V, seed):
    """Edges drawn with replacement from few sources: every list holds runs of the same neighbour, across
    the ends of vectors too.  And the smallest such list, 10 11 12 15 | 15 16 17 18
    into the last vertex, with 15 and 16 behind the vertex before it."""
    rng = np.random.RandomState(seed)
    n = 12 * V
    src, dst = rng.randint(0, V, size=n) // 3 * 3 % V, rng.randint(0, V, size=n)
    first = np.array([0, 1, 2, 5, 5, 6, 7, 8]) + 10
    keep = (src != dst) & (dst != V - 1) & (src != V - 1)
    src = np.concatenate([src[keep], first, np.full(2, V - 2), np.full(3, 4)])
    dst = np.concatenate([dst[keep], np.full(8, V - 1), [15, 16], [V - 2] * 3])
    return _edges(V, src, dst)


@pytest.mark.parametrize("V", [60, 700, 4000])
@pytest.mark.parametrize("hubs", [0, 16])
def test_parents_over_repeated_edges(V, hubs):
    """A repeated in-edge may end one vector and begin the next: the first vector that holds a frontier
    source decides the parent, whatever runs the pull."""
    from grazelle import native, switch
    from grazelle.engine import Graph
    g = _repeated(V, V)
    pull, push = g.pull_order().pairs(), g.push_order().pairs()
    L = O.layout(V, pull, push)
    with Graph(0) as G:
        G.tune(hubs=hubs)
        G.load_pairs(V, pull, push)
        net = switch.pretrained(0)
        for learned in (False, True):
            G.set_policy(native.POLICY_LEARNED if learned else native.POLICY_THRESHOLD, net if learned else None)
            for flags in (0, native.FORCE_PULL, native.FORCE_PUSH):
                for r in (0, 4, V // 2, V - 2):
                    what = "learned %s flags %d root %d" % (learned, flags, r)
                    par, lv = G.bfs(r, flags)
                    par2, lv2 = G.bfs(r, flags | native.FLAG_HOST_LOOP)
                    np.testing.assert_array_equal(lv, lv2, err_msg=what)
                    np.testing.assert_array_equal(par, par2, err_msg=what)
        G.set_policy(native.POLICY_THRESHOLD)
        for flags in (0, native.FORCE_PULL, native.FORCE_PUSH):
            np.testing.assert_array_equal(G.bfs(0, flags)[0], O.bfs(L, flags)[0], err_msg="flags %d" % flags)
        assert G.bfs(V - 2, native.FORCE_PULL)[0][V - 1] == 15  # of the first vector, 10 11 12 15


@pytest.mark.parametrize("sizes", [[512], [513], [508, 509, 512, 516, 517], [520] * 50, [517] * 57, [20000], [8200, 8300, 513, 4, 600], [31000]])
def test_hubs_in_the_starting_frontier(sizes):
    """Vertices of 128 vectors and around it, of many times as many, and as many such as a starting frontier can
    hold, listed by all blocks: CC, whose first frontier is every vertex, and BFS from each hub."""
    from grazelle import native
    from grazelle.engine import Graph
    hubs = np.arange(len(sizes))
    src = np.repeat(hubs, sizes)
    V = len(sizes) + sum(sizes) + 1
    dst = len(sizes) + np.arange(sum(sizes))
    src, dst = np.concatenate([src, dst[::7]]), np.concatenate([dst, np.full(dst[::7].shape[0], V - 1)])
    g = _edges(V, src, dst)
    pull, push = g.pull_order().pairs(), g.push_order().pairs()
    with Graph(0) as G:
        G.load_pairs(V, pull, push)
        for flags in (0, native.FORCE_PUSH):
            np.testing.assert_array_equal(G.connected_components(flags), O.cc_min_labels(pull, V).astype(np.float64))
            for r in sorted({0, len(sizes) // 2, len(sizes) - 1}):
                par, lv = G.bfs(r, flags)
                par2, lv2 = G.bfs(r, flags | native.FLAG_HOST_LOOP)
                np.testing.assert_array_equal(lv, lv2)
                np.testing.assert_array_equal(par, par2)
                np.testing.assert_array_equal(lv, O.bfs_levels(push, V, r))
