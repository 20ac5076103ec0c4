"""The packed PageRank gather (hot sources in shared memory, a contiguous range per warp) against the
general gather of 16-byte props, bit for bit, and the oracle within 1e-12 relative L1.

Both forms sum the same fixed-point values exactly, so nothing may differ: sizes are chosen at the
edges of a thread's four vectors, a warp's 128, a range and a segment.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
PR_TOL = 1e-12


def pagerank(g, iterations=6, **tune):
    from grazelle.engine import Graph
    with Graph(0) as G:
        G.tune(**tune)
        G.load_pairs(g.num_vertices, g.pull_order().pairs())
        return G.pagerank(iterations, damping=0.85)


@pytest.mark.parametrize("V,degree", [(64, 0.02), (65, 1), (129, 2), (1000, 0.3), (1021, 4), (4099, 12), (40009, 31)])
def test_small_and_ragged_lists(V, degree):
    from grazelle import graphgen as gg
    g = gg.erdos_renyi(V, degree, seed=V)
    ref = pagerank(g, pr_props=1)
    np.testing.assert_array_equal(pagerank(g), ref)
    for grid in (1, 2, 151):
        np.testing.assert_array_equal(pagerank(g, pr_grid=grid), ref, err_msg="grid %d" % grid)


@pytest.mark.parametrize("vectors", [1, 3, 4, 5, 31, 32, 33, 127, 128, 129, 255, 257])
def test_one_destination_of_every_length(vectors):
    """A hub of `vectors` in-vectors (the last one partial) between short destinations: cut by a
    thread, a group and ranges."""
    from grazelle import graphgen as gg
    n = 4 * vectors - 1
    V = n + 70
    hub = 35
    src = np.concatenate([np.arange(3), np.setdiff1d(np.arange(V), [hub])[:n], np.arange(5)]).astype(np.uint64)
    dst = np.concatenate([np.full(3, 20), np.full(n, hub), np.full(5, 60)]).astype(np.uint64)
    g = gg.EdgeList(V, src, dst)
    ref = pagerank(g, pr_props=1)
    np.testing.assert_array_equal(pagerank(g), ref)
    np.testing.assert_array_equal(pagerank(g, pr_grid=1), ref)


@pytest.mark.parametrize("seg", [1, 12, 14])
def test_hot_sources(seg):
    """A power-law graph large enough for the hot table (2^21 vectors and more), unsegmented and in
    segments: grids of any size, a reload with the same V, the phase API and CC on the encoded
    segments."""
    import ctypes as C
    from grazelle import graphgen as gg, native
    from grazelle.engine import Graph
    g, h = gg.rmat(18, 44, seed=81), gg.rmat(18, 44, seed=82)
    V = g.num_vertices
    pull, push = g.pull_order().pairs(), g.push_order().pairs()
    ref, ref_h = pagerank(g, pr_props=1, pr_segment_bits=1), pagerank(h, pr_props=1, pr_segment_bits=1)
    L = O.layout(V, pull, push)
    assert O.relative_l1(ref, O.pr_pull(L, 6, damping=0.85)) < PR_TOL
    with Graph(0) as G:
        G.tune(pr_segment_bits=seg)
        G.load_pairs(V, pull, push)
        np.testing.assert_array_equal(G.pagerank(6, damping=0.85), ref)
        for grid in (1, 37, 3000):
            G.tune(pr_grid=grid)
            np.testing.assert_array_equal(G.pagerank(6, damping=0.85), ref, err_msg="grid %d" % grid)
        G.tune(pr_grid=0, pr_persistent=2)
        G.pr_init(0.85).pr_iterate(3)
        G.tune(pr_persistent=0)
        G.pr_iterate(3)  # the hot table is packed again after the persistent form
        np.testing.assert_array_equal(G.props(), ref)
        native.check(G.lib.grz_phases_bind(G.h, native.APP_PAGERANK))
        G.pr_init(0.85).pr_iterate(5)
        info, rb = G.info(), np.zeros(8, dtype=np.uint64)
        G.lib.phase_op_reset_global_accum()
        G.lib.perform_edge_pull_phase_pr(C.c_void_p(info.pull_list_device), info.pull_vectors)
        G.lib.phase_op_write_global_accum_to_buf(C.c_void_p(rb.ctypes.data))
        G.lib.perform_vertex_phase_pr(0, V, C.c_void_p(rb.ctypes.data))
        assert G.lib.grz_phases_last_status() == 0
        np.testing.assert_array_equal(G.props(), ref)
        G.tune(cc_pull_first=0)
        np.testing.assert_array_equal(G.connected_components(), O.cc(L)[0])
        G.load_pairs(V, h.pull_order().pairs(), h.push_order().pairs())
        np.testing.assert_array_equal(G.pagerank(6, damping=0.85), ref_h)


def test_segments_follow_the_hot_choice():
    """Segments built for CC before the hot sources are known are built again, encoded, for PageRank,
    and a CC run captured on the first build reads the second."""
    from grazelle import graphgen as gg
    from grazelle.engine import Graph
    g = gg.rmat(18, 44, seed=83)
    pull, push = g.pull_order().pairs(), g.push_order().pairs()
    with Graph(0) as G:
        G.tune(cc_pull_first=0, cc_segments=2, pr_segment_bits=13)
        G.load_pairs(g.num_vertices, pull, push)
        lab = G.connected_components()
        np.testing.assert_array_equal(lab, O.cc(O.layout(g.num_vertices, pull, push))[0])
        p = G.pagerank(6, damping=0.85)
        np.testing.assert_array_equal(G.connected_components(), lab)
    np.testing.assert_array_equal(p, pagerank(g, pr_props=1, pr_segment_bits=1))


@pytest.mark.parametrize("V,degree", [(1, 0), (2, 1), (15, 2), (16, 3), (33, 0.5), (1000, 4), (4096, 16), (6143, 5), (6144, 13), (6145, 5)])
def test_small_graphs_in_one_launch(V, degree):
    """Graphs small enough for the one-cluster form, and just too large: the same props after any split
    of the iterations, with the two-kernel form in between, and as the general gather."""
    from grazelle import graphgen as gg
    from grazelle.engine import Graph
    if degree and V > 2:
        g = gg.erdos_renyi(V, degree, seed=V)
    else:
        g = gg.EdgeList(V, np.arange(V - 1, dtype=np.uint64)[:degree], np.arange(1, V, dtype=np.uint64)[:degree])
    ref = pagerank(g, 7, pr_props=1)
    with Graph(0) as G:
        G.load_pairs(V, g.pull_order().pairs())
        for split in ((7,), (1, 6), (2, 5), (3, 1, 3)):
            G.pr_init(0.85)
            for n in split:
                G.pr_iterate(n)
            np.testing.assert_array_equal(G.props(), ref, err_msg=str(split))
        G.pr_init(0.85).pr_iterate(3)
        G.tune(pr_persistent=1)
        G.pr_iterate(2)
        G.tune(pr_persistent=0)
        G.pr_iterate(2)
        np.testing.assert_array_equal(G.props(), ref)
        G.load_pairs(V, g.pull_order().pairs())
        np.testing.assert_array_equal(G.pagerank(7, damping=0.85), ref)


@pytest.mark.parametrize("hub_edges", [600, 4000, 6000])
def test_small_graph_with_most_edges_at_few_destinations(hub_edges):
    """Destinations whose vectors outgrow a block's share, and its shared memory."""
    from grazelle import graphgen as gg
    V = 6100
    rng = np.random.RandomState(3)
    src, dst = [], []
    for hub in (5, 6, 7, 8, 9, 4000, 6099):
        s = rng.permutation(V - 1)[:hub_edges]
        src.append(s + (s >= hub))
        dst.append(np.full(hub_edges, hub))
    src.append(np.arange(20))
    dst.append(np.arange(20) + 100)
    g = gg.EdgeList(V, np.concatenate(src).astype(np.uint64), np.concatenate(dst).astype(np.uint64))
    np.testing.assert_array_equal(pagerank(g, 9), pagerank(g, 9, pr_props=1))


@pytest.mark.parametrize("V", [300, 5017, 30011])
def test_negative_constant_at_damping_one(V):
    """At damping 1 the sum of ranks can round above 1, and a vertex without in-edges then gets a negative
    prop, which every form takes without its sign.  Every vertex has 5 out-edges, and for these V the sum of
    V * 5 * ((1 / V) / 5) in doubles is 1 + 2^-52; vertex 0 has no in-edges."""
    from grazelle import graphgen as gg
    from grazelle.engine import Graph
    rng = np.random.RandomState(V)
    g = gg.EdgeList(V, np.repeat(np.arange(V), 5).astype(np.uint64), rng.randint(1, V, size=5 * V).astype(np.uint64))
    found = []
    for tune in ({"pr_props": 1}, {}, {"pr_persistent": 1}, {"pr_segment_bits": 9}):
        with Graph(0) as G:
            G.tune(**tune)
            G.load_pairs(V, g.pull_order().pairs())
            G.pr_init(1.0)
            found.append(np.stack([G.pr_iterate(n).props() for n in (1, 1, 3)]))
    np.testing.assert_allclose(found[0][0, 0], 2.0 ** -52 / V / 5, rtol=1e-12)
    for other in found[1:]:
        np.testing.assert_array_equal(other, found[0])


@pytest.mark.parametrize("V,degree", [(500, 6), (20011, 9)])
@pytest.mark.parametrize("before", [{}, {"pr_props": 1}, {"pr_persistent": 1}, {"pr_persistent": 2}])
def test_segmented_after_unsegmented(V, degree, before):
    """A loaded graph whose iterations become segmented, and back: the segmented gather adds into the
    accumulators, so nothing of the iterations before may be left in them."""
    from grazelle import graphgen as gg
    from grazelle.engine import Graph
    g = gg.erdos_renyi(V, degree, seed=V)
    ref = pagerank(g, 6, pr_props=1)
    with Graph(0) as G:
        G.load_pairs(V, g.pull_order().pairs())
        for seg in (1, 9, 1, 9, 9):
            G.tune(pr_segment_bits=seg, pr_props=0, pr_persistent=0)
            if seg == 1:
                G.tune(**before)
            np.testing.assert_array_equal(G.pagerank(6, damping=0.85), ref, err_msg="segment bits %d" % seg)


@pytest.mark.parametrize("V", [1501, 1777, 4099, 65537, 1000003])
@pytest.mark.parametrize("props", [0, 1])
def test_starting_props_are_the_quotients(V, props):
    """The starting props, one Newton step on the reciprocal, equal the division's (1 / V) / degree bit for
    bit: every degree up to 1500, and one of 300 thousand, on both sides of powers of two in V."""
    from grazelle import graphgen as gg
    from grazelle.engine import Graph
    deg = np.concatenate([np.arange(1500), [300007 if V > 60000 else 1501]])
    src = np.repeat(np.arange(deg.shape[0]), deg)
    g = gg.EdgeList(V, src.astype(np.uint64), np.random.RandomState(V % 1000).randint(0, V, size=src.shape[0]).astype(np.uint64))
    d = np.full(V, V, dtype=np.float64)
    d[1:deg.shape[0]] = deg[1:]
    with Graph(0) as G:
        G.tune(pr_props=props)
        G.load_pairs(V, g.pull_order().pairs())
        np.testing.assert_array_equal(G.pr_init(0.85).props(), 1.0 / V / d)
