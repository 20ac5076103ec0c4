"""Results read into the caller's memory: page-locked or not, at any address."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1, 4, 8, 12])
@pytest.mark.parametrize("pinned", [False, True])
def test_results_at_any_address(offset, pinned):
    """The results are the same bytes wherever they go, and nothing around them is written.  Kernels store
    8-byte values straight into page-locked memory, so an address between two multiples of 8 gets a copy."""
    import torch
    from grazelle import graphgen as gg
    from grazelle.engine import Graph
    g = gg.rmat(10, 8, seed=3)
    V = g.num_vertices
    buf = torch.zeros(8 * V + 64, dtype=torch.uint8, pin_memory=pinned)
    assert buf.data_ptr() % 8 == 0

    def at_offset(read):
        buf.fill_(0xa5)
        assert read(C.c_void_p(buf.data_ptr() + offset)) == 0
        out = buf.numpy()
        assert (out[:offset] == 0xa5).all() and (out[offset + 8 * V:] == 0xa5).all()
        return out[offset:offset + 8 * V].copy()

    with Graph(0) as G:
        G.load_pairs(V, g.pull_order().pairs(), g.push_order().pairs())
        G.pr_init(0.85).pr_iterate(3)
        np.testing.assert_array_equal(at_offset(lambda p: G.lib.grz_read_props(G.h, p, V)).view(np.float64), G.props())
        G.cc_run()
        np.testing.assert_array_equal(at_offset(lambda p: G.lib.grz_read_props(G.h, p, V)).view(np.float64), G.props())
        G.bfs_run(0)
        np.testing.assert_array_equal(at_offset(lambda p: G.lib.grz_read_props(G.h, p, V)).view(np.float64), G.props())
        parents, free = G.props(), torch.cuda.mem_get_info()[0]
        np.testing.assert_array_equal(at_offset(lambda p: G.lib.grz_read_levels(G.h, p, V)).view(np.int64), G.levels())
        assert torch.cuda.mem_get_info()[0] == free  # levels need no memory of their own
        np.testing.assert_array_equal(G.props(), parents)
