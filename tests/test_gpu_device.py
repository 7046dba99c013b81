"""User kernels that allocate through the device calls (tests/device/device_test.cu)
and single steps of the allocator in an order of the test's choosing."""
import ctypes as C
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIB = os.path.join(os.path.dirname(os.path.abspath(__file__)), "device", "libdevice_test.so")
GIB = 1 << 30


@pytest.fixture(scope="module")
def D():
    import gallatin_gb300
    gallatin_gb300.lib()
    L = C.CDLL(LIB)
    u32, u64, vp = C.c_uint32, C.c_uint64, C.c_void_p
    L.dev_give_back.argtypes = [vp, u32, C.c_int, vp]
    return L


def _bottom(e, d):
    """The lowest words of every class's tree: the segments it lists."""
    per_tree = e.sub_tree_words.reshape(d.num_trees, -1)
    return per_tree[:, per_tree.shape[1] - (d.num_segments + 63) // 64:]


@pytest.mark.parametrize("cls,fresh", [(0, 0), (4, 0), (7, 0), (8, 1)])
def test_reservation_given_back_lists_the_segment_again(D, cls, fresh):
    """A segment whose last block a stale reservation held while a request met it
    is in its class's tree again once the reservation is given back."""
    import torch
    import gallatin_gb300 as G
    out = torch.full((4,), -1, dtype=torch.int64, device="cuda")
    g = G.Gallatin.generate_on_device(2 * GIB, 42, zero_arena=0)
    try:
        fresh_trees = _bottom(g.export(), g.dims())
        assert D.dev_give_back(g.device_state, cls, fresh, out.data_ptr()) == 0
        assert out.tolist() == [1, 0, 0, 1]
        g.trim()
        assert (_bottom(g.export(), g.dims()) == fresh_trees).all()
        assert g.error_word() == 0, g.error_info()
    finally:
        g.close()
