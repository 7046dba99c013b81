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
    L.dev_blocks.argtypes = [vp, u64, u32, u32, u32, u32, u64, vp, vp]
    L.dev_churn.argtypes = [vp, u32, u32, u32, u32, u32, C.c_int, u64, vp]
    L.dev_fill.argtypes = [vp, u64, u64, vp]
    L.dev_state_copy.argtypes = [vp, C.c_int, u64, vp]
    L.dev_chunk_claim.argtypes = [vp, u32, u32, u32, u32, vp]
    L.dev_give_back.argtypes = [vp, u32, C.c_int, vp]
    return L


def _bottom(e, d):
    """The lowest words of every class's tree: the segments it lists."""
    per_tree = e.sub_tree_words.reshape(d.num_trees, -1)
    return per_tree[:, per_tree.shape[1] - (d.num_segments + 63) // 64:]


def _as_fresh(g, fresh):
    """After a trim the allocator is as it was when it was made (but for bits of
    the trees' upper layers, which may outlast the items below them)."""
    g.trim()
    assert g.error_word() == 0, g.error_info()
    now = g.export()
    assert now.diff(fresh, fields=["seg_tree_words", "tree_ids", "slots", "free_counters"]) == []
    assert (_bottom(now, g.dims()) == _bottom(fresh, g.dims())).all()


TUNED = dict(pinned_slots_first=0, pinned_slots_min=0, gather_unlocked_below=16, bytes_per_segment=64 << 20,
             spare_blocks=1)


@pytest.mark.parametrize("form", [0, 1, 2], ids=["free", "free_sized", "cached"])
@pytest.mark.parametrize("cfg,hi_bits", [(dict(), 9), (dict(), 17), (dict(team_width=8), 15), (TUNED, 15),
                                         (dict(min_size=128, max_size=16384, bytes_per_segment=64 << 20), 20)],
                         ids=["small", "blocks", "narrow-teams", "tuned", "large-classes"])
def test_mallocs_and_frees_inside_a_kernel(D, cfg, hi_bits, form):
    """A grid that fills the chip, every thread allocating and freeing mixed sizes
    by itself (single slices, runs of slices and whole blocks): each allocation
    is its owner's alone, and once all are free every block is home with its
    free counter at 0."""
    import torch
    import gallatin_gb300 as G
    out = torch.zeros(2, dtype=torch.int64, device="cuda")
    g = G.Gallatin.generate_on_device(48 * GIB, 42, zero_arena=0, **cfg)
    try:
        fresh = g.export()
        ctas = 608 if hi_bits <= 15 else 76
        for seed in range(3):
            assert D.dev_churn(g.device_state, ctas, 256, 24, hi_bits, 3, form, seed << 40, out.data_ptr()) == 0
            assert out.tolist() == [0, 0]
        _as_fresh(g, fresh)
    finally:
        g.close()


@pytest.mark.parametrize("size", [64, 1000, 4096, 9000, 4 << 20])
def test_one_request_per_thread_until_nothing_is_left(D, size):
    """One malloc per thread of a user's kernel, a few thousand more than the arena
    can serve: what is handed out is disjoint and no less than the segments that
    were free at first hold; freed, all of it is home."""
    import torch
    import gallatin_gb300 as G
    held = 1 << (size - 1).bit_length()
    g = G.Gallatin.generate_on_device(1 * GIB, 42, zero_arena=0)
    try:
        fresh = g.export()
        free = int(g.stats().free_segments) * (16 << 20)
        n = int(1.1 * free) // held + 4000
        ptrs = torch.zeros(n, dtype=torch.int64, device="cuda")
        assert D.dev_fill(g.device_state, size, n, ptrs.data_ptr()) == 0
        off = np.sort(ptrs.cpu().numpy())
        off = off[off != 0] - g.arena_base
        assert off[0] >= 0 and off[-1] + held <= g.arena_bytes
        assert (np.diff(off) >= held).all()
        assert free <= len(off) * held and len(off) < n
        assert g.error_word() == 0, g.error_info()
        g.free_per_thread(ptrs)
        torch.cuda.synchronize()
        _as_fresh(g, fresh)
    finally:
        g.close()


@pytest.mark.parametrize("form", range(6), ids=["global", "shared", "local", "constant", "parameter", "grid-constant"])
def test_state_by_value(D, form):
    """Every device call through the state itself and through copies of it."""
    import torch
    import gallatin_gb300 as G
    out = torch.zeros(2, dtype=torch.int64, device="cuda")
    g = G.Gallatin.generate_on_device(4 * GIB, 42, zero_arena=0, spare_blocks=1)
    try:
        fresh = g.export()
        for seed in range(3):
            assert D.dev_state_copy(g.device_state, form, seed << 32, out.data_ptr()) == 0
            assert out.tolist() == [0, 0]
        _as_fresh(g, fresh)
    finally:
        g.close()


@pytest.mark.parametrize("spares", [0, 1])
@pytest.mark.parametrize("slot_left,spare_left,want,left", [
    (0, 4096, 100, 3996),      # a block that nobody replaces
    (6, 96, 200, 3998),        # the next one used up by this claim
    (6, 0, 200, 3902),         # ... or already by others
    (200, 70, 200, 70),        # nothing more wanted
    (50, 4096, 4095, 51),
])
def test_chunk_claim_of_blocks_used_up_by_slow_teams(D, slot_left, spare_left, want, left, spares):
    """A chunk's claim gets all its slices and leaves a block to claim from in the
    slot, whatever slow teams took of the pinned block and of its successor."""
    import torch
    import gallatin_gb300 as G
    out = torch.zeros(4, dtype=torch.int64, device="cuda")
    g = G.Gallatin.generate_on_device(2 * GIB, 42, zero_arena=0, spare_blocks=spares)
    try:
        fresh = g.export()
        assert D.dev_chunk_claim(g.device_state, 2, want, slot_left, spare_left, out.data_ptr()) == 0
        claimed, runs, there, unread = out.tolist()
        assert claimed == want and unread == 0
        assert there == (left if spares else 4096 - (want - slot_left))
        _as_fresh(g, fresh)
    finally:
        g.close()


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


def _unlisted_past_crossing(g):
    """(segment, class) of every owned segment that has blocks to give and is in
    no tree although one of them came home at the ring position that lists a
    segment (the first of which ten times is more than the segment's blocks).
    The first to come home since the segment was last empty is left out: it may
    have taken its position before, and been counted after, the last block went."""
    e, d = g.export(), g.dims()
    listed = _bottom(e, d)
    bad = []
    for seg in range(d.num_segments):
        t, home = int(e.tree_ids[seg]), int(e.active_counts[seg]) + 1
        if t >= d.num_trees or home <= 0 or (int(listed[t, seg // 64]) >> (seg % 64)) & 1:
            continue
        nb, back = d.blocks_per_segment >> t, int(e.queue_free_counters[seg])
        if any(p % nb == nb // 10 + 1 for p in range(max(back - home, 0) + 1, back)):
            bad.append((seg, t))
    return bad


@pytest.mark.parametrize("cls", [3, 4, 5])
def test_returned_blocks_stay_listed(D, cls):
    """Whole blocks of one class (32, 16 and 8 to a segment) asked for and returned
    by many threads at once, its segments emptying and filling all the time: a
    segment that a returned block put back into its class's tree stays there."""
    import torch
    import gallatin_gb300 as G
    size = (16 << cls) * 4096
    failed = torch.zeros(1, dtype=torch.int64, device="cuda")
    g = G.Gallatin.generate_on_device(8 * GIB, 42, zero_arena=0)
    try:
        fresh = g.export()
        kept = torch.zeros(4 * 1024, dtype=torch.int64, device="cuda")
        for seed in range(30):
            assert D.dev_blocks(g.device_state, size, 32, 32, 41, 2, seed, kept.data_ptr(), failed.data_ptr()) == 0
            assert _unlisted_past_crossing(g) == []
        assert int(failed) == 0 and g.error_word() == 0, g.error_info()
        g.free_per_thread(kept)
        torch.cuda.synchronize()
        _as_fresh(g, fresh)
    finally:
        g.close()
