"""Requests of more segments than the arena has, up to 2^64 - 1 bytes: refused, with
nothing changed (their number of segments does not fit 32 bits)."""
import numpy as np
import pytest

from oracle.oracle import FAIL, Oracle

SEG = 16 << 20
HUGE = [2 * (1 << 30) + 1, 1 << 40, (1 << 56) + 1, (1 << 56) + SEG, 1 << 62, 1 << 63, (1 << 64) - SEG, (1 << 64) - 1]


@pytest.mark.parametrize("size", HUGE)
def test_oracle_refuses(size):
    o = Oracle(2 << 30, 42)
    before = o.export()
    assert o.malloc(size) == FAIL
    assert o.export().diff(before) == []


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 33, 40000], ids=["alone", "short-list", "chunked-list"])
@pytest.mark.parametrize("cfg", [dict(), dict(zero_fill=1)], ids=["malloc", "calloc"])
def test_lists_refuse(n, cfg):
    """Every size above in a list of small requests: null pointers for them, the
    others served, the trees as before once those are free."""
    import torch
    import gallatin_gb300 as G
    g = G.Gallatin.generate_on_device(2 << 30, 42, zero_arena=0, **cfg)
    try:
        fresh = g.export()
        sizes = np.full(n + len(HUGE), 64, dtype=np.uint64)
        at = np.random.default_rng(n).permutation(len(sizes))[: len(HUGE)]
        sizes[at] = HUGE
        d = torch.from_numpy(sizes.view(np.int64)).cuda()
        ptrs = torch.full_like(d, -1)
        g.malloc_batched(d, ptrs)
        got = ptrs.cpu().numpy()
        assert (got[at] == 0).all() and np.count_nonzero(got) == n
        g.free_batched(ptrs)
        torch.cuda.synchronize()
        assert g.error_word() == 0, g.error_info()
        g.trim()
        fields = ["seg_tree_words", "sub_tree_words", "tree_ids", "slots", "free_counters"]
        assert g.export().diff(fresh, fields=fields) == []
    finally:
        g.close()


@pytest.mark.gpu
def test_serial_calls_match_the_oracle():
    """The sizes that a trace can name (below its free bit), alone and in between."""
    import gallatin_gb300 as G
    ops = []
    for size in HUGE[:5]:
        ops += [64, size, 3 * SEG, size, 70000]
    ops = np.array(ops, dtype=np.uint64)
    g = G.Gallatin.generate_on_device(2 << 30, 42, zero_arena=0)
    try:
        offsets, smid = g.replay(ops)
        o = Oracle(2 << 30, 42)
        assert np.array_equal(offsets, o.replay(ops, smid=smid))
        assert (offsets.reshape(-1, 5)[:, [1, 3]] == FAIL).all()
        assert g.export().diff(o.export()) == []
        assert g.error_word() == 0
    finally:
        g.close()
