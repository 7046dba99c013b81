"""Block requests of one class that arrive together: the class lock, the
segments gathered along for the threads that wait for it, the threads that
lose a segment to one another, and the class's last blocks taken while others
come home.  Classes of one, a few and many blocks per segment, in trees of one
to three layers, lowest-id and hashed segment choice, ahead and on demand."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TREE_FIELDS = ["seg_tree_words", "sub_tree_words", "tree_ids", "slots", "free_counters"]
GIB = 1 << 30


@pytest.mark.parametrize("cls", [2, 4, 6, 8])
@pytest.mark.parametrize("nbytes,cfg", [
    (1008 << 20, dict()),                                          # 63 segments: one layer
    (8 * GIB, dict(gather_unlocked_below=0)),                      # every class behind its lock
    (16 * GIB, dict(gather_unlocked_below=0, subtree_policy=1, gather_ahead=0)),
    (80 * GIB, dict(spare_blocks=1)),                              # 5,120 segments: deep trees
], ids=["one-layer", "locked", "lowest", "deep"])
def test_whole_blocks_requested_together(nbytes, cfg, cls):
    """Whole blocks of one class from every thread, half of them freed and asked
    for again three times over; then everything freed and trimmed."""
    import torch
    import gallatin_gb300 as G
    block = (16 << cls) * 4096
    n = min(2048, int(nbytes * 0.3) // block)
    g = G.Gallatin.generate_on_device(nbytes, 42, zero_arena=0, **cfg)
    try:
        fresh = g.export()
        sizes = torch.full((n,), block, dtype=torch.int64, device="cuda")
        ptrs = torch.zeros(n, dtype=torch.int64, device="cuda")
        g.malloc_per_thread(sizes, ptrs)
        rng = np.random.default_rng(cls)
        for _ in range(3):
            some = torch.from_numpy(rng.permutation(n)[: n // 2].copy()).cuda()
            g.free_per_thread(ptrs[some].contiguous())
            again = torch.zeros(len(some), dtype=torch.int64, device="cuda")
            g.malloc_per_thread(sizes[: len(some)], again)
            ptrs[some] = again
            off = np.sort(ptrs.cpu().numpy() - g.arena_base)
            assert off[0] >= 0 and off[-1] + block <= g.arena_bytes
            assert (off % block == 0).all() and (np.diff(off) >= block).all()
        g.free_per_thread(ptrs)
        torch.cuda.synchronize()
        assert g.error_word() == 0, g.error_info()
        g.trim()
        assert g.error_word() == 0, g.error_info()
        assert g.export().diff(fresh, fields=TREE_FIELDS) == []
    finally:
        g.close()


def test_runs_requested_together():
    """Runs of 2-64 segments from every thread at once, more than one word of
    the segment tree holds, with whole blocks taken meanwhile."""
    import torch
    import gallatin_gb300 as G
    seg = 16 << 20
    rng = np.random.default_rng(1)
    counts = np.concatenate([rng.integers(2, 17, 120), [64, 33, 65]])
    sizes = np.concatenate([counts * seg, np.full(200, 1 << 20)])
    rng.shuffle(sizes)
    g = G.Gallatin.generate_on_device(40 * GIB, 42, zero_arena=0)
    try:
        fresh = g.export()
        d = torch.from_numpy(sizes).cuda()
        for _ in range(3):
            p = torch.zeros(len(sizes), dtype=torch.int64, device="cuda")
            g.malloc_per_thread(d, p)
            off = p.cpu().numpy() - g.arena_base
            assert (off >= 0).all()
            order = np.argsort(off)
            assert (off[order][:-1] + sizes[order][:-1] <= off[order][1:]).all()
            assert (off[sizes > seg] % seg == 0).all()
            g.free_per_thread(p)
            torch.cuda.synchronize()
            assert g.error_word() == 0, g.error_info()
        assert g.stats().multi_segment_allocs == 0
        g.trim()
        assert g.export().diff(fresh, fields=TREE_FIELDS) == []
    finally:
        g.close()
