"""The parallel boot and trim (gallatin_gb300/csrc/gal_boot.cuh) against the
one-thread order of the oracle: the whole state, word for word, where the two
could part — live allocations in the slots' blocks, trees of one, two and three
layers, one slot per SM with spares, more slots than a tile holds, an arena too
full to boot, segments gathered only on demand."""
import numpy as np
import pytest

from gallatin_gb300._abi import FAIL
from oracle.oracle import PRODUCT_FIXES, Oracle, gen_log_trace, gen_serial_trace

pytestmark = pytest.mark.gpu

MIB, GIB = 1 << 20, 1 << 30
BOOT_ERROR = 0x40


@pytest.fixture(scope="module")
def G():
    import gallatin_gb300
    return gallatin_gb300


@pytest.mark.parametrize("nbytes,slots,seg,spares,ops", [
    (512 * MIB, (128, 4), 16 * MIB, False, lambda: gen_serial_trace(11, 6000, 70, 16, 64)),
    (2 * GIB, (128, 4), 16 * MIB, True, lambda: gen_serial_trace(12, 30000, 58, 16, 256)),
    (64 * GIB, (128, 4), 16 * MIB, False, lambda: gen_log_trace(13, 3000, 60, 4, 22)),
    (16 * GIB, (152, 152), 64 * MIB, True, lambda: gen_log_trace(14, 30000, 60, 4, 16)),
    (16 * GIB, (2500, 7), 16 * MIB, False, lambda: gen_serial_trace(15, 30000, 75, 16, 32)),
], ids=["one-layer", "spares", "three-layers", "slot-per-sm", "many-slots"])
def test_trim_with_live_allocations_matches_oracle(G, nbytes, slots, seg, spares, ops):
    ops = ops()
    g = G.Gallatin.generate_on_device(nbytes, 9, bytes_per_segment=seg, pinned_slots_first=slots[0],
                                      pinned_slots_min=slots[1], spare_blocks=int(spares), zero_arena=0)
    try:
        o = Oracle(nbytes, 9, bytes_per_segment=seg, pinned_first=slots[0], pinned_min=slots[1],
                   fixes=PRODUCT_FIXES, spares=spares)
        assert g.export().diff(o.export()) == []
        out, smid = g.replay(ops)
        np.testing.assert_array_equal(out, o.replay(ops, smid=smid))
        for _ in range(2):  # the second trim retires fresh blocks beside the listed, partly used segments
            g.trim()
            o.trim()
            assert g.export().diff(o.export()) == []
        assert g.error_word() == 0, g.error_info()
    finally:
        g.close()


def test_trim_on_a_full_arena_matches_oracle(G):
    """Live slices in every slot of the first sixteen SMs and 1 MiB blocks up to
    the last: the slots that find no block stay empty and the trim says so."""
    g = G.Gallatin.generate_on_device(1 * GIB, 42)
    try:
        o = Oracle(1 * GIB, 42, fixes=PRODUCT_FIXES)
        sizes = np.array([16 << t for t in range(9)], dtype=np.uint64)
        for sm in range(16):
            g.set_smid_override(sm)
            out, _ = g.replay(sizes)
            assert out.tolist() == [o.malloc(int(x), smid=sm) for x in sizes]
        fill = np.full(1100, 1 * MIB, dtype=np.uint64)
        out, _ = g.replay(fill)
        np.testing.assert_array_equal(out, o.replay(fill, smid=15))
        assert out[-1] == FAIL
        g.trim()
        with pytest.raises(RuntimeError):
            o.trim()
        assert g.error_word() == BOOT_ERROR
        g.clear_error()
        assert g.export().diff(o.export(), fields=["seg_tree_words", "sub_tree_words", "tree_ids", "slots",
                                                   "active_counts", "queue_counters", "queues",
                                                   "free_counters", "malloc_counters"]) == []
    finally:
        g.close()


@pytest.mark.parametrize("slots", [(128, 4), (64, 64)])
def test_boot_without_gathering_ahead_matches_one_thread(G, slots):
    """With every class lock held and no class needing it, one thread boots the
    slots and gathers nothing ahead: the parallel boot of an allocator that
    gathers only on demand leaves the same state."""
    cfg = dict(pinned_slots_first=slots[0], pinned_slots_min=slots[1])
    a = G.Gallatin.generate_on_device(4 * GIB, 42, gather_ahead=0, **cfg)
    b = G.Gallatin.generate_on_device(4 * GIB, 42, boot=False, gather_unlocked_below=1 << 20, **cfg)
    try:
        sv = b.export()
        sv.locks = 0x1FF
        b.load(sv)
        b.trim()
        want, got = b.export(), a.export()
        want.locks = 0
        assert got.diff(want) == []
        assert a.error_word() == 0 and b.error_word() == 0
    finally:
        a.close()
        b.close()


def test_stats_longest_free_run(G):
    """Runs inside a word, across words and ending at the arena's end."""
    g = G.Gallatin.generate_on_device(5 * GIB, 42, boot=False)  # 320 segments: five words
    try:
        rng = np.random.default_rng(3)
        bits = [np.ones(320, bool), np.zeros(320, bool), np.arange(320) >= 100,
                (np.arange(320) % 64 < 60), rng.random(320) < 0.9, rng.random(320) < 0.3]
        fresh = g.export()
        off = len(fresh.seg_tree_words) - 5
        for b in bits:
            sv = g.export()
            sv.seg_tree_words[off:] = np.packbits(b, bitorder="little").view(np.uint64)
            g.load(sv)
            edges = np.flatnonzero(np.diff(np.concatenate([[0], b.astype(np.int8), [0]])))
            longest = int((edges[1::2] - edges[::2]).max()) if b.any() else 0
            st = g.stats()
            assert (st.largest_free_run, st.free_segments) == (longest, int(b.sum()))
    finally:
        g.close()
