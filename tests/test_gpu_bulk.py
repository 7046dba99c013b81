"""The batched malloc's chunked kernel (gallatin_gb300/csrc/gal_bulk.cuh) at the
sizes where it can go wrong: the shortest list it serves and the one before it,
lists that end inside a chunk for every chunk size, multi-slice requests (which
may straddle two block runs), requests of the other tiers among them, empty and
smallest requests, calloc mode, few and many size classes, an arena that runs
out.  Every allocation is disjoint from the others and aligned to its class,
and once all are freed a trim leaves the trees of a fresh allocator."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TREE_FIELDS = ["seg_tree_words", "sub_tree_words", "tree_ids", "slots", "free_counters"]
GIB = 1 << 30
TUNED = dict(pinned_slots_first=0, pinned_slots_min=0, gather_unlocked_below=16, bytes_per_segment=64 << 20,
             spare_blocks=1)


@pytest.fixture(scope="module")
def G():
    import gallatin_gb300
    return gallatin_gb300


def _occupied(sizes, cfg):
    """Bytes held and alignment of each request (slices, runs of slices, blocks, segments)."""
    mn, mx, seg = cfg.get("min_size", 16), cfg.get("max_size", 4096), cfg.get("bytes_per_segment", 16 << 20)
    s = np.maximum(sizes, 1).astype(np.int64)
    up = 1 << np.ceil(np.log2(s)).astype(np.int64)
    held = np.maximum(up, mn)
    align = np.minimum(held, mx)                       # runs of slices: one slice
    block = up >= mn * 4096
    block &= up > mx
    align[block] = held[block]
    segs = up > seg
    held[segs] = -(-s[segs] // seg) * seg
    align[segs] = seg
    return held, align


def _check(G, torch, sizes, nbytes, rounds=2, may_fail=False, **cfg):
    g = G.Gallatin.generate_on_device(nbytes, 42, **dict(dict(zero_arena=0), **cfg))
    try:
        fresh = g.export()
        d_sizes = torch.from_numpy(sizes.astype(np.int64)).cuda()
        held, align = _occupied(sizes, cfg)
        for _ in range(rounds):
            d_ptrs = torch.full((len(sizes),), -1, dtype=torch.int64, device="cuda")
            g.malloc_batched(d_sizes, d_ptrs)
            torch.cuda.synchronize()
            off = d_ptrs.cpu().numpy() - g.arena_base
            ok = off != -g.arena_base
            assert ok.all() or may_fail
            assert ok.any()
            assert (off[ok] >= 0).all() and (off[ok] + held[ok] <= g.arena_bytes).all()
            assert (off[ok] % align[ok] == 0).all()
            order = np.argsort(off[ok])
            o, h = off[ok][order], held[ok][order]
            assert (o[:-1] + h[:-1] <= o[1:]).all()
            assert g.error_word() == 0, g.error_info()
            if cfg.get("zero_fill"):
                _scribble(torch, g, d_ptrs, sizes)
            g.free_batched(d_ptrs)
            torch.cuda.synchronize()
        g.trim()
        assert g.error_word() == 0, g.error_info()
        assert g.export().diff(fresh, fields=TREE_FIELDS) == []
    finally:
        g.close()


def _scribble(torch, g, ptrs, sizes):
    """The first and last whole words of every request read 0; then they are set."""
    class Words:
        __cuda_array_interface__ = {"shape": (g.arena_bytes // 8,), "typestr": "<i8", "data": (g.arena_base, False),
                                    "version": 2, "strides": None}
    words = torch.as_tensor(Words(), device="cuda")
    at = (ptrs - g.arena_base) >> 3
    end = at + torch.from_numpy(np.maximum(sizes.astype(np.int64) // 8 - 1, 0)).cuda()
    assert int(words[at].abs().max()) == 0 and int(words[end].abs().max()) == 0
    words[at] = -1
    words[end] = -1


@pytest.mark.parametrize("n", [32767, 32768, 32769, 155648 + 1, 311296 + 511, 622592 + 513])
def test_list_lengths_around_the_chunks(G, torch_mod, n):
    rng = np.random.default_rng(n)
    _check(G, torch_mod, np.rint(2.0 ** rng.uniform(0, 12, n)), 8 * GIB)


@pytest.mark.parametrize("n,lo,hi,nbytes,cfg", [
    (40000, 12.0, 15.0, 8 * GIB, {}),                     # runs of slices only
    (200000, 10.0, 13.5, 16 * GIB, TUNED),                # slices and runs of the last class
    (60000, 0.0, 18.0, 16 * GIB, {}),                     # blocks among them
    (33000, 14.9, 15.2, 16 * GIB, {}),                    # 8-slice runs and the smallest blocks
    (300001, 4.0, 15.0, 4 * GIB, dict(min_size=16, max_size=64)),    # three classes, runs of up to 512 slices
    (100000, 4.0, 20.0, 48 * GIB, dict(min_size=128, max_size=16384, bytes_per_segment=64 << 20)),
    (70000, 0.0, 13.0, 4 * GIB, dict(zero_fill=1)),
    (70000, 0.0, 13.0, 16 * GIB, dict(TUNED, zero_fill=1, block_layout=0)),
    (50000, 4.0, 4.0, 2 * GIB, dict(team_width=8)),
], ids=["runs", "tuned-runs", "blocks", "edge-15", "three-classes", "wide", "calloc", "calloc-tuned", "one-size"])
def test_mixes(G, torch_mod, n, lo, hi, nbytes, cfg):
    rng = np.random.default_rng(7)
    sizes = np.rint(2.0 ** rng.uniform(lo, hi, n))
    sizes[:: n // 50] = 0
    _check(G, torch_mod, sizes, nbytes, **cfg)


def test_segments_among_slices(G, torch_mod):
    sizes = np.full(40000, 100)
    sizes[::8000] = 40 << 20
    _check(G, torch_mod, sizes, 4 * GIB)


@pytest.mark.parametrize("size,n", [(4096, 400000), (256, 2300000), (32768, 40000)])
def test_arena_runs_out(G, torch_mod, size, n):
    # one round: a slot that found no block stays empty until the trim
    _check(G, torch_mod, np.full(n, size), 512 << 20, rounds=1, may_fail=True)


@pytest.fixture(scope="module")
def torch_mod():
    import torch
    return torch


@pytest.mark.parametrize("order", ["same", "reversed", "shuffled"])
@pytest.mark.parametrize("n,cfg", [(2047, {}), (2048, TUNED), (2049, {}), (300000, TUNED),
                                   (311297, {}), (700001, TUNED), (257, {}),
                                   (50000, dict(min_size=16, max_size=16, bytes_per_segment=64 << 10))],
                         ids=["2047", "2048", "2049", "two-each", "four-each", "eight-each", "257", "unstaged"])
def test_frees_in_any_order_with_gaps(G, torch_mod, n, cfg, order):
    """Lists with null entries, in the order of the mallocs or not, of classes
    looked up in shared memory or (32,768 segments) not: what is freed comes
    back, what is not stays."""
    torch = torch_mod
    rng = np.random.default_rng(n)
    sizes = np.rint(2.0 ** rng.uniform(0, 4 if "max_size" in cfg else 12.5, n)).astype(np.int64)
    g = G.Gallatin.generate_on_device((2 if "max_size" in cfg else 16) << 30, 42, zero_arena=0, **cfg)
    try:
        fresh = g.export()
        ptrs = torch.zeros(n, dtype=torch.int64, device="cuda")
        g.malloc_batched(torch.from_numpy(sizes).cuda(), ptrs)
        assert bool((ptrs != 0).all())
        at = np.arange(n) if order == "same" else np.arange(n)[::-1].copy() if order == "reversed" else rng.permutation(n)
        lst = ptrs[torch.from_numpy(at).cuda()]
        gap = torch.from_numpy(rng.random(n) < 0.3).cuda()
        first = lst.clone()
        first[gap] = 0
        g.free_batched(first)
        second = lst.clone()
        second[~gap] = 0
        assert g.error_word() == 0, g.error_info()
        counted = torch.zeros(1, dtype=torch.int64, device="cuda")
        for k in (0, 1, min(n, 2048), n // 2):  # the rest, up to counts the device knows
            counted[0] = k
            part = second.clone()
            g.free_batched_n(part, counted)
            second[:k] = 0
        counted[0] = n + 5  # more than the list holds
        g.free_batched_n(second, counted)
        g.trim()
        assert g.error_word() == 0, g.error_info()
        assert g.export().diff(fresh, fields=TREE_FIELDS) == []
    finally:
        g.close()


def test_frees_of_runs_and_of_pointers_that_are_none(G, torch_mod):
    torch = torch_mod
    g = G.Gallatin.generate_on_device(4 << 30, 42, zero_arena=0)
    try:
        sizes = torch.full((4000,), 64, dtype=torch.int64, device="cuda")
        sizes[::1000] = 40 << 20
        ptrs = torch.zeros(4000, dtype=torch.int64, device="cuda")
        g.malloc_per_thread(sizes, ptrs)
        g.free_batched(ptrs)
        assert g.error_word() == 0 and g.stats().multi_segment_allocs == 0
        for bad in (g.arena_base + g.arena_bytes + 64,          # outside
                    g.arena_base + g.arena_bytes - 64):         # in a free segment
            g.free_batched(torch.full((3,), bad, dtype=torch.int64, device="cuda"))
            assert g.error_word() == 0x2
            g.clear_error()
    finally:
        g.close()
