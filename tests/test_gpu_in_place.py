"""Sizes and pointers in one buffer: every pointer takes the place of its size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GIB = 1 << 30


def _mixed(n, seed):
    """Single slices, runs, whole blocks, runs of segments and empty requests."""
    rng = np.random.default_rng(seed)
    sizes = np.rint(2.0 ** rng.uniform(0, 15, n)).astype(np.int64)
    at = rng.permutation(n)
    sizes[at[:40]] = 65536
    sizes[at[40:50]] = 1 << 20
    sizes[at[50:53]] = 3 * (16 << 20)
    sizes[at[53:60]] = 0
    return sizes


@pytest.mark.parametrize("zero_fill", [0, 1])
@pytest.mark.parametrize("n", [500, 40000, 200003, 700001, 1300001])
def test_list_in_place(n, zero_fill):
    """Short lists and chunks of every size, also in calloc mode over an arena of
    ones: every request has its own bytes and, in calloc mode, zeros."""
    import torch
    import gallatin_gb300 as G
    sizes = _mixed(n, n)
    g = G.Gallatin.generate_on_device(16 * GIB, 42, zero_arena=0, zero_fill=zero_fill)
    try:
        class Words:
            __cuda_array_interface__ = {"shape": (g.arena_bytes // 8,), "typestr": "<i8", "data": (g.arena_base, False),
                                        "version": 2, "strides": None}
        words = torch.as_tensor(Words(), device="cuda")
        words.fill_(-1)
        buf = torch.from_numpy(sizes).cuda()
        g.malloc_batched(buf, buf)
        off = buf.cpu().numpy() - g.arena_base
        assert (off >= 0).all() and (off + sizes <= g.arena_bytes).all()
        assert g.error_word() == 0, g.error_info()
        up = np.maximum(sizes, 1)
        order = np.argsort(off)
        assert (off[order][:-1] + np.maximum(up[order][:-1], 16) <= off[order][1:]).all()
        block = sizes == 65536
        assert (off[block] % 65536 == 0).all() and (off[sizes > (16 << 20)] % (16 << 20) == 0).all()
        if zero_fill:   # the first 4 KiB and the last word of each
            d_off, d_len = torch.from_numpy(off).cuda() >> 3, torch.from_numpy(sizes).cuda() >> 3
            for k in range(512):
                m = d_len > k
                if not bool(m.any()):
                    break
                assert int(words[d_off[m] + k].abs().max()) == 0
            last = d_len > 0
            assert int(words[(d_off + d_len - 1)[last]].abs().max()) == 0
        g.free_batched(buf)
        torch.cuda.synchronize()
        assert g.error_word() == 0, g.error_info()
    finally:
        g.close()
