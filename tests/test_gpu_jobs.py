"""The served jobs' kernels (gallatin_gb300/csrc/gal_serve.cu) at the sizes where
their shares and buffers end: around the first capacity and its doublings, an
odd tail, shares that differ between CTAs, fewer operations than threads, one
operation more than they divide; every result against the host's, and an arena
too small for the growth."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _job_value(job, j):
    with np.errstate(over="ignore"):
        x = np.uint64(job) * np.uint64(0x9E3779B97F4A7C15) + j * np.uint64(0xBF58476D1CE4E5B9) \
            + np.uint64(0x94D049BB133111EB)
        x ^= x >> np.uint64(31)
        x *= np.uint64(0xD6E8FEB86659FD93)
    return x >> np.uint64(32)


def _queue(job, n, nt):
    """(checksum, mallocs + frees) of a queue job: every enqueued value is dequeued."""
    t = np.arange(nt, dtype=np.uint64)
    mine = n // nt + (t < np.uint64(n % nt))
    length = np.zeros(nt, dtype=np.int64)
    total = enq = 0
    for o in range(int(mine.max())):
        on = o < mine
        h = _job_value(job, (t << np.uint64(40)) ^ np.uint64(o))
        put = on & ((length == 0) | (h % np.uint64(10) < 6))
        total += int(h[put].sum())
        enq += int(put.sum())
        length += put.astype(np.int64) - (on & ~put)
    return total, 2 * enq


def _run(G, g, kind, job, n):
    import torch
    out = torch.zeros(3, dtype=torch.int64, device="cuda")
    hist = torch.zeros(320, dtype=torch.int64, device="cuda")
    rc = G.lib().gal_job_launch(g.handle, kind, job, n, C.c_void_p(out.data_ptr()), C.c_void_p(hist.data_ptr()), None)
    assert rc == 0
    r = out.cpu().numpy().view(np.uint64)
    h = hist.cpu().numpy()
    return int(r[0]), int(r[1]), int(r[2]), int(h[:160].sum()), int(h[160:].sum())


@pytest.fixture(scope="module")
def G():
    import gallatin_gb300
    return gallatin_gb300


@pytest.mark.parametrize("n", [0, 1, 3, 1023, 1024, 1025, 2048, 4095, 4097, 65537, (1 << 20) - 1, (2 << 20) + 5, (9 << 20) + 3])
def test_vector_jobs(G, n):
    g = G.Gallatin.generate_on_device(4 << 30, 42, zero_arena=0)
    try:
        ctas = G.lib().gal_job_ctas(0, n)
        shares = [n * (b + 1) // ctas - n * b // ctas for b in range(ctas)]
        ops = sum(2 + 2 * max(0, int(np.ceil(np.log2(max(m, 1) / 1024)))) for m in shares)
        want = int(_job_value(11, np.arange(n, dtype=np.uint64)).sum())
        total, done, failed, mallocs, frees = _run(G, g, 0, 11, n)
        assert (total, done, failed) == (want, ops, 0)
        assert mallocs == frees == ops // 2
        assert g.error_word() == 0
    finally:
        g.close()


@pytest.mark.parametrize("n", [0, 1, 1000, 1024, 1025, 20000, (1 << 18) + 1, (3 << 18) - 7])
@pytest.mark.parametrize("cfg", [dict(), dict(min_size=16, max_size=16), dict(spare_blocks=1, team_width=8)],
                         ids=["default", "one-class", "spares"])
def test_queue_jobs(G, n, cfg):
    g = G.Gallatin.generate_on_device(4 << 30, 42, zero_arena=0, **cfg)
    try:
        ctas = G.lib().gal_job_ctas(1, n)
        for job in (5, 77):
            total, done, failed, mallocs, frees = _run(G, g, 1, job, n)
            assert (total, done) == _queue(job, n, ctas * 1024) and failed == 0
            assert mallocs == frees == done // 2
        assert g.error_word() == 0, g.error_info()
        sv = g.export()
        assert (sv.free_counters < 4096).all()
    finally:
        g.close()


def test_vector_job_that_cannot_grow(G):
    g = G.Gallatin.generate_on_device(512 << 20, 42, zero_arena=0)
    try:
        total, done, failed, mallocs, frees = _run(G, g, 0, 3, 200 << 20)   # 8 shares of 100 MiB
        assert total == 0 or failed < 8
        assert failed > 0 and mallocs - frees == failed and done == mallocs + frees
        assert _run(G, g, 0, 3, 5000)[2] == 0
    finally:
        g.close()
