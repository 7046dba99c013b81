"""The table workload (gallatin_gb300/csrc/gal_tables.cu) where its turns and
its per-bucket kernels can go wrong: one pair, fewer pairs than a warp, empty
tables between others, one bucket under every lane, the most tables a launch
takes, more buckets than one pass of the per-table CTAs covers, keys of other
seeds; nodes per thread and per CTA."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batched", [False, True])
@pytest.mark.parametrize("sizes,dump", [
    ([1], 0), ([31], 0), ([0, 7, 0, 8, 1, 0], 3), ([64] * 4, 1), ([16, 17, 15], 2),
    ([5] * 4096, 4095), ([100000, 3, 257], 0), ([300000], 0),
], ids=["one", "under-a-warp", "empties", "one-bucket-sizes", "edges", "most-tables", "uneven", "long"])
def test_tables_of_every_shape(sizes, dump, batched):
    import gallatin_gb300 as G
    from gallatin_gb300 import tables as T
    sizes = np.array(sizes, dtype=np.uint64)
    g = G.Gallatin.generate_on_device(4 << 30, 42, zero_arena=0)
    try:
        fresh = g.export()
        for seed in (3, 1234567):
            d = T.run(g, sizes, seed=seed, batched=batched, dump_table=dump)
            assert d["violations"] == 0, d
            want = np.sort(T.table_keys(dump, int(sizes[dump]), seed))
            keys, vals = d["dump"]
            order = np.argsort(keys)
            np.testing.assert_array_equal(keys[order], want)
            np.testing.assert_array_equal(vals[order], T.table_values(want))
            n_del = sum(int(T.table_coins(T.table_keys(t, int(n), seed)).sum()) for t, n in enumerate(sizes))
            assert d["deleted"] == n_del and d["inserted"] == int(sizes.sum()) + n_del
            assert d["nodes_allocated"] == d["nodes_freed"] + d["spare_nodes_freed"]
        g.trim()
        assert g.export().diff(fresh, fields=["seg_tree_words", "sub_tree_words", "tree_ids", "slots",
                                              "free_counters"]) == []
    finally:
        g.close()


@pytest.mark.parametrize("batched", [False, True])
def test_table_without_buckets(batched):
    """A table whose bucket array the arena cannot hold has no ops; the tables
    on both sides of it are served whole."""
    import gallatin_gb300 as G
    from gallatin_gb300 import tables as T
    sizes = np.array([500, 1 << 29, 300], dtype=np.uint64)  # 2**27 heads: as large as the arena
    g = G.Gallatin.generate_on_device(1 << 30, 42, zero_arena=0)
    try:
        d = T.run(g, sizes, seed=5, batched=batched)
        n_del = sum(int(T.table_coins(T.table_keys(t, int(sizes[t]), 5)).sum()) for t in (0, 2))
        assert d["setup_failed"] == 1
        for k in ("missing", "unexpected", "wrong_value", "count_mismatch", "malloc_failed", "lock_timeouts"):
            assert d[k] == 0, k
        assert d["deleted"] == n_del and d["inserted"] == 800 + n_del
    finally:
        g.close()
