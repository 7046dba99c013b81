"""Hash tables (gallatin_gb300/csrc/gal_tables.cu) in an arena that holds their
nodes and hardly more: nodes that threads hold ready must not be the ones that
others lack."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SEG = 16 << 20


@pytest.mark.parametrize("batched", [False, True])
@pytest.mark.parametrize("pairs,segments", [(200000, 17), (1000000, 20)])
def test_tables_that_just_fit(pairs, segments, batched):
    import gallatin_gb300 as G
    from gallatin_gb300 import tables as T
    g = G.Gallatin.generate_on_device(segments * SEG, 42, zero_arena=0)
    try:
        for seed in range(4):
            d = T.run(g, np.full(16, pairs // 16, dtype=np.uint64), seed=seed, batched=batched)
            assert d["violations"] == 0, d
            assert d["nodes_allocated"] == d["nodes_freed"] + d["spare_nodes_freed"]
            g.trim()
    finally:
        g.close()


@pytest.mark.parametrize("batched", [False, True])
def test_tables_that_do_not_fit(batched):
    """Inserts without a node fail and are counted; everything else goes on, and
    what was allocated is given back."""
    import gallatin_gb300 as G
    from gallatin_gb300 import tables as T
    g = G.Gallatin.generate_on_device(15 * SEG, 42, zero_arena=0)
    try:
        fresh = g.export()
        sizes = np.full(16, 1000000 // 16, dtype=np.uint64)
        d = T.run(g, sizes, seed=3, batched=batched)
        assert d["malloc_failed"] > 0
        coins = sum(int(T.table_coins(T.table_keys(t, int(n), 3)).sum()) for t, n in enumerate(sizes))
        assert d["missing"] > 0 and d["deleted"] < coins
        for k in ("unexpected", "wrong_value", "lock_timeouts", "setup_failed", "error_word"):
            assert d[k] == 0, k
        assert d["nodes_allocated"] == d["nodes_freed"] + d["spare_nodes_freed"]
        g.trim()
        assert g.export().diff(fresh, fields=["seg_tree_words", "tree_ids", "slots", "free_counters"]) == []
    finally:
        g.close()
