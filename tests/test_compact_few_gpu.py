"""Compaction on either side of 2^16 vertices, where a warp takes a vertex or a
lane group does, with every vertex dirty and with a few."""
import numpy as np
import pytest

gv_b200 = pytest.importorskip("gv_b200")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [37, 9_473, 1 << 16, (1 << 16) + 1])
@pytest.mark.parametrize("share", [0.001, 0.5, 1.0])
def test_compaction_packs_every_dirty_vertex(n, share):
    rng = np.random.default_rng(n)
    s, d = rng.integers(0, n, (2, 6 * n)).astype(np.uint32)
    key = np.unique(s.astype(np.uint64) * n + d)
    key = key[key // n != key % n]
    s, d = (key // n).astype(np.uint32), (key % n).astype(np.uint32)
    drop = rng.random(len(s)) < 0.5 if share == 1.0 else rng.random(n)[s] < share
    if share == 1.0:
        drop |= np.r_[True, s[1:] != s[:-1]]  # the first entry of every vertex
    with gv_b200.GraphVine(n, block_size=32, directed=True, hbm_budget_bytes=1 << 28) as g:
        g.batch_insert(s, d)
        g.batch_delete(s[drop], d[drop])
        g.compaction()
        g.synchronize()
        assert g.check()[0] == 0
        off, dst, _ = g.export_csr()
        cap, free = g.pool_stats()
    deg = np.bincount(s[~drop], minlength=n)
    assert np.array_equal(np.diff(off.astype(np.int64)), deg)
    assert np.array_equal(dst, d[~drop])  # one batch is stored in order, and packing keeps it
    assert cap - free == int(((deg + 31) // 32).sum())
