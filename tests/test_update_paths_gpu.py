"""Updates at the sizes where a vertex or a batch segment passes from a lane
group to a whole CTA, and where a CTA's list of dirty vertices runs over."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _adjacency(g):
    off, dst, _ = g.export_csr()
    src = np.repeat(np.arange(g.n, dtype=np.uint32), np.diff(off.astype(np.int64)))
    return set(zip(src.tolist(), dst.tolist()))


@pytest.mark.parametrize("window", [False, True])
@pytest.mark.parametrize("block,tpv", [(32, 4), (64, 8), (128, 16), (128, 32)])
def test_updates_around_the_cta_threshold(block, tpv, window):
    import gv_b200
    rng = np.random.default_rng(tpv + window)
    line = 128 * tpv  # slots above which a vertex is a CTA's
    deg = [1, block, line - 1, line, line + 1, line + 4 * block + 3, 9000, 2048, 2049]  # 2048: a segment's line
    n = 12_000
    src = np.repeat(np.arange(len(deg), dtype=np.uint32), deg)
    dst = np.concatenate([rng.choice(n - 20, d, replace=False) + 20 for d in deg]).astype(np.uint32)
    cut = rng.random(len(src)) < 0.5
    with gv_b200.GraphVine(n, block_size=block, threads_per_vertex=tpv, directed=True, hbm_budget_bytes=1 << 28) as g:
        g.batch_insert(src[cut], dst[cut])
        drop = rng.random(len(src)) < 0.3  # stored and absent pairs alike
        if window:
            g.batch_run([(src[~cut], dst[~cut], src[drop], dst[drop])], compact=True)
        else:
            g.batch_insert(src[~cut], dst[~cut])  # fills the same vertices further
            g.batch_delete(src[drop], dst[drop])
            g.compaction()
        g.synchronize()
        assert g.check()[0] == 0
        assert g.num_edges() == int((~drop).sum())
        assert _adjacency(g) == set(zip(src[~drop].tolist(), dst[~drop].tolist()))


@pytest.mark.parametrize("n", [1_000, 1_500_000])  # 1,184 CTAs: none, then every CTA, over its 1,024 listed vertices
def test_many_dirty_vertices(n):
    import gv_b200
    u = np.arange(n, dtype=np.uint32)
    v = (u + 1) % n
    with gv_b200.GraphVine(n, block_size=32, threads_per_vertex=32, directed=True, pool_blocks=n + 64,
                           max_batch_pairs=n) as g:
        g.batch_insert(u, v.astype(np.uint32))
        g.batch_delete(u, v.astype(np.uint32))
        g.synchronize()
        assert g.num_edges() == 0
        g.compaction()
        g.synchronize()
        assert g.check()[0] == 0
        assert g.pool_stats()[1] == n + 64  # every block is free again: no vertex was missed
