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


@pytest.mark.parametrize("pairs", [1, 31, 33, 511, 2047, 2048, 2049, 4096, 4097])
@pytest.mark.parametrize("directed,weighted", [(False, False), (True, True)])
@pytest.mark.parametrize("n", [2, 300, 70_001])  # keys of 2, 18 and 34 bits
def test_batches_around_the_one_launch_size(pairs, directed, weighted, n):
    """A batch that one CTA expands, sorts and cuts: repeats (the first weight
    wins), self-loops and, rejected whole, ids out of range (device arrays,
    which the host does not look through)."""
    import gv_b200
    import torch
    rng = np.random.default_rng(pairs + n)
    s, d = rng.integers(0, n, (2, pairs)).astype(np.uint32)
    w = rng.random(pairs).astype(np.float32)
    with gv_b200.GraphVine(n, block_size=32, directed=directed, weighted=weighted, hbm_budget_bytes=1 << 28) as g:
        g.batch_insert(s, d, w if weighted else None)
        g.synchronize()
        want = {}
        for a, b, x in zip(s.tolist(), d.tolist(), w.tolist()):
            if a != b:
                want.setdefault((a, b), x)
                if not directed:
                    want.setdefault((b, a), x)
        off, dst, wt = g.export_csr(with_weights=weighted)
        src = np.repeat(np.arange(n), np.diff(off.astype(np.int64)))
        assert list(zip(src.tolist(), dst.tolist())) == sorted(want)
        if weighted:
            assert np.array_equal(wt, np.array([want[k] for k in sorted(want)], np.float32))
        aff = np.zeros(n, np.uint8)
        for a, b in want:
            aff[a] = aff[b] = 1
        assert np.array_equal(g.affected(), aff)
        bad = torch.from_numpy(s.astype(np.int32)).cuda()
        bad[-1] = n
        with pytest.raises(gv_b200.GvError):
            g.batch_insert(bad, torch.from_numpy(d.astype(np.int32)).cuda(),
                           torch.from_numpy(w).cuda() if weighted else None)
            g.synchronize()
        assert g.num_edges() == len(want) and g.check()[0] == 0
        g.batch_delete(s[::2], d[::2])
        g.compaction()
        g.synchronize()
        gone = {(a, b) for a, b in zip(s[::2].tolist(), d[::2].tolist())}
        gone |= set() if directed else {(b, a) for a, b in gone}
        off, dst, _ = g.export_csr()
        src = np.repeat(np.arange(n), np.diff(off.astype(np.int64)))
        assert list(zip(src.tolist(), dst.tolist())) == sorted(set(want) - gone)


@pytest.mark.parametrize("n", [1, 32, 16383, 16384, 16385, 32767, 32768, 32769, 70_000])
def test_offsets_of_every_scan_size(n):
    """Export offsets come from the exclusive scan: one row, whole and ragged
    tiles of the one-launch scan, and past it."""
    import gv_b200
    deg = np.random.default_rng(n).integers(0, 3, n)
    src = np.repeat(np.arange(n, dtype=np.uint32), deg)
    dst = (src + 1 + np.concatenate([np.arange(k) for k in deg]).astype(np.uint32)) % max(n, 1) if n > 3 else src * 0
    keep = src != dst
    with gv_b200.GraphVine(n, block_size=32, directed=True, hbm_budget_bytes=1 << 27) as g:
        if keep.any():
            g.batch_insert(src[keep], dst[keep].astype(np.uint32))
        g.synchronize()
        off, _, _ = g.export_csr()
    assert np.array_equal(np.diff(off.astype(np.int64)), np.bincount(src[keep], minlength=n))
