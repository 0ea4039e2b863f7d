"""gv_export_csr over the vertex sizes where its paths meet: warp runs of
vertices without tombstones, packed vertices with tombstones, and hubs that
span several warp shares or, with tombstones, are packed by one CTA."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _neighbours(n, deg, rng):
    src = np.repeat(np.arange(len(deg), dtype=np.uint32), deg)
    dst = np.concatenate([rng.choice(n - len(deg), d, replace=False) + len(deg) for d in deg]).astype(np.uint32)
    return src, dst


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("block", [32, 64, 128])
@pytest.mark.parametrize("deletes", [False, True])
def test_export_matches_the_sets(block, deletes, weighted):
    import gv_b200
    rng = np.random.default_rng(block + deletes)
    # edges of a block, of a step of 32 entries, of a warp share (256 units) and of the CTA threshold (32 blocks)
    deg = [0, 1, 31, 32, 33, 247, 248, 249, 512, block - 1, block, block + 1, 32 * block - 1, 32 * block, 32 * block + 1, 33 * block,
           64 * block, 64 * block + 1, 100 * block + 7, 0, 3] + [2] * 30
    n = 100 * block + 7 + len(deg) + 50
    src, dst = _neighbours(n, deg, rng)
    w = rng.random(len(src)).astype(np.float32) + 0.5
    order = rng.permutation(len(src))
    with gv_b200.GraphVine(n, block_size=block, directed=True, weighted=weighted, hbm_budget_bytes=1 << 28) as g:
        g.batch_insert(src[order], dst[order], w[order] if weighted else None)
        keep = np.ones(len(src), bool)
        if deletes:  # tombstones in some vertices of every size, none in others
            keep = ~((src % 2 == 0) & (rng.random(len(src)) < 0.3))
            g.batch_delete(src[~keep], dst[~keep])
        g.synchronize()
        off, out, wout = g.export_csr(with_weights=weighted)
        assert g.check()[0] == 0
    assert np.array_equal(np.diff(off.astype(np.int64)), np.bincount(src[keep], minlength=n))
    # one batch is stored sorted by destination, and deletes keep the order
    want = np.lexsort((dst[keep], src[keep]))
    assert np.array_equal(out, dst[keep][want])
    if weighted:
        assert np.array_equal(wout, w[keep][want])
