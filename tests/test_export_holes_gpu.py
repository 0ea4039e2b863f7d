"""gv_export_csr of vertices that are mostly tombstones: around the rows of 32
slots, the blocks and the eight blocks above which a CTA packs a vertex, with
nothing, the first, the last or every other entry left."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("block", [32, 64, 128])
@pytest.mark.parametrize("left", ["none", "first", "last", "odd", "few"])
def test_mostly_tombstones(block, left, weighted):
    import gv_b200
    rng = np.random.default_rng(block)
    deg = [1, 2, 31, 32, 33, 63, 64, 65, block - 1, block, block + 1, 7 * block, 8 * block - 1, 8 * block, 8 * block + 1,
           9 * block, 40 * block + 5] + [5] * 20 + [8 * block] * 40
    n = 40 * block + 5 + len(deg) + 10
    src = np.repeat(np.arange(len(deg), dtype=np.uint32), deg)
    dst = np.concatenate([np.sort(rng.choice(n - len(deg), d, replace=False)) + len(deg) for d in deg]).astype(np.uint32)
    w = rng.random(len(src)).astype(np.float32) + 0.5
    at = np.concatenate([np.arange(d) for d in deg])
    size = np.repeat(deg, deg)
    keep = {"none": at < 0, "first": at == 0, "last": at == size - 1, "odd": at % 2 == 1,
            "few": rng.random(len(src)) < 0.02}[left]
    keep = keep | (src % 5 == 4)  # and vertices without tombstones in between
    with gv_b200.GraphVine(n, block_size=block, directed=True, weighted=weighted, hbm_budget_bytes=1 << 28) as g:
        g.batch_insert(src, dst, w if weighted else None)
        g.batch_delete(src[~keep], dst[~keep])
        g.synchronize()
        off, out, wout = g.export_csr(with_weights=weighted)
    assert np.array_equal(np.diff(off.astype(np.int64)), np.bincount(src[keep], minlength=n))
    assert np.array_equal(out, dst[keep])  # one batch is stored sorted by destination, and deletes keep the order
    if weighted:
        assert np.array_equal(wout, w[keep])


def test_deleted_lists_do_not_hold_the_export_up():
    """A clique before and after the edges of its first vertices are deleted."""
    import torch
    import gv_b200
    from gv_b200 import _lib
    i, j = np.triu_indices(1500, 1)
    i, j = i.astype(np.uint32), j.astype(np.uint32)
    half = len(i) // 2
    with gv_b200.GraphVine(2048, hbm_budget_bytes=1 << 28, max_batch_pairs=len(i)) as g:
        g.batch_insert(i, j)
        g.synchronize()
        off = torch.empty(2049, dtype=torch.int64, device="cuda")
        dst = torch.empty(2 * len(i), dtype=torch.int32, device="cuda")
        best = []
        for _ in range(2):
            ts = []
            for _ in range(8):
                t = time.perf_counter()
                assert _lib.lib().gv_export_csr(g.handle, off.data_ptr(), dst.data_ptr(), None, dst.numel(),
                                                _lib.GV_MEM_DEVICE, None) == 0
                ts.append(time.perf_counter() - t)
            best.append(min(ts))
            g.batch_delete(i[:half], j[:half])
            g.synchronize()
    assert best[1] < 4 * best[0]  # 11 times with the deleted lists packed one after another
