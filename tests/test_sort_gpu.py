"""The radix sort through the batches that use it: sizes around its tiles (2,048
and 4,096 keys) and a few hundred of them, keys of few and of many bits, one
destination for most of a batch (a digit that fills whole tiles), weights that
show whether the sort is stable, and (GV_RS_WAIT=0) tiles that count the digits
of those before them rather than wait."""
import numpy as np
import pytest

gv_b200 = pytest.importorskip("gv_b200")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wait", [None, "0", "1"])
@pytest.mark.parametrize("pairs", [4_097, 6_144, 6_145, 300_000, 4_200_000])
@pytest.mark.parametrize("n", [40, 5_000, 1 << 20])
def test_weighted_batch_keeps_the_first_of_each_pair(wait, pairs, n, monkeypatch):
    import torch
    if wait is not None:
        monkeypatch.setenv("GV_RS_WAIT", wait)
        if pairs > 300_000:
            pytest.skip("a recount reads a tile per digit: kept to the smaller batches")
    gen = torch.Generator(device="cuda").manual_seed(pairs + n)
    s = torch.randint(0, n, (pairs,), generator=gen, device="cuda")
    d = torch.randint(0, n, (pairs,), generator=gen, device="cuda")
    d[: pairs // 2] = n // 2
    w = torch.rand(pairs, generator=gen, device="cuda")
    with gv_b200.GraphVine(n, block_size=32, directed=True, weighted=True, pool_blocks=n + pairs // 16 + 64,
                           max_batch_pairs=pairs) as g:
        g.batch_insert(s.int(), d.int(), w)
        g.synchronize()
        off, dst, wt = g.export_csr(with_weights=True)
    key = (s * n + d)[s != d]
    uniq, inv = torch.unique(key, return_inverse=True)
    first = torch.full((uniq.numel(),), pairs, device="cuda").scatter_reduce_(
        0, inv, torch.arange(key.numel(), device="cuda"), "amin")
    want_w = w[s != d][first].cpu().numpy()
    src = np.repeat(np.arange(n), np.diff(off.astype(np.int64)))
    assert np.array_equal(src * n + dst, uniq.cpu().numpy())
    assert np.array_equal(wt, want_w)
