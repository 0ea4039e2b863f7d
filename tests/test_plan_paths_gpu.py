"""The sweep plan's forms against the store's own sweeps (GV_PR_PLAN=0): plain,
personalised and batched on undirected stores, in-edge transposes of directed
and weighted ones, the adjoint; one launch for all sweeps (GV_PL_LOOP) and
launches per sweep; graphs without hubs, with hubs of several items, with
rows that have no entries in one direction, and without edges."""
import numpy as np
import pytest

gv_b200 = pytest.importorskip("gv_b200")
pytestmark = pytest.mark.gpu


def _pairs(shape, n, rng):
    if shape == "empty":
        return np.zeros((2, 0), np.uint32)
    if shape == "sparse":  # rows of 0 to a few entries
        return rng.integers(0, n, (2, n // 2)).astype(np.uint32)
    # hubs: rows of 63..2049 entries and one of 3 items, many vertices that only receive
    deg = [63, 64, 65, 7, 8, 9, 2047, 2048, 2049, 5000]
    src = np.repeat(np.arange(len(deg), dtype=np.uint32), deg)
    dst = np.concatenate([rng.choice(np.arange(20, n), d, replace=False) for d in deg]).astype(np.uint32)
    more = rng.integers(0, n // 2, (2, n)).astype(np.uint32)
    return np.concatenate([np.stack([src, dst]), more], 1)


def _l1(a, b):
    return float(np.abs(a.astype(np.float64) - b.astype(np.float64)).sum())


# The two runs differ in summation order only.  A sum of d terms of one sign in
# fp32 is within d * 2^-24 of itself, lanes and items cut d to at most 2048 / 32
# + 32 terms in a chain, and the sweeps' errors add up to at most 1 / (1 - alpha)
# of one sweep's: 96 * 6e-8 / 0.15 = 4e-5 of an L1 norm of 1; and either may stop
# a sweep earlier: 2 * eps * alpha / (1 - alpha) = 1.1e-5.
TOL = 4e-5 + 1.1e-5


@pytest.mark.parametrize("loop", ["0", "1e12"])
@pytest.mark.parametrize("shape", ["hubs", "sparse", "empty"])
@pytest.mark.parametrize("directed,weighted", [(False, False), (True, False), (True, True), (False, True)])
def test_plan_equals_store_sweeps(directed, weighted, shape, loop, monkeypatch):
    n = 9_001
    rng = np.random.default_rng(directed + 2 * weighted)
    src, dst = _pairs(shape, n, rng)
    w = (0.1 + 0.9 * rng.random(len(src))).astype(np.float32)
    c = rng.standard_normal(n).astype(np.float32)
    got = {}
    with gv_b200.GraphVine(n, block_size=64, directed=directed, weighted=weighted, hbm_budget_bytes=1 << 28) as g:
        if len(src):
            g.batch_insert(src, dst, w if weighted else None)
            g.batch_delete(src[::17], dst[::17])  # tombstones in the rows
        g.synchronize()
        for plan in ("0", "1"):
            monkeypatch.setenv("GV_PR_PLAN", plan)
            monkeypatch.setenv("GV_PL_LOOP", loop)
            r = {}
            if weighted:
                r["x"], _ = g.wpr_forward()
                r["grad"], r["lambda"], _ = g.wpr_backward(r["x"], c)
            else:
                r["x"], _ = g.static_pagerank()
                r["warm"], _ = g.dynamic_pagerank(r["x"])
                r["ppr"], _ = g.ppr(int(src[0]) if len(src) else 3)
                if not directed:
                    r["batch"], _ = g.ppr_batch([0, 5, n - 1])
            got[plan] = r
    for key, a in got["0"].items():
        b = got["1"][key]
        if key in ("lambda", "grad"):  # signed: against the largest entry, the same chains of terms
            assert np.abs(a - b).max(initial=0.0) <= TOL * max(1.0, np.abs(a).max(initial=0.0))
        else:
            cols = a.shape[1] if a.ndim == 2 else 1
            assert _l1(a, b) <= cols * TOL, key


@pytest.mark.parametrize("max_iter", [0, 1, 2, 3, 8, 9])
@pytest.mark.parametrize("loop", ["0", "1e12"])
def test_sweep_limit(max_iter, loop, monkeypatch):
    """Both iterates hold every row after any number of sweeps."""
    n = 5_000
    rng = np.random.default_rng(1)
    src, dst = _pairs("sparse", n, rng)
    monkeypatch.setenv("GV_PL_LOOP", loop)
    with gv_b200.GraphVine(n, directed=True, hbm_budget_bytes=1 << 28) as g:
        g.batch_insert(src, dst)
        g.synchronize()
        x, sweeps = g.static_pagerank(max_iter=max_iter, epsilon=0.0)
        off, nb, _ = g.export_csr()
    assert sweeps == max_iter
    deg = np.diff(off.astype(np.int64))
    u = np.repeat(np.arange(n), deg)
    want = np.full(n, 1.0 / n)
    for _ in range(max_iter):
        y = np.bincount(nb, (want / np.maximum(deg, 1))[u], minlength=n)
        want = 0.15 / n + 0.85 * y
    assert np.abs(x - want).sum() <= 1e-6
