"""Per-vertex triangle counts where the oriented lists are short: hubs that
most triangles go to, and many vertices of a few entries each."""
import time

import numpy as np
import pytest

import oracle

gv_b200 = pytest.importorskip("gv_b200")
pytestmark = pytest.mark.gpu


def _hubs(n, hubs, next_ones, low):
    """`hubs` vertices over all others, each linked to the next ones; low: the hubs have the smallest ids."""
    leaf = np.arange(hubs, n)
    s = [np.full(len(leaf), h) for h in range(hubs)] + [leaf[:-k] for k in range(1, next_ones + 1)]
    d = [leaf] * hubs + [leaf[k:] for k in range(1, next_ones + 1)]
    s, d = np.concatenate(s), np.concatenate(d)
    if not low:
        s, d = n - 1 - s, n - 1 - d
    return s.astype(np.uint32), d.astype(np.uint32)


def _best(f, k=5):
    best = 1e9
    for _ in range(k):
        t = time.perf_counter()
        f()
        best = min(best, time.perf_counter() - t)
    return best


@pytest.mark.parametrize("n,hubs,next_ones", [(50, 1, 1), (5_000, 1, 2), (9_001, 100, 20), (40_000, 3, 120),
                                              (3_000, 1_500, 0)])
@pytest.mark.parametrize("low", [True, False])
def test_hubs_over_short_lists(n, hubs, next_ones, low, monkeypatch):
    """One key for nearly all credits, and more keys than a CTA's table has slots."""
    s, d = _hubs(n, hubs, next_ones, low)
    if hubs == 1_500:  # rather: cliques of 60 under shuffled ids, every vertex credited
        rng = np.random.default_rng(1)
        i, j = np.triu_indices(60, 1)
        p, base = rng.permutation(n), np.arange(0, n, 60)[:, None]
        s, d = p[(base + i).ravel()].astype(np.uint32), p[(base + j).ravel()].astype(np.uint32)
    o = oracle.OracleGraph(n)
    o.insert(s, d)
    monkeypatch.setenv("GV_TC_SUBSET", "global")
    with gv_b200.GraphVine(n, hbm_budget_bytes=1 << 28) as g:
        g.batch_insert(s, d)
        for packed in (None, "1"):
            if packed:
                monkeypatch.setenv("GV_TC_PACKED", packed)
            own, total = g.static_tc()
            want, wtotal = o.tc()
            assert total == wtotal and np.array_equal(own, want)
            every = np.arange(n, dtype=np.uint32)
            assert np.array_equal(g.tc_subset(every), o.tc_incident(every))


def test_hub_does_not_hold_the_count_up():
    """A million triangles and more for one vertex cost little more than their total."""
    n = 1 << 19
    s, d = _hubs(n, 1, 10, True)
    with gv_b200.GraphVine(n, hbm_budget_bytes=2 << 30) as g:
        g.batch_insert(s, d)
        g.synchronize()
        import ctypes as C
        import torch
        from gv_b200 import _lib
        pv, tot = torch.empty(n, dtype=torch.int64, device="cuda"), C.c_uint64()
        L = _lib.lib()
        own = _best(lambda: L.gv_tc(g.handle, pv.data_ptr(), C.byref(tot), _lib.GV_MEM_DEVICE, None))
        total = _best(lambda: L.gv_tc(g.handle, None, C.byref(tot), _lib.GV_MEM_DEVICE, None))
        assert int(pv.sum()) == tot.value
    assert own < 3 * total  # an atomic of its own per triangle: 7 times


@pytest.mark.parametrize("per", [1, 2, 3, 4])
def test_sparse_vertices(per):
    """More than 2^18 vertices with lists of a few entries, on either side of the line."""
    n = (1 << 18) + 77
    rng = np.random.default_rng(per)
    s, d = rng.integers(0, n, (2, per * n)).astype(np.uint32)
    a, b = _hubs(900, 2, 3, True)  # and triangles
    s, d = np.concatenate([s, a]), np.concatenate([d, b])
    o = oracle.OracleGraph(n)
    o.insert(s, d)
    with gv_b200.GraphVine(n, hbm_budget_bytes=1 << 29) as g:
        g.batch_insert(s, d)
        own, total = g.static_tc()
        want, wtotal = o.tc()
    assert total == wtotal and np.array_equal(own, want)


def test_sparse_vertices_take_the_cheaper_way(monkeypatch):
    """A wheel: lists of two entries on two million vertices, per owner."""
    import ctypes as C
    import torch
    from gv_b200 import _lib
    n = 1 << 21
    s, d = _hubs(n, 1, 1, True)
    L, tot, t = _lib.lib(), C.c_uint64(), {}
    with gv_b200.GraphVine(n, hbm_budget_bytes=4 << 30, max_batch_pairs=len(s)) as g:
        g.batch_insert(s, d)
        g.synchronize()
        pv = torch.empty(n, dtype=torch.int64, device="cuda")
        for way in (None, "0", "1"):
            if way:
                monkeypatch.setenv("GV_TC_PACKED", way)
            t[way] = _best(lambda: L.gv_tc(g.handle, pv.data_ptr(), C.byref(tot), _lib.GV_MEM_DEVICE, None), 9)
    assert t[None] < 1.25 * min(t["0"], t["1"])
