"""Betweenness scratch: sized for the graph at hand, its level counters growing
with the search, and pieces of hubs larger where the store is dense."""
import numpy as np
import pytest
import torch

import oracle

gv_b200 = pytest.importorskip("gv_b200")
pytestmark = pytest.mark.gpu


def _same(g, o, src):
    got, want = g.bc(src), o.bc(src)
    # fp64 sums in another order, rounded once to fp32
    assert np.abs(got - want).max() <= 1.2e-7 * max(1.0, np.abs(want).max())


def _both(n, s, d, **kw):
    s, d = np.asarray(s, np.uint32), np.asarray(d, np.uint32)
    o = oracle.OracleGraph(n)
    o.insert(s, d)
    g = gv_b200.GraphVine(n, **kw)
    g.batch_insert(s, d)
    g.synchronize()
    return g, o


@pytest.mark.parametrize("length", [509, 510, 513, 1400])
def test_more_levels_than_the_first_counters(length):
    n = length + 1
    g, o = _both(n, np.arange(length), np.arange(1, n), hbm_budget_bytes=1 << 27)
    for src in (np.array([0], np.uint32), np.arange(0, 64, dtype=np.uint32), np.array([length], np.uint32)):
        _same(g, o, src)  # the second and third calls find the grown counters
    dist, sigma = g.bfs_sigma(0)
    assert np.array_equal(dist, np.arange(n)) and np.all(sigma == 1)
    g.close()


@pytest.mark.parametrize("sources", [3, 40])
def test_dense_store_has_larger_pieces(sources):
    """100 hubs over 8,900 vertices: more entries than pieces of the least size hold."""
    a, b = np.meshgrid(np.arange(100), np.arange(100, 9000))
    g, o = _both(9000, a.ravel(), b.ravel(), hbm_budget_bytes=1 << 28)
    _same(g, o, np.random.default_rng(sources).integers(0, 9000, sources).astype(np.uint32))
    g.close()


def test_tight_pool():
    """A pool of fewer slots than the least number of pieces of the least size."""
    g, o = _both(1500, np.zeros(1400, int), np.arange(1, 1401), block_size=32, pool_blocks=1600)
    _same(g, o, np.array([0, 5, 1499], np.uint32))
    g.close()


def test_first_call_takes_what_the_graph_needs():
    n = 1 << 14
    s, d = oracle.rmat_pairs(14, 1 << 18, 5)
    g = gv_b200.GraphVine(n, pool_blocks=1 << 15)
    g.batch_insert(s, d)
    g.synchronize()
    with gv_b200.GraphVine(64, pool_blocks=64) as warm:  # modules and their memory, not this graph's
        warm.batch_insert(np.array([0], np.uint32), np.array([1], np.uint32))
        warm.bc(np.array([0], np.uint32))
    before = torch.cuda.mem_get_info()[0]
    g.bc(np.arange(32, dtype=np.uint32))
    took = before - torch.cuda.mem_get_info()[0]
    # per vertex: a row of 256, 40 of masks, lists and the score, an eighth of a
    # piece and a half (268 each); a quarter more; 32 levels of masks; 2 MB
    # rounding of three allocations
    assert took <= 1.25 * n * (256 + 40 + 268 * 1.5 / 8) + 128 * n + (6 << 20)
    g.close()
