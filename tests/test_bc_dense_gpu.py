"""Betweenness on few vertices with long lists: nearly every vertex is a whole
CTA's, and all CTAs have to take part."""
import time

import numpy as np
import pytest

import oracle

gv_b200 = pytest.importorskip("gv_b200")
pytestmark = pytest.mark.gpu


def _graph(n, deg, seed):
    s, d = np.random.default_rng(seed).integers(0, n, (2, n * deg // 2)).astype(np.uint32)
    g = gv_b200.GraphVine(n, hbm_budget_bytes=1 << 29, max_batch_pairs=len(s))
    g.batch_insert(s, d)
    g.synchronize()
    return g, s, d


@pytest.mark.parametrize("n,deg", [(40, 30), (700, 350), (3_000, 300), (1 << 16, 20), ((1 << 16) + 1, 20)])
@pytest.mark.parametrize("sources", [1, 33])
def test_dense(n, deg, sources):
    g, s, d = _graph(n, deg, n)
    o = oracle.OracleGraph(n)
    o.insert(s, d)
    src = np.random.default_rng(1).integers(0, n, sources).astype(np.uint32)
    got, want = g.bc(src), o.bc(src)
    # fp64 sums in another order, rounded once to fp32
    assert np.abs(got - want).max() <= 1.2e-7 * max(1.0, np.abs(want).max())
    g.close()


def test_entries_and_not_vertices_set_the_time():
    """The same million entries on 4 K vertices and on 64 K: the first have fewer rows to fill."""
    src, best = np.arange(32, dtype=np.uint32), []
    for n, deg in ((1 << 12, 512), (1 << 16, 32)):
        g, _, _ = _graph(n, deg, 2)
        ts = []
        for _ in range(6):
            t = time.perf_counter()
            g.bc(src)
            ts.append(time.perf_counter() - t)
        best.append(min(ts))
        g.close()
    assert best[0] < 1.1 * best[1]  # 1.5 times with a fifth of the CTAs, few of them
