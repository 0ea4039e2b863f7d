"""The one-launch sweep loop when a wait for its other CTAs runs out
(GV_PL_WAIT=0: at the first): the call gives what the sweeps give launch by
launch, bit for bit, and later calls take the loop again."""
import numpy as np
import pytest

gv_b200 = pytest.importorskip("gv_b200")
pytestmark = pytest.mark.gpu


def _calls(g, c, weighted, directed):
    if weighted:
        x, s1 = g.wpr_forward()
        grad, lam, s2 = g.wpr_backward(x, c)
        return [x, grad, lam, s1, s2]
    x, s1 = g.static_pagerank()
    warm, s2 = g.dynamic_pagerank(x)
    ppr, s3 = g.ppr(3)
    one, s4 = g.static_pagerank(max_iter=1)
    return [x, warm, ppr, one, s1, s2, s3, s4]


def _equal(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("directed,weighted", [(False, False), (True, False), (True, True)])
def test_wait_runs_out(directed, weighted, monkeypatch):
    n = 6_007
    rng = np.random.default_rng(4)
    hub = rng.choice(np.arange(20, n), 5000, replace=False)  # three items: summed otherwise in the loop
    s = np.concatenate([np.full(5000, 2), rng.integers(0, n // 2, n)]).astype(np.uint32)
    d = np.concatenate([hub, rng.integers(0, n, n)]).astype(np.uint32)
    if directed:
        s, d = np.concatenate([s, d]), np.concatenate([d, s])
    w = (0.1 + 0.9 * rng.random(len(s))).astype(np.float32)
    c = rng.standard_normal(n).astype(np.float32)
    with gv_b200.GraphVine(n, directed=directed, weighted=weighted, hbm_budget_bytes=1 << 28) as g:
        g.batch_insert(s, d, w if weighted else None)
        g.synchronize()
        loop = _calls(g, c, weighted, directed)
        monkeypatch.setenv("GV_PL_WAIT", "0")
        out = _calls(g, c, weighted, directed)
        monkeypatch.delenv("GV_PL_WAIT")
        again = _calls(g, c, weighted, directed)
        monkeypatch.setenv("GV_PL_LOOP", "0")
        sweeps = _calls(g, c, weighted, directed)
    assert _equal(out, sweeps)
    assert _equal(again, loop)
    assert not _equal(loop, sweeps)  # the two ways can be told apart here
