"""Betweenness over level shapes: more levels than keep their lists, levels of
one vertex, vertices on either side of the CTA threshold, one vertex in
several source slots, and rounds that end inside a listing kernel's share."""
import numpy as np
import pytest

import oracle

gv_b200 = pytest.importorskip("gv_b200")
pytestmark = pytest.mark.gpu


def _edges(shape):
    if shape == "path":       # 30 levels
        return 31, np.arange(30), np.arange(1, 31)
    if shape == "layers":     # 9 layers of 150, complete between neighbours: wide late levels
        a, b = np.meshgrid(np.arange(150), np.arange(150))
        s = np.concatenate([a.ravel() + 150 * i for i in range(8)])
        return 1350, s, np.concatenate([b.ravel() + 150 * (i + 1) for i in range(8)])
    # stars whose hubs have 511, 512, 513, 1024 and 1025 entries, joined in a ring with a tail
    deg = [511, 512, 513, 1024, 1025, 4097]
    s, d, at = [], [], len(deg)
    for h, k in enumerate(deg):
        s += [h] * (k - 2) + [h]
        d += list(range(at, at + k - 2)) + [(h + 1) % len(deg)]
        at += k - 2
    s += [at - 1, at]
    d += [at, at + 1]
    return at + 2, np.array(s), np.array(d)


@pytest.mark.parametrize("shape", ["path", "layers", "stars"])
@pytest.mark.parametrize("sources", [1, 33, 64])
@pytest.mark.parametrize("block", [32, 128])
def test_bc_shapes(shape, sources, block):
    n, s, d = _edges(shape)
    rng = np.random.default_rng(sources)
    src = rng.integers(0, n, sources).astype(np.uint32)  # repeats among them
    if sources > 2:
        src[1] = src[0]
    with gv_b200.GraphVine(n, block_size=block, hbm_budget_bytes=1 << 27) as g:
        g.batch_insert(s.astype(np.uint32), d.astype(np.uint32))
        g.synchronize()
        got = g.bc(src)
        dist, sigma = g.bfs_sigma(int(src[0]))
    o = oracle.OracleGraph(n)
    o.insert(s.astype(np.uint32), d.astype(np.uint32))
    want = o.bc(src)
    # fp64 sums in another order, rounded once to fp32
    assert np.abs(got - want).max() <= 1.2e-7 * max(1.0, np.abs(want).max())
    od, osg = o.bfs_sigma(int(src[0]))
    assert np.array_equal(dist, od) and np.array_equal(sigma, osg)
