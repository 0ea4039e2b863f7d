"""Betweenness and BFS over out-edges alone: directed stores, and CSRs whose
entries do not come in pairs.  The last level is often of vertices without
out-entries, on its own or under vertices of every size class."""
import numpy as np
import pytest

import oracle

gv_b200 = pytest.importorskip("gv_b200")
pytestmark = pytest.mark.gpu


def _edges(shape):
    if shape == "path":     # a level of one sink
        return 3, [0, 1], [1, 2]
    if shape == "tree":     # binary, 7 levels of which the last has no out-entries: one past the lists that are kept
        return 127, np.repeat(np.arange(63), 2), np.arange(1, 127)
    if shape == "star":     # a hub of 3,000 out-entries, cut into pieces, above sinks only
        return 3001, np.zeros(3000, int), np.arange(1, 3001)
    if shape == "mixed":    # levels of sinks and others, then sinks only; parallel paths
        s = [0, 0, 0, 1, 1, 2, 2, 4, 5, 6, 6]
        d = [1, 2, 3, 4, 5, 5, 6, 7, 7, 7, 8]
        return 9, s, d
    if shape == "hub":      # a source above a hub of 5,000 and one of 700, whose leaves meet in two sinks
        s = np.concatenate([[0, 0], np.full(5000, 1), np.full(700, 2), np.arange(3, 5703)])
        d = np.concatenate([[1, 2], np.arange(3, 5003), np.arange(5003, 5703), 5703 + np.arange(5700) % 2])
        return 5705, s, d
    # nearly all vertices reach nearly all others at once, over edges that lead one way
    rng = np.random.default_rng(3)
    s, d = rng.integers(0, 1500, 12000), rng.integers(1500, 2000, 12000)
    t, e = rng.integers(0, 1500, 6000), rng.integers(0, 1500, 6000)
    return 2000, np.concatenate([s, t]), np.concatenate([d, e])


SHAPES = ["path", "tree", "star", "mixed", "hub", "random"]


def _check(g, o, src):
    got, want = g.bc(src), o.bc(src)
    # fp64 sums in another order, rounded once to fp32
    assert np.abs(got - want).max() <= 1.2e-7 * max(1.0, np.abs(want).max())
    for v in {int(src[0]), int(src[-1])}:
        (dist, sigma), (od, osg) = g.bfs_sigma(v), o.bfs_sigma(v)
        assert np.array_equal(dist, od) and np.array_equal(sigma, osg)


def _sources(n, k):
    src = np.random.default_rng(k).integers(0, n, k).astype(np.uint32)
    src[0] = 0
    return src


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("sources", [1, 32])
@pytest.mark.parametrize("block", [32, 128])
def test_directed_store(shape, sources, block):
    n, s, d = _edges(shape)
    s, d = np.asarray(s, np.uint32), np.asarray(d, np.uint32)
    o = oracle.OracleGraph(n, directed=True)
    o.insert(s, d)
    with gv_b200.GraphVine(n, block_size=block, directed=True, hbm_budget_bytes=1 << 27) as g:
        g.batch_insert(s, d)
        g.synchronize()
        _check(g, o, _sources(n, sources))


@pytest.mark.parametrize("shape", SHAPES)
def test_one_way_csr(shape):
    """A bulk build keeps a CSR as it is given, on undirected stores too."""
    n, s, d = _edges(shape)
    o = oracle.OracleGraph(n)
    o.insert(np.asarray(s, np.uint32), np.asarray(d, np.uint32), directed_entries=True)
    off, dst, _ = o.export()
    with gv_b200.GraphVine(n, hbm_budget_bytes=1 << 27) as g:
        g.bulk_build(off, dst)
        g.synchronize()
        _check(g, o, _sources(n, 32))


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("sources", [33, 64])
def test_directed_store_two_words(shape, sources):
    """More than 32 sources: passes that pull their wide levels on undirected stores."""
    n, s, d = _edges(shape)
    s, d = np.asarray(s, np.uint32), np.asarray(d, np.uint32)
    o = oracle.OracleGraph(n, directed=True)
    o.insert(s, d)
    with gv_b200.GraphVine(n, directed=True, hbm_budget_bytes=1 << 27) as g:
        g.batch_insert(s, d)
        g.synchronize()
        _check(g, o, _sources(n, sources))


def test_directed_store_pull_asked_for(monkeypatch):
    """GV_BC_PULL does not make a directed store pull."""
    monkeypatch.setenv("GV_BC_PULL", "1000000")
    n, s, d = _edges("random")
    s, d = np.asarray(s, np.uint32), np.asarray(d, np.uint32)
    o = oracle.OracleGraph(n, directed=True)
    o.insert(s, d)
    with gv_b200.GraphVine(n, directed=True, hbm_budget_bytes=1 << 27) as g:
        g.batch_insert(s, d)
        g.synchronize()
        _check(g, o, _sources(n, 16))
