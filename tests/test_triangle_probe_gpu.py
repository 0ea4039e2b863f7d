"""Triangle counts on graphs of short oriented lists, which take the hash
probes: lists around a warp's 32, the 128 a warp takes at most (and 129, which
leaves that path), many vertices without any, deletes in between."""
import numpy as np
import pytest

import oracle

gv_b200 = pytest.importorskip("gv_b200")
pytestmark = pytest.mark.gpu


def _cliques(sizes, n, rng):
    perm, at, s, d = rng.permutation(n), 0, [], []
    for k in sizes:
        i, j = np.triu_indices(k, 1)
        s.append(perm[at + i])
        d.append(perm[at + j])
        at += k
    return np.concatenate(s).astype(np.uint32), np.concatenate(d).astype(np.uint32)


@pytest.mark.parametrize("sizes", [[2, 3], [32, 33, 34, 65], [128, 129], [129, 130], []])
@pytest.mark.parametrize("block", [32, 128])
def test_short_lists(sizes, block, monkeypatch):
    n = 6_007
    rng = np.random.default_rng(len(sizes) + block)
    s, d = rng.integers(0, n, (2, 5 * n)).astype(np.uint32)
    if sizes:
        a, b = _cliques(sizes, n, rng)
        s, d = np.concatenate([s, a]), np.concatenate([d, b])
    o = oracle.OracleGraph(n)
    o.insert(s, d)
    monkeypatch.setenv("GV_TC_SUBSET", "global")
    with gv_b200.GraphVine(n, block_size=block, hbm_budget_bytes=1 << 27) as g:
        g.batch_insert(s, d)
        for _ in range(2):
            own, total = g.static_tc()
            want, wtotal = o.tc()
            assert total == wtotal and np.array_equal(own, want)
            assert g.static_tc(per_vertex=False)[1] == wtotal
            sub = rng.choice(n, 300, replace=False).astype(np.uint32)
            assert np.array_equal(g.tc_subset(sub), o.tc_incident(sub))
            g.batch_delete(s[::3], d[::3])  # tombstones stay in the lists
            o.delete(s[::3], d[::3])


@pytest.mark.parametrize("core", ["32", "700", "65504"])
@pytest.mark.parametrize("n,k", [(40, 3), (1_500, 400), (3_000, 1_100)])
def test_core_lists_around_their_tiles(n, k, core, monkeypatch):
    """The core's lists, rows and merge list come from prefix counts over tiles
    of 1,024 edges: fewer edges than a tile, lists over several tiles, runs of
    one source and of many in a warp's 32 edges, and a core of every vertex."""
    monkeypatch.setenv("GV_TC_CORE", core)
    rng = np.random.default_rng(n + k)
    s, d = _cliques([k], n, rng)
    a, b = rng.integers(0, n, (2, 3 * n)).astype(np.uint32)
    s, d = np.concatenate([s, a]), np.concatenate([d, b])
    o = oracle.OracleGraph(n)
    o.insert(s, d)
    with gv_b200.GraphVine(n, hbm_budget_bytes=1 << 28) as g:
        g.batch_insert(s, d)
        assert g.static_tc(per_vertex=False)[1] == o.tc()[1]
        g.batch_delete(s[::2], d[::2])
        o.delete(s[::2], d[::2])
        assert g.static_tc(per_vertex=False)[1] == o.tc()[1]


@pytest.mark.parametrize("n,deg,hubs,core", [
    (6_000, 300, 0, "65504"),    # bitmaps of more than 32 chunks, then indices
    (6_000, 300, 0, "96"),       # few core entries a list: indices alone
    (200, 60, 0, "65504"),       # a bitmap of two chunks holds all of a list
    (40_000, 14, 40, "65504"),   # core indices past those counted in shared memory
    (40_000, 14, 40, "33000"),
    (7, 6, 0, "65504"),          # a core smaller than a word
])
def test_core_chunks(n, deg, hubs, core, monkeypatch):
    """Runs of bitmap and index chunks up to each edge's end: dense lists, sparse
    ones, both, ties of degree in the core's order, and cores on either side of
    the shared-memory counters."""
    monkeypatch.setenv("GV_TC_CORE", core)
    rng = np.random.default_rng(n + deg + hubs)
    s = rng.integers(0, n, n * deg // 2).astype(np.uint32)
    d = rng.integers(0, n, n * deg // 2).astype(np.uint32)
    if hubs:
        top = rng.choice(n, hubs, replace=False).astype(np.uint32)
        s = np.concatenate([s, np.repeat(top, 3_000)])
        d = np.concatenate([d, rng.integers(0, n, 3_000 * hubs).astype(np.uint32)])
    s, d = s[s != d], d[s != d]
    o = oracle.OracleGraph(n)
    o.insert(s, d)
    with gv_b200.GraphVine(n, hbm_budget_bytes=1 << 28) as g:
        g.batch_insert(s, d)
        assert g.static_tc(per_vertex=False)[1] == o.tc()[1]
        assert 0 < g.last_stat("tc_core") <= int(core)
        g.batch_delete(s[::3], d[::3])
        o.delete(s[::3], d[::3])
        assert g.static_tc(per_vertex=False)[1] == o.tc()[1]


@pytest.mark.parametrize("k", [17, 33, 34, 65, 66, 129, 130, 257, 258, 514, 1_026])
def test_list_sorts(k, monkeypatch):
    """Oriented lists of up to k - 1 entries (a clique's, one of each length), so
    around 16, 32, 64, 128, 256, 512 and 1,024, where the sorts change over."""
    monkeypatch.setenv("GV_TC_PACKED", "0")
    n = 2_000
    rng = np.random.default_rng(k)
    s, d = _cliques([k], n, rng)
    a, b = rng.integers(0, n, (2, n)).astype(np.uint32)
    s, d = np.concatenate([s, a]), np.concatenate([d, b])
    perm = rng.permutation(len(s))
    o = oracle.OracleGraph(n)
    o.insert(s, d)
    with gv_b200.GraphVine(n, hbm_budget_bytes=1 << 27) as g:
        for part in np.array_split(perm, 3):  # lists in no order
            g.batch_insert(s[part], d[part])
        own, total = g.static_tc()
        want, wtotal = o.tc()
        assert total == wtotal and np.array_equal(own, want)
        for core in ("0", "32"):
            monkeypatch.setenv("GV_TC_CORE", core)
            assert g.static_tc(per_vertex=False)[1] == wtotal
