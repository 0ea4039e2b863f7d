"""Windows whose pairs are just below, at and above the power of two that their
buffers are rounded up to, and tiny ones: the sort and the net effect stop at the
window's own entries, whatever an earlier and larger window left behind them."""
import numpy as np
import pytest

import oracle
from tests.helpers import assert_same_adjacency, assert_sound

gv_b200 = pytest.importorskip("gv_b200")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("graph", [False, True])
def test_window_sizes_around_their_capacity(directed, graph):
    n = 5_003
    rng = np.random.default_rng(7)
    o = oracle.OracleGraph(n, directed=directed)
    with gv_b200.GraphVine(n, directed=directed, hbm_budget_bytes=1 << 28, max_batch_pairs=1 << 16) as g:
        for pairs in (16_384, 16_385, 16_383, 8_193, 3, 1, 4_096):
            s, d = rng.integers(0, n, (2, pairs)).astype(np.uint32)
            s[0] = d[0] = 5  # a loop
            a, b = pairs // 2, pairs - pairs // 2
            c = a // 3
            batches = [(s[:a], d[:a], s[:c], d[:c]), (s[a:], d[a:], d[:c], s[:c])]
            total = sum(len(x) for q in batches for x in (q[0], q[2]))
            g.clear_affected()
            g.batch_run(batches, compact=True, graph=graph)
            g.synchronize()
            for q in batches:
                o.insert(q[0], q[1])
                o.delete(q[2], q[3])
            ends = np.zeros(n, np.uint8)
            for q in batches:
                for x, y in ((q[0], q[1]), (q[2], q[3])):
                    ends[x[x != y]] = 1
                    ends[y[x != y]] = 1
            assert np.array_equal(g.affected() != 0, ends != 0), (pairs, total)
            assert_same_adjacency(g, o)
        assert_sound(g)
