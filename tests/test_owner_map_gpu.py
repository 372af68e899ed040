"""CTA-wide sub-rounds on levels of several sub-rounds per CTA (a small grid), where
each thread searches for its positions' entries: lists of one edge, of one and more
than a sub-round, and mixed, at ragged ends, against the oracle."""
import numpy as np
import pytest

import oracle
from back40computing_b200 import CsrGraph, CsrProblem, search, EXPAND_CONTRACT, DIRECTION_OPTIMIZING
from back40computing_b200 import _native as N

pytestmark = pytest.mark.gpu


def _two_levels(degrees):
    """A source, `degrees.size` vertices one level on, each with its own leaves."""
    d = np.asarray(degrees)
    k, n = d.size, 1 + d.size + int(d.sum())
    u = np.concatenate([np.zeros(k, np.int64), np.repeat(np.arange(1, k + 1), d)])
    g = CsrGraph()
    g.FromCoo(u, np.arange(1, n), n)
    return g


@pytest.mark.parametrize("threads", [128, 256, 512])
@pytest.mark.parametrize("grid", [1, 3])
@pytest.mark.parametrize("kind", ["ones", "long", "mixed", "exact"])
def test_entries_of_a_large_level(threads, grid, kind):
    degrees = {"ones": np.ones(6 * 2048 + 1, int), "long": [2047, 2048, 2049, 7000, 1],
               "mixed": np.random.default_rng(1).choice([1, 2, 31, 33, 300, 2100], 400),
               "exact": np.full(3 * 2048 // 16, 16)}[kind]
    g = _two_levels(degrees)
    p = CsrProblem.from_graph(g)
    pol = N.Policy()
    pol.threads, pol.warp_contract, pol.subgrid_frontier_edges, pol.small_frontier_edges = threads, -1, -1, -1
    want = oracle.bfs(g.row_offsets, g.column_indices, 0)[0]
    for strategy in (EXPAND_CONTRACT, DIRECTION_OPTIMIZING):
        got = search(p, 0, strategy=strategy, policy=pol, max_grid_size=grid)
        assert oracle.compare_labels(got, want) == -1
    p.Destroy()
