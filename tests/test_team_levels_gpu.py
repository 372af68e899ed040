"""Resident levels (a team of CTAs that keeps its frontier in shared memory):
entered, grown, shrunk and left at the sizes where their bookkeeping can go
wrong, against the oracle's distances, search depth and queue totals."""
import numpy as np
import pytest

import oracle
from back40computing_b200 import (CsrGraph, CsrProblem, BuildGrid3dGraph, search, EXPAND_CONTRACT, CONTRACT_EXPAND,
                                  TWO_PHASE, HYBRID, DIRECTION_OPTIMIZING)
from back40computing_b200 import _native as N
from back40computing_b200.bfs import ENACTORS

pytestmark = pytest.mark.gpu


def _undirected(n, u, v):
    u, v = np.concatenate([np.atleast_1d(x) for x in u]), np.concatenate([np.atleast_1d(x) for x in v])
    g = CsrGraph()
    g.FromCoo(np.concatenate([u, v]), np.concatenate([v, u]), n)
    return g


def _chains(first, heads, length):
    """`length` further vertices behind each head, level by level: (edges, next id, last vertices)."""
    us, vs, last = [], [], heads
    for _ in range(length):
        new = np.arange(first, first + last.size)
        us.append(last)
        vs.append(new)
        first, last = first + new.size, new
    return us, vs, first, last


def _graph(kind):
    if kind == "lattice":  # grows to 4000 edges a level and shrinks again, team sizes 1 to 8
        g = CsrGraph()
        BuildGrid3dGraph(24, g)
        return g
    if kind == "path":     # one vertex a level, past the levels of a phase
        i = np.arange(4200)
        return _undirected(4201, [i], [i + 1])
    if kind == "tree":     # four times the edges each level: every phase overflows
        child = np.arange(1, (4 ** 9 - 1) // 3)
        return _undirected(child.size + 1, [(child - 1) // 4], [child])
    if kind == "fan":      # 700 chains of 30, one sink, one chain: a team that shrinks to one CTA
        us, vs, n, last = _chains(701, np.arange(1, 701), 30)
        sink = n
        u2, v2, n, _ = _chains(sink + 1, np.array([sink]), 50)
        return _undirected(n, [np.zeros(700, int), *us, last, *u2], [np.arange(1, 701), *vs, np.full(700, sink), *v2])
    # "hub": a chain, then a hub of 40,000 leaves with a chain of 3 behind each
    u0, v0, n, _ = _chains(1, np.array([0]), 20)
    hub = n - 1
    leaves = np.arange(n, n + 40000)
    us, vs, n, _ = _chains(n + 40000, leaves, 3)
    return _undirected(n, [*u0, np.full(40000, hub), *us], [*v0, leaves, *vs])


@pytest.mark.parametrize("kind", ["lattice", "path", "tree", "fan", "hub"])
@pytest.mark.parametrize("threads,knobs", [(0, {}), (128, {}), (256, {"small_frontier_edges": -1}),
                                           (512, {"small_frontier_edges": 2048, "ctas_per_sm": 1}),
                                           (256, {"subgrid_frontier_edges": 3000}),
                                           (512, {"subgrid_frontier_edges": -1})])
@pytest.mark.parametrize("preds", [False, True])
def test_team_levels(kind, threads, knobs, preds):
    g = _graph(kind)
    p = CsrProblem.from_graph(g, mark_predecessors=preds)
    pol = None
    if threads:
        pol = N.Policy()
        pol.threads = threads
        for k, v in knobs.items():
            setattr(pol, k, v)
    for strategy in (EXPAND_CONTRACT, DIRECTION_OPTIMIZING):
        for limit in (-1, 19):
            got = search(p, 0, strategy=strategy, policy=pol, depth_limit=limit)
            want, depth = oracle.bfs(g.row_offsets, g.column_indices, 0)
            if limit >= 0:
                want = np.where(want > limit, -1, want)
                depth = int(want.max()) + 1
            if preds:
                assert got[0] == -2
                assert np.array_equal(got != -1, want != -1)
                reached = np.flatnonzero(got >= 0)
                assert np.array_equal(want[got[reached]] + 1, want[reached])
            else:
                assert oracle.compare_labels(got, want) == -1
            e = ENACTORS[strategy]()
            e._problem = p
            queued, got_depth, _ = e.GetStatistics()
            assert got_depth == depth
            if limit < 0:
                assert queued == int((want >= 0).sum()) - 1
    p.Destroy()


@pytest.mark.parametrize("n,degree", [(2, 40), (33, 200), (2154, 16), (20000, 8)])
@pytest.mark.parametrize("threads,precheck", [(0, 0), (256, 0), (256, -1), (512, 0)])
def test_levels_of_more_edges_than_vertices(n, degree, threads, precheck):
    """Few vertices, many edges: team levels and levels launched one by one."""
    rng = np.random.default_rng(n)
    u, v = rng.integers(0, n, n * degree), rng.integers(0, n, n * degree)
    g = _undirected(n, [u], [v])
    want, _ = oracle.bfs(g.row_offsets, g.column_indices, 0)
    pol = None
    if threads:
        pol = N.Policy()
        pol.threads, pol.bitmask_precheck = threads, precheck
    for preds in (False, True):
        p = CsrProblem.from_graph(g, mark_predecessors=preds)
        for mode in (N.ENACT_FUSED, N.ENACT_ITERATIVE, N.ENACT_GRAPH):
            got = search(p, 0, strategy=EXPAND_CONTRACT, policy=pol, mode=mode)
            assert np.array_equal(got != -1, want != -1)
            if preds:
                reached = np.flatnonzero(got >= 0)
                assert np.array_equal(want[got[reached]] + 1, want[reached])
            else:
                assert oracle.compare_labels(got, want) == -1


@pytest.mark.parametrize("strategy", [CONTRACT_EXPAND, TWO_PHASE, HYBRID])
@pytest.mark.parametrize("threads", [128, 256, 512])
def test_edge_strategies_take_a_subgrid_threshold(strategy, threads):
    """With any CTA size, where the vertex-frontier strategies ask for 256 threads."""
    g = _graph("lattice")
    p = CsrProblem.from_graph(g)
    pol = N.Policy()
    pol.threads, pol.subgrid_frontier_edges = threads, 3000
    want = oracle.bfs(g.row_offsets, g.column_indices, 0)[0]
    assert oracle.compare_labels(search(p, 0, strategy=strategy, policy=pol), want) == -1
    if threads != 256:
        with pytest.raises(N.B40cError):
            search(p, 0, strategy=EXPAND_CONTRACT, policy=pol)
    p.Destroy()


@pytest.mark.parametrize("kind", ["lattice", "hub"])
@pytest.mark.parametrize("strategy", [EXPAND_CONTRACT, DIRECTION_OPTIMIZING])
@pytest.mark.parametrize("mode", [N.ENACT_FUSED, N.ENACT_GRAPH])
def test_host_mapped_graph(kind, strategy, mode):
    """Levels of a CSR read from host memory take their winners' rows only."""
    g = _graph(kind)
    want = oracle.bfs(g.row_offsets, g.column_indices, 0)[0]
    p = CsrProblem.from_graph(g, stream_from_host=True)
    for _ in range(2):
        assert oracle.compare_labels(search(p, 0, strategy=strategy, mode=mode), want) == -1
    p.Destroy()
