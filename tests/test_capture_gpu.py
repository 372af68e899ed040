"""Searches captured into a CUDA graph by the caller and replayed, mixed with plain
ones on the same handle: a fused launch sets its search up itself and takes turns
with two barrier counters, which a replay must not depend on."""
import numpy as np
import pytest

import oracle
from back40computing_b200 import (CsrGraph, CsrProblem, BuildRmatGraph, sample_sources, EXPAND_CONTRACT,
                                  DIRECTION_OPTIMIZING, HYBRID)
from back40computing_b200 import _native as N
from back40computing_b200.bfs import ENACTORS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("strategy", [EXPAND_CONTRACT, DIRECTION_OPTIMIZING, HYBRID])
@pytest.mark.parametrize("preds", [False, True])
def test_captured_searches_replay(strategy, preds):
    import torch
    g = CsrGraph()
    BuildRmatGraph(1 << 13, 1 << 17, g, True, 0.57, 0.19, 0.19, seed=1, permute=True)
    a, b = (int(s) for s in sample_sources(g, 2, seed=9))
    p = CsrProblem.from_graph(g, mark_predecessors=preds)
    e = ENACTORS[strategy]()
    stream = torch.cuda.Stream()
    p.set_stream(stream.cuda_stream)
    N.check(p.Reset(e.GetFrontierType(), 1.3))
    want = {s: oracle.bfs(g.row_offsets, g.column_indices, s)[0] for s in (a, b)}

    def right(src):
        got = p.labels()
        if preds:
            return got[src] == -2 and oracle.check_predecessors(g.row_offsets, g.column_indices, want[src], got) == (-1, 0)
        return oracle.compare_labels(got, want[src]) == -1

    N.check(e.EnactFusedSearch(p, b))  # lazily built buffers and the handle's first search
    assert right(b)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        graph.capture_begin()
        N.check(e.EnactFusedSearch(p, a))
        assert p.Reset(e.GetFrontierType(), 1.3) != 0  # a reset cannot be captured
        graph.capture_end()
    for plain in (0, 1, 2):  # odd and even numbers of plain searches between replays
        for _ in range(plain):
            N.check(e.EnactFusedSearch(p, b))
            assert right(b)
        for _ in range(2):
            with torch.cuda.stream(stream):
                graph.replay()
            assert right(a)
    p.Destroy()


@pytest.mark.parametrize("strategy", [EXPAND_CONTRACT, DIRECTION_OPTIMIZING, HYBRID])
@pytest.mark.parametrize("preds", [False, True])
def test_capture_right_after_a_reset(strategy, preds):
    """The handle is clean when the search is captured and dirty when it is replayed."""
    import torch
    g = CsrGraph()
    BuildRmatGraph(1 << 12, 1 << 15, g, True, 0.57, 0.19, 0.19, seed=1, permute=True)
    a, b = (int(s) for s in sample_sources(g, 2, seed=9))
    p = CsrProblem.from_graph(g, mark_predecessors=preds)
    e = ENACTORS[strategy]()
    stream = torch.cuda.Stream()
    p.set_stream(stream.cuda_stream)
    N.check(p.Reset(e.GetFrontierType(), 1.3))
    want = {s: oracle.bfs(g.row_offsets, g.column_indices, s)[0] for s in (a, b)}

    def right(src):
        got = p.labels()
        if preds:
            return got[src] == -2 and oracle.check_predecessors(g.row_offsets, g.column_indices, want[src], got) == (-1, 0)
        return oracle.compare_labels(got, want[src]) == -1

    N.check(e.EnactFusedSearch(p, b))  # lazily built buffers
    N.check(p.Reset(e.GetFrontierType(), 1.3))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        graph.capture_begin()
        N.check(e.EnactFusedSearch(p, a))
        graph.capture_end()
    for _ in range(2):
        for _ in range(2):
            with torch.cuda.stream(stream):
                graph.replay()
            assert right(a)
        N.check(e.EnactFusedSearch(p, b))
        assert right(b)
    p.Destroy()
