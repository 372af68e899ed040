"""What a reset and a change of stream leave behind: a reset's fills are done when it
returns, whatever stream reads them, and a change of stream touches no stream."""
import ctypes as C
import time

import numpy as np
import pytest

import oracle
from back40computing_b200 import CsrGraph, CsrProblem, BuildRmatGraph, sample_sources, EXPAND_CONTRACT
from back40computing_b200 import _native as N
from back40computing_b200.bfs import ENACTORS

pytestmark = pytest.mark.gpu


class _View:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": (n,), "typestr": "<i4", "version": 3}


@pytest.fixture
def searched():
    """(problem after one search on a stream of its own, enactor, stream, source, labels)"""
    import torch
    g = CsrGraph()
    BuildRmatGraph(1 << 14, 1 << 17, g, True, 0.57, 0.19, 0.19, seed=3, permute=True)
    src = int(sample_sources(g, 1, seed=5)[0])
    p = CsrProblem.from_graph(g)
    e = ENACTORS[EXPAND_CONTRACT]()
    stream = torch.cuda.Stream()
    p.set_stream(stream.cuda_stream)
    N.check(p.Reset(e.GetFrontierType(), 1.3))
    N.check(e.EnactFusedSearch(p, src))
    want = oracle.bfs(g.row_offsets, g.column_indices, src)[0]
    assert oracle.compare_labels(p.labels(), want) == -1
    yield p, e, stream, src, want
    p.Destroy()


def _busy(stream, ms):
    """Keeps a stream busy for about that long (at up to 2 GHz)."""
    import torch
    with torch.cuda.stream(stream):
        torch.cuda._sleep(int(ms * 2e6))


def test_reset_is_seen_from_any_stream(searched):
    import torch
    p, e, stream, _, _ = searched
    labels = torch.as_tensor(_View(p.device_view().d_labels, p.nodes), device="cuda")
    other = torch.cuda.Stream()
    _busy(stream, 100)
    N.check(p.Reset(e.GetFrontierType(), 1.3))
    with torch.cuda.stream(other):
        seen = labels.clone()
    other.synchronize()
    assert bool((seen == -1).all())


def test_reset_then_search_on_another_stream(searched):
    import torch
    p, e, stream, src, want = searched
    _busy(stream, 100)
    N.check(p.Reset(e.GetFrontierType(), 1.3))
    p.set_stream(torch.cuda.Stream().cuda_stream)
    N.check(e.EnactFusedSearch(p, src))
    assert oracle.compare_labels(p.labels(), want) == -1


def test_change_of_stream_does_not_wait(searched):
    import torch
    p, e, stream, src, want = searched
    N.check(p.Reset(e.GetFrontierType(), 1.3))
    N.check(e.EnactFusedSearch(p, src))
    _busy(stream, 500)
    t0 = time.perf_counter()
    p.set_stream(None)
    took = time.perf_counter() - t0
    stream.synchronize()
    assert took < 0.1
    assert oracle.compare_labels(p.labels(), want) == -1


def test_change_of_stream_beside_a_capture(searched):
    import torch
    p, e, stream, src, want = searched
    N.check(p.Reset(e.GetFrontierType(), 1.3))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        graph.capture_begin()
        N.check(e.EnactFusedSearch(p, src))
        p.set_stream(None)
        graph.capture_end()
    p.set_stream(stream.cuda_stream)
    with torch.cuda.stream(stream):
        graph.replay()
    assert oracle.compare_labels(p.labels(), want) == -1


def test_change_from_a_destroyed_stream(searched):
    import torch
    p, e, _, src, want = searched
    raw = C.c_void_p()
    assert int(torch.cuda.cudart().cudaStreamCreate(C.addressof(raw))) == 0
    p.set_stream(raw.value)
    N.check(p.Reset(e.GetFrontierType(), 1.3))
    N.check(e.EnactFusedSearch(p, src))
    assert oracle.compare_labels(p.labels(), want) == -1  # (waits for the stream)
    assert int(torch.cuda.cudart().cudaStreamDestroy(raw.value)) == 0
    p.set_stream(None)
    N.check(p.Reset(e.GetFrontierType(), 1.3))
    N.check(e.EnactFusedSearch(p, src))
    assert oracle.compare_labels(p.labels(), want) == -1
