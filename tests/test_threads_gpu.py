"""Searches of the same kernel from several threads, each with a handle and a stream
of its own and a policy that asks for a different amount of shared memory."""
import threading

import pytest

import oracle
from back40computing_b200 import (CsrGraph, CsrProblem, BuildRmatGraph, sample_sources, search, EXPAND_CONTRACT,
                                  DIRECTION_OPTIMIZING)
from back40computing_b200 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("strategy,mode", [(EXPAND_CONTRACT, N.ENACT_FUSED), (DIRECTION_OPTIMIZING, N.ENACT_FUSED),
                                           (EXPAND_CONTRACT, N.ENACT_ITERATIVE)])
def test_policies_side_by_side(strategy, mode):
    g = CsrGraph()
    BuildRmatGraph(1 << 10, 1 << 13, g, True, 0.57, 0.19, 0.19, seed=1, permute=True)
    src = int(sample_sources(g, 1, seed=2)[0])
    want = oracle.bfs(g.row_offsets, g.column_indices, src)[0]
    wrong = []

    def work(knobs):
        p = CsrProblem.from_graph(g)
        pol = N.Policy()
        pol.threads, pol.ctas_per_sm = 512, 1
        for name, x in knobs.items():
            setattr(pol, name, x)
        try:
            for _ in range(300):
                if oracle.compare_labels(search(p, src, strategy=strategy, mode=mode, policy=pol, max_grid_size=16),
                                         want) != -1:
                    wrong.append((knobs, "labels"))
                    return
        except N.B40cError as e:
            wrong.append((knobs, str(e)))
        finally:
            p.Destroy()

    threads = [threading.Thread(target=work, args=(k,)) for k in
               ({}, {"history_cull": 1}, {"warp_contract": -1}, {"bottom_up_prefetch": 1, "warp_bottom_up": -1})]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
