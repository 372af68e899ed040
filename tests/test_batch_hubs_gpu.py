"""Batched searches on graphs whose longest lists are searched in segments spread
over the grid: degrees at the limits (2048 kept whole, 2049 in three segments, an
exact and a ragged number of segments), hubs reached late, by sources that join a
running batch and in CTA-wide pull levels, with both ways of taking frontier
slots, against the oracle."""
import numpy as np
import pytest

import oracle
from back40computing_b200 import CsrGraph, CsrProblem
from back40computing_b200 import _native as N

pytestmark = pytest.mark.gpu

DEGREES = (2047, 2048, 2049, 3072, 5000, 9001)


def _hubs(tail=0):
    """One hub per degree, its leaves shared with the next hub's, a chain of 6
    before the first hub, a uniform random part that keeps levels dense and a
    chain of `tail` vertices behind the last leaf."""
    rng = np.random.default_rng(3)
    leaves = 12000
    n = 6 + len(DEGREES) + leaves + tail
    u, v = [np.arange(6)], [np.arange(1, 7)]
    for i, d in enumerate(DEGREES):
        u.append(np.full(d, 6 + i))
        v.append(6 + len(DEGREES) + rng.choice(leaves, d, replace=False))
    u.append(6 + len(DEGREES) + rng.integers(0, leaves, 30000))
    v.append(6 + len(DEGREES) + rng.integers(0, leaves, 30000))
    u.append(np.arange(n - tail - 1, n - 1))
    v.append(np.arange(n - tail, n))
    u, v = np.concatenate(u), np.concatenate(v)
    g = CsrGraph()
    g.FromCoo(np.concatenate([u, v]), np.concatenate([v, u]), n)
    return g


@pytest.mark.parametrize("k", [1, 33, 64])
@pytest.mark.parametrize("knobs", [{}, {"threads": 128}, {"threads": 256, "warp_contract": -1},
                                   {"threads": 512, "bottom_up_alpha": 1 << 20},
                                   {"bottom_up_hub_probes": -1, "bottom_up_alpha": 1 << 20},
                                   {"warp_contract": -1, "queue_allocation": 1},
                                   {"warp_contract": -1, "queue_allocation": 1, "bottom_up_alpha": 1 << 20}])
def test_segmented_lists(k, knobs):
    g = _hubs()
    p = CsrProblem.from_graph(g)
    pol = N.Policy()
    for name, x in knobs.items():
        setattr(pol, name, x)
    rng = np.random.default_rng(k)
    srcs = np.concatenate([[0, 6], rng.integers(0, g.nodes, 62)])[:k].astype(np.int32)
    limits = np.where(np.arange(k) % 5 == 4, 3, -1).astype(np.int32)
    p.msbfs(srcs, depth_limits=limits, policy=pol)
    depths = p.msbfs_depths()
    for slot in range(k):
        want, _ = oracle.bfs(g.row_offsets, g.column_indices, int(srcs[slot]))
        if limits[slot] >= 0:
            want = np.where(want > limits[slot], -1, want)
        assert oracle.compare_labels(p.labels_of(slot), want) == -1, f"slot {slot}"
        assert depths[slot] == int(want.max()) + 1
    p.Destroy()


@pytest.mark.parametrize("warp_contract", [1, -1])
def test_many_warps_claim_one_hub(warp_contract):
    """A hub in 196 segments, first reached by 64 sources at once: the segments'
    warps read and set the hub's word while the others do."""
    leaves = 200_000
    hub = np.zeros(leaves, np.int64)
    leaf = np.arange(1, leaves + 1)
    g = CsrGraph()
    g.FromCoo(np.concatenate([hub, leaf]), np.concatenate([leaf, hub]), leaves + 1)
    p = CsrProblem.from_graph(g)
    pol = N.Policy()
    pol.bottom_up_alpha, pol.warp_contract, pol.bottom_up_hub_probes = 1 << 20, warp_contract, -1
    for run in range(20):
        srcs = np.random.default_rng(run).choice(leaf, 64, replace=False).astype(np.int32)
        p.msbfs(srcs, policy=pol)
        assert (p.msbfs_depths() == 3).all()
        for slot in (0, 31, 63):
            want = np.full(leaves + 1, 2, np.int32)
            want[[0, srcs[slot]]] = 1, 0
            assert np.array_equal(p.labels_of(slot), want)
    p.Destroy()


@pytest.mark.parametrize("knobs", [{}, {"queue_allocation": 1}, {"warp_contract": -1},
                                   {"warp_contract": -1, "queue_allocation": 1}])
def test_joins_beside_segmented_lists(knobs):
    """Sources that join while every level pulls: their frontier entries go beside
    the segments' and the chunks' or warps', whichever way those took their slots.
    The chain keeps the batch running while the requests arrive."""
    g = _hubs(tail=3000)
    p = CsrProblem.from_graph(g)
    pol = N.Policy()
    pol.bottom_up_alpha = 1 << 20
    for name, x in knobs.items():
        setattr(pol, name, x)
    p.msbfs(np.arange(12, dtype=np.int32), policy=pol)  # label rows for 12 slots
    base = np.array([g.nodes - 1, 0, 9], np.int32)
    joins = [0, 6, 11, 8, 500, 11000, g.nodes - 1500, 7]
    p.msbfs(base, policy=pol)
    for j, src in enumerate(joins):
        p.msbfs_join(3 + j, src)
    taken, depths = p.msbfs_joined()
    assert taken > 0
    for slot, src in enumerate([*base, *joins[:taken]]):
        want, depth = oracle.bfs(g.row_offsets, g.column_indices, int(src))
        assert oracle.compare_labels(p.labels_of(slot), want) == -1, f"slot {slot}"
        assert depths[slot] == depth
    p.Destroy()
