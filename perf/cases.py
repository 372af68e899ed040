"""Performance cases: what users of this library run, through its public entry points.

Each case is a dict of plain values:

* ``kind``: ``search`` (one single-source search), ``batch`` (up to 64 sources
  together), ``served`` (a burst of queries to the query server), ``coo``
  (device COO -> CSR conversion) or ``noalloc`` (the allocation-free search);
* the graph: ``graph`` is ``rmat`` (``scale``, ``degree``), ``random``
  (``nodes``, ``degree``), ``grid2d`` / ``grid3d`` (``width``); ``directed``
  keeps the generated edges as they are instead of adding their reversals;
* for searches: ``strategy``, ``mode`` (``fused``, ``iterative``, ``graph``),
  ``pred`` (predecessors instead of distances), ``policy`` (``default`` or the
  autotuner's ``tuned`` one), ``api`` (``search``: the one-call search that
  resets, searches and returns host labels; ``enact``: an enactor on a
  resident problem, results left on the device) and ``depth`` (limit, -1 none);
* ``k`` sources of a batch, ``queries`` of a served burst, ``nodes`` and
  ``edges`` of a conversion.

Graph shapes are the generators' of this library (R-MAT a=.57 b=.19 c=.19 with
permuted ids, uniform random, lattices with self-loops); the random ones are
generated on the GPU from the seed.
"""
import math

import numpy as np
import torch

from back40computing_b200 import CsrGraph, CsrProblem, BuildGrid2dGraph, BuildGrid3dGraph, autotune, search
from back40computing_b200 import _native as N
from back40computing_b200.bfs import ENACTORS
from back40computing_b200.server import BfsServer

STRATEGIES = {"expand-contract": N.EXPAND_CONTRACT, "contract-expand": N.CONTRACT_EXPAND, "two-phase": N.TWO_PHASE,
              "hybrid": N.HYBRID, "direction-optimizing": N.DIRECTION_OPTIMIZING}
MODES = {"fused": N.ENACT_FUSED, "iterative": N.ENACT_ITERATIVE, "graph": N.ENACT_GRAPH}


def _search(graph, strategy, **more):
    c = {"kind": "search", "graph": graph, "strategy": strategy, "mode": "fused", "pred": False, "policy": "default",
         "api": "enact", "depth": -1, "directed": False}
    c.update(more)
    return c


def listed():
    return [
        # the smallest call: one search on a small graph, host labels back (latency and launches)
        dict(_search("random", "expand-contract", nodes=2000, degree=4, api="search"), name="small-call"),
        # an ordinary single query on a resident social-network-like graph, library defaults
        dict(_search("rmat", "direction-optimizing", scale=16, degree=16), name="rmat16-do"),
        # the reference's drop-in enactors on ordinary graphs, called without a policy
        dict(_search("rmat", "expand-contract", scale=20, degree=16), name="rmat20-ec"),
        dict(_search("random", "hybrid", nodes=1000003, degree=8), name="random1m-hybrid"),
        # BFS trees: reachability through predecessors
        dict(_search("rmat", "expand-contract", scale=20, degree=16, pred=True), name="rmat20-ec-pred"),
        # the headline workload: R-MAT 22, tuned direction-optimizing search
        dict(_search("rmat", "direction-optimizing", scale=22, degree=16, policy="tuned"), name="rmat22-do"),
        # the largest call: the reference's default strategy on the same graph
        dict(_search("rmat", "contract-expand", scale=22, degree=16), name="rmat22-ce"),
        # high-diameter meshes: thousands of small levels, and hundreds of wide ones of an odd width
        dict(_search("grid2d", "expand-contract", width=1000, policy="tuned"), name="grid2d1000-ec"),
        dict(_search("grid3d", "direction-optimizing", width=201), name="grid3d201-do"),
        # 64 sources searched together (all-pairs style analytics, full server batches)
        {"name": "random21-batch64", "kind": "batch", "graph": "random", "nodes": 1 << 21, "degree": 16, "k": 64,
         "directed": False},
        # a burst of queries over two resident graphs: full and ragged batches through the server
        {"name": "served-burst", "kind": "served", "graph": "rmat", "scale": 16, "degree": 16, "queries": 300,
         "directed": False},
        # building a graph: device edge list to CSR
        {"name": "coo-16m", "kind": "coo", "nodes": 1 << 20, "edges": 16 << 20},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_graph(rng, small=False):
    directed = rng.random() < 0.15
    degree = rng.choice([3, 5, 8, 12, 16])
    if rng.random() < 0.5:
        return {"graph": "rmat", "scale": rng.randint(9, 18 if small else 21), "degree": degree, "directed": directed}
    return {"graph": "random", "nodes": _log(rng, 700, 250000 if small else 2500000), "degree": degree,
            "directed": directed}


def draw(rng):
    kind = rng.choice(["search"] * 6 + ["lattice"] * 2 + ["batch"] * 2 + ["coo", "noalloc"])
    if kind == "coo":
        return {"kind": "coo", "nodes": _log(rng, 500, 3000000), "edges": _log(rng, 1000, 30000000)}
    if kind == "noalloc":
        n = _log(rng, 500, 250000)
        return {"kind": "noalloc", "graph": "random", "nodes": n, "degree": rng.choice([2, 4, 8]), "directed": False}
    if kind == "batch":
        c = {"kind": "batch", "k": rng.randint(1, 64)}
        c.update(_draw_graph(rng, small=rng.random() < 0.5))
        if c["graph"] == "rmat":
            c["scale"] = min(c["scale"], 20)
        else:
            c["nodes"] = min(c["nodes"], 1500000)
        return c
    strategy = rng.choice(list(STRATEGIES))
    more = {"mode": rng.choice(["fused"] * 6 + ["iterative", "graph"]), "pred": rng.random() < 0.2,
            "policy": rng.choice(["default", "default", "tuned"]),
            "api": "search" if rng.random() < 0.25 else "enact"}
    if more["api"] == "search" and rng.random() < 0.3:
        more["depth"] = rng.randint(1, 6)
    if kind == "lattice":
        if rng.random() < 0.5:
            return _search("grid2d", strategy, width=_log(rng, 15, 1000), **more)
        return _search("grid3d", strategy, width=_log(rng, 7, 200), **more)
    g = _draw_graph(rng)
    return _search(g.pop("graph"), strategy, **more, **g)


# ---- graphs ---------------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _edge_list(case, seed):
    """(rows, cols, nodes): int32 edge list of a random graph on the GPU."""
    gen = _generator(seed)
    if case["graph"] == "rmat":
        scale, nodes = case["scale"], 1 << case["scale"]
        m = nodes * case["degree"]
        u = torch.empty(m, dtype=torch.int32, device="cuda")
        v = torch.empty(m, dtype=torch.int32, device="cuda")
        for b in range(0, m, 1 << 24):
            e = min(m, b + (1 << 24))
            x = torch.zeros(e - b, dtype=torch.int32, device="cuda")
            y = torch.zeros(e - b, dtype=torch.int32, device="cuda")
            for _ in range(scale):
                r = torch.rand(e - b, generator=gen, device="cuda")
                x = 2 * x + (r >= 0.76)
                y = 2 * y + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
            u[b:e], v[b:e] = x, y
        perm = torch.randperm(nodes, generator=gen, device="cuda").to(torch.int32)
        u, v = perm[u.long()], perm[v.long()]
    else:
        nodes = case["nodes"]
        m = nodes * case["degree"]
        u = torch.randint(0, nodes, (m,), generator=gen, device="cuda", dtype=torch.int32)
        v = torch.randint(0, nodes, (m,), generator=gen, device="cuda", dtype=torch.int32)
    if not case["directed"]:
        u, v = torch.cat([u, v]), torch.cat([v, u])
    return u, v, nodes


def _to_csr(rows, cols, nodes):
    """Device CSR of an edge list, rows in input order."""
    srt, idx = torch.sort(rows, stable=True)
    ci = cols[idx]
    ro = torch.searchsorted(srt, torch.arange(nodes + 1, device="cuda", dtype=torch.int32)).to(torch.int32)
    return ro, ci


def _lattice_nodes(case):
    return case["width"] ** (2 if case["graph"] == "grid2d" else 3)


def _sources(ro, count, seed):
    """`count` seeded sources among the vertices with edges (host array of row offsets)."""
    ok = np.nonzero(np.diff(ro) > 0)[0]
    return np.random.default_rng(int(seed)).choice(ok, size=count, replace=count > ok.size).astype(np.int32)


def _host_graph(case, seed):
    """CsrGraph of a case (host arrays), and its row offsets."""
    if case["graph"] in ("grid2d", "grid3d"):
        g = CsrGraph()
        (BuildGrid2dGraph if case["graph"] == "grid2d" else BuildGrid3dGraph)(case["width"], g)
        return g
    rows, cols, nodes = _edge_list(case, seed)
    ro, ci = _to_csr(rows, cols, nodes)
    return CsrGraph.from_arrays(ro.cpu().numpy(), ci.cpu().numpy())


def _served_cases(case):
    """The graphs a served burst is spread over: the case's own and a uniform one a quarter its size."""
    n = 1 << case["scale"]
    return [case, {"graph": "random", "nodes": n // 4 + 1, "degree": case["degree"], "directed": case["directed"]}]


_stream = []


def _torch_stream():
    """The one torch stream the program's searches run on, in order with its torch operations."""
    if not _stream:
        _stream.append(torch.cuda.Stream())
    return _stream[0]


class _Device:
    """Wraps a device pointer of the library for torch.as_tensor (no copy)."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": tuple(shape), "typestr": "<i4",
                                         "version": 3}


def _view(ptr, shape, owner):
    return torch.as_tensor(_Device(ptr, shape, owner), device="cuda")


# ---- the cases ------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "coo":
        gen = _generator(seed)
        n, m = case["nodes"], case["edges"]
        return {"kind": kind, "n": n, "m": m,
                "rows": torch.randint(0, n, (m,), generator=gen, device="cuda", dtype=torch.int32),
                "cols": torch.randint(0, n, (m,), generator=gen, device="cuda", dtype=torch.int32),
                "ro": torch.empty(n + 1, dtype=torch.int32, device="cuda"),
                "ci": torch.empty(m, dtype=torch.int32, device="cuda")}
    if kind == "served":
        server = BfsServer(memory_budget_bytes=8 << 30)
        ids, graphs, srcs = [], [], []
        for i, c in enumerate(_served_cases(case)):
            g = _host_graph(c, seed + 1000 * i)
            ids.append(server.add_tuned_graph(g))
            srcs.append(_sources(g.row_offsets, case["queries"], seed + i))
        q = np.arange(case["queries"])
        which = (q % 3 == 2).astype(np.int32)  # two thirds of the queries to the larger graph
        return {"kind": kind, "server": server, "graph_ids": np.asarray(ids, np.int32)[which],
                "sources": np.where(which == 0, srcs[0], srcs[1]).astype(np.int32)}
    if kind == "noalloc":
        rows, cols, n = _edge_list(case, seed)
        ro, ci = _to_csr(rows, cols, n)
        return {"kind": kind, "ro": ro, "ci": ci, "n": n, "m": int(ci.numel()),
                "src": int(_sources(ro.cpu().numpy(), 1, seed)[0]),
                "labels": torch.empty(n, dtype=torch.int32, device="cuda")}
    g = _host_graph(case, seed)
    state = {"kind": kind, "n": g.nodes}
    if kind == "batch":
        state["sources"] = _sources(g.row_offsets, case["k"], seed)
        state["policy"] = autotune.policy_for(g, "batched")
        p = state["problem"] = CsrProblem.from_graph(g)
        p.set_stream(_torch_stream().cuda_stream)
        N.check(p.Reset(N.VERTEX_FRONTIERS, 1.3), "Reset")
        return state
    strategy = STRATEGIES[case["strategy"]]
    state["src"] = int(_sources(g.row_offsets, 1, seed)[0])
    policy = None
    if case["policy"] == "tuned":
        policy = autotune.policy_for(g, "direction-optimizing" if strategy == N.DIRECTION_OPTIMIZING
                                     else "expand-contract")
        if case["pred"] and policy is not None and policy.threads == 512:
            policy.threads = 256
    if policy is not None and strategy in (N.CONTRACT_EXPAND, N.TWO_PHASE, N.HYBRID):
        policy = None  # the autotuner has no policies for the edge-frontier strategies
    p = state["problem"] = CsrProblem.from_graph(g, mark_predecessors=case["pred"])
    p.set_stream(_torch_stream().cuda_stream)
    state.update(policy=policy, strategy=strategy, mode=MODES[case["mode"]], depth=case["depth"], api=case["api"],
                 pred=case["pred"])
    enactor = state["enactor"] = ENACTORS[strategy](policy=policy)
    N.check(p.Reset(enactor.GetFrontierType(), 1.3), "Reset")
    state["labels"] = _view(p.device_view().d_labels, (g.nodes,), p)
    state["call"] = {N.ENACT_FUSED: getattr(enactor, "EnactFusedSearch"),
                     N.ENACT_ITERATIVE: enactor.EnactIterativeSearch,
                     N.ENACT_GRAPH: enactor.EnactGraphSearch}[state["mode"]]
    return state


def run(state):
    kind = state["kind"]
    if kind == "coo":
        N.check(N.lib().b40c_coo_to_csr_device(state["rows"].data_ptr(), state["cols"].data_ptr(), state["n"],
                                               state["m"], state["ro"].data_ptr(), state["ci"].data_ptr(),
                                               torch.cuda.current_stream().cuda_stream), "coo_to_csr")
        return state["ro"], state["ci"]
    if kind == "noalloc":
        N.check(N.lib().b40c_bfs_search_noalloc(state["ro"].data_ptr(), state["ci"].data_ptr(), state["n"], state["m"],
                                                state["src"], state["labels"].data_ptr(),
                                                torch.cuda.current_stream().cuda_stream), "search_noalloc")
        return state["labels"]
    if kind == "served":
        server = state["server"]
        tickets = server.submit_many(state["graph_ids"], state["sources"])
        server.drain()
        r = server.results(int(tickets[0]), tickets.size)
        return {"status": r["status"].copy(), "search_depth": r["search_depth"].copy()}
    p = state["problem"]
    if kind == "batch":
        p.msbfs(state["sources"], policy=state["policy"])
        if "labels" not in state:  # the label rows are allocated by the first batch
            ptr, k = N.C.c_void_p(), N.C.c_int32(0)
            N.check(N.lib().b40c_msbfs_device_labels(p.handle, N.C.byref(ptr), N.C.byref(k)), "device_labels")
            state["labels"] = _view(ptr.value, (k.value, state["n"]), p)
        return state["labels"]
    if state["api"] == "search":
        out = search(p, state["src"], strategy=state["strategy"], mode=state["mode"], depth_limit=state["depth"],
                     policy=state["policy"])
        # several parents can be right: what a predecessor search answers for certain is who was reached
        return np.minimum(out, 0) if state["pred"] else out
    N.check(state["call"](p, state["src"]), "Enact")
    if state["pred"]:
        with torch.cuda.stream(_torch_stream()):
            return state["labels"].clamp(max=0)
    return state["labels"]


def _edges(case):
    if case["graph"] == "grid2d":
        w = case["width"]
        return 5 * w * w - 4 * w
    if case["graph"] == "grid3d":
        w = case["width"]
        return 7 * w ** 3 - 6 * w * w
    n = (1 << case["scale"]) if case["graph"] == "rmat" else case["nodes"]
    return n * case["degree"] * (1 if case["directed"] else 2)


def _nodes(case):
    if case["graph"] in ("grid2d", "grid3d"):
        return _lattice_nodes(case)
    return (1 << case["scale"]) if case["graph"] == "rmat" else case["nodes"]


def work(case):
    """Bytes one pass reads and writes at least once: the CSR and the labels."""
    kind = case["kind"]
    if kind == "coo":
        return {"bytes": 12 * case["edges"] + 4 * (case["nodes"] + 1), "flops": 0}
    if kind == "served":
        return {"bytes": sum(4 * _edges(c) + 4 * _nodes(c) for c in _served_cases(case)) + 4 * case["queries"],
                "flops": 0}
    rows = case["k"] if kind == "batch" else 1
    return {"bytes": 4 * _edges(case) + 4 * (_nodes(case) + 1) + 4 * rows * _nodes(case), "flops": 0}


# ---- the answers, from plain torch and numpy --------------------------------------------

def _lattice_labels(case, src):
    w, d = case["width"], 2 if case["graph"] == "grid2d" else 3
    v = torch.arange(w ** d, device="cuda")
    out = torch.zeros_like(v)
    for _ in range(d):
        out += (v % w - src % w).abs()
        v, src = v // w, src // w
    return out


def _levels(ro, ci, src, limit=-1):
    """Distances from src, level by level, on the GPU (-1 unreached or beyond the limit)."""
    labels = torch.full((ro.numel() - 1,), -1, dtype=torch.int64, device="cuda")
    labels[src] = 0
    f = torch.tensor([src], device="cuda")
    level = 0
    while f.numel() and (limit < 0 or level < limit):
        start = ro[f].long()
        deg = ro[f + 1].long() - start
        first = torch.cumsum(deg, 0) - deg
        e = torch.repeat_interleave(start - first, deg)
        nb = ci[e + torch.arange(e.numel(), device="cuda")].long()
        nb = nb[labels[nb] < 0]
        level += 1
        labels[nb] = level
        f = torch.unique(nb)
    return labels


def exact(case, seed):
    kind = case["kind"]
    if kind == "coo":
        s = prepare(case, seed)
        return _to_csr(s["rows"], s["cols"], s["n"])
    if kind == "served":
        depth = []
        for i, c in enumerate(_served_cases(case)):
            ro, ci = _to_csr(*_edge_list(c, seed + 1000 * i))
            depth.append([int(_levels(ro, ci, int(s)).max()) + 1
                          for s in _sources(ro.cpu().numpy(), case["queries"], seed + i)])
        q = np.arange(case["queries"])
        return {"status": np.zeros(q.size, np.int64),
                "search_depth": np.where(q % 3 == 2, depth[1], depth[0]).astype(np.int64)}
    if case["graph"] in ("grid2d", "grid3d"):
        # every vertex of a lattice has edges: a source is drawn from all of them
        src = int(_sources(np.arange(_lattice_nodes(case) + 1), 1, seed)[0])
        out = _lattice_labels(case, src)
        if case["depth"] >= 0:
            out[out > case["depth"]] = -1
    else:
        ro, ci = _to_csr(*_edge_list(case, seed))
        h_ro = ro.cpu().numpy()
        if kind == "batch":
            return torch.stack([_levels(ro, ci, int(s)) for s in _sources(h_ro, case["k"], seed)])
        src = int(_sources(h_ro, 1, seed)[0])
        out = _levels(ro, ci, src, case.get("depth", -1))
    if case.get("pred"):
        out = out.clamp(max=0)
        out[src] = -2
    return out
