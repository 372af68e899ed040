"""COO -> CSR on the GPU (b40c_coo_to_csr_device) against the host
conversion, which keeps each row in input order like CsrGraph::FromCoo."""
import ctypes as C

import numpy as np
import pytest

import oracle
from back40computing_b200 import CsrProblem, search, B40cError, DIRECTION_OPTIMIZING
from back40computing_b200 import _native as N

pytestmark = pytest.mark.gpu


def _host_csr(n, rows, cols):
    order = np.argsort(rows, kind="stable")
    ro = np.zeros(n + 1, np.int64)
    np.add.at(ro, rows.astype(np.int64) + 1, 1)
    return np.cumsum(ro).astype(np.int32), cols[order].astype(np.int32)


def _device(n, rows, cols):
    import torch
    d_r = torch.from_numpy(rows.astype(np.int32)).cuda()
    d_c = torch.from_numpy(cols.astype(np.int32)).cuda()
    d_ro = torch.empty(n + 1, dtype=torch.int32, device="cuda")
    d_ci = torch.empty(max(rows.size, 1), dtype=torch.int32, device="cuda")
    s = torch.cuda.current_stream()
    rc = N.lib().b40c_coo_to_csr_device(C.c_void_p(d_r.data_ptr()), C.c_void_p(d_c.data_ptr()), n, rows.size,
                                        C.c_void_p(d_ro.data_ptr()), C.c_void_p(d_ci.data_ptr()),
                                        C.c_void_p(s.cuda_stream))
    return rc, d_ro.cpu().numpy(), d_ci.cpu().numpy()[:rows.size]


@pytest.mark.parametrize("n,m", [(1, 0), (1, 5), (200, 5000), (1 << 12, 1 << 16), (1 << 20, 1 << 22),
                                 (1 << 25, 1 << 20), ((1 << 24) + 3, 3 * (1 << 20) + 17)])
def test_matches_stable_host_conversion(n, m):
    rng = np.random.default_rng(n + m)
    # skewed rows (many duplicates) so runs cross tiles and passes
    rows = (rng.pareto(1.5, m) * n / 50).astype(np.int64) % n
    cols = rng.integers(0, n, m)
    rc, ro, ci = _device(n, rows, cols)
    assert rc == 0
    want_ro, want_ci = _host_csr(n, rows, cols)
    assert np.array_equal(ro, want_ro)
    assert np.array_equal(ci, want_ci)


# one, two and three digits of every width class; tiles of 2048 and 16384 edges
# with full and ragged ends, the switch between them (148 SMs x 16384 edges); rows
# all equal, all different mod 32, and uniform
@pytest.mark.parametrize("n,m", [(31, 2047), (32, 2048), (33, 2049), (2048, 6143), (2049, 70001), (1 << 22, 4097),
                                 ((1 << 22) + 1, 200003), (1000, 148 * 16384 - 1), (5000, 148 * 16384),
                                 (1 << 21, 148 * 16384 + 1)])
@pytest.mark.parametrize("kind", ["uniform", "one-row", "cyclic"])
def test_radix_pass_edges(n, m, kind):
    rng = np.random.default_rng(m)
    rows = {"uniform": rng.integers(0, n, m), "one-row": np.full(m, n - 1), "cyclic": np.arange(m) % n}[kind]
    cols = rng.integers(0, n, m)
    rc, ro, ci = _device(n, rows, cols)
    assert rc == 0
    want_ro, want_ci = _host_csr(n, rows, cols)
    assert np.array_equal(ro, want_ro)
    assert np.array_equal(ci, want_ci)


@pytest.mark.parametrize("n", [200, 1500, 70000])
def test_columns_converted_in_place(n):
    """The column array may take the result: every pass but the last writes elsewhere."""
    import torch
    rng = np.random.default_rng(n)
    rows, cols = rng.integers(0, n, 100001), rng.integers(0, n, 100001)
    d_r = torch.from_numpy(rows.astype(np.int32)).cuda()
    d_c = torch.from_numpy(cols.astype(np.int32)).cuda()
    d_ro = torch.empty(n + 1, dtype=torch.int32, device="cuda")
    assert N.lib().b40c_coo_to_csr_device(C.c_void_p(d_r.data_ptr()), C.c_void_p(d_c.data_ptr()), n, rows.size,
                                          C.c_void_p(d_ro.data_ptr()), C.c_void_p(d_c.data_ptr()),
                                          C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    want_ro, want_ci = _host_csr(n, rows, cols)
    assert np.array_equal(d_ro.cpu().numpy(), want_ro)
    assert np.array_equal(d_c.cpu().numpy(), want_ci)


def test_conversions_from_several_threads():
    """Digits of different widths at the same time, in short and in long tiles: the
    kernels' shared memory differs with the width."""
    import threading
    import torch
    cases = []
    for n, m in ((2048, 100_000), (40, 100_000), (1 << 22, 70_000), (2048, 148 * 16384), (40, 148 * 16384)):
        rng = np.random.default_rng(n + m)
        rows, cols = rng.integers(0, n, m), rng.integers(0, n, m)
        cases.append((n, rows, cols, _host_csr(n, rows, cols)))
    wrong = []

    def work(n, rows, cols, want):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(60):
                rc, ro, ci = _device(n, rows, cols)
                if rc != 0 or not np.array_equal(ro, want[0]) or not np.array_equal(ci, want[1]):
                    wrong.append((n, rows.size, rc))
                    return

    threads = [threading.Thread(target=work, args=c) for c in cases]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def _in_use():
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, total = torch.cuda.mem_get_info()
    return total - free


def test_conversion_memory_is_bounded_and_given_back():
    """60 M edges need 720 MB of workspace: at most 512 MB stay when the call returns
    (mapped in steps of 32 MB), nothing after the release."""
    import torch
    n, m = 1 << 20, 60_000_000
    gen = torch.Generator(device="cuda").manual_seed(1)
    _device(n, np.arange(1000), np.arange(1000))
    assert N.lib().b40c_coo_release_memory(0) == 0
    base = _in_use()
    r = torch.randint(0, n, (m,), generator=gen, device="cuda", dtype=torch.int32)
    ro = torch.empty(n + 1, dtype=torch.int32, device="cuda")
    ci = torch.empty(m, dtype=torch.int32, device="cuda")
    assert N.lib().b40c_coo_to_csr_device(r.data_ptr(), r.data_ptr(), n, m, ro.data_ptr(), ci.data_ptr(),
                                          torch.cuda.current_stream().cuda_stream) == 0
    del r, ro, ci
    assert _in_use() - base <= (512 + 32) << 20
    assert N.lib().b40c_coo_release_memory(0) == 0
    assert _in_use() - base <= 8 << 20
    assert N.lib().b40c_coo_release_memory(99) == N.ERROR_INVALID_VALUE


def test_problem_from_coo_keeps_no_conversion_memory():
    rng = np.random.default_rng(4)
    n, m = 100_000, 16_000_000
    rows, cols = rng.integers(0, n, m), rng.integers(0, n, m)
    CsrProblem.from_coo(rows[:1000], cols[:1000], n).Destroy()
    base = _in_use()
    p = CsrProblem.from_coo(rows, cols, n)
    held = C.c_int64()
    N.check(N.lib().b40c_bfs_problem_device_bytes(p.handle, C.byref(held)))
    assert _in_use() - base <= held.value + (32 << 20)  # (192 MB of workspace)
    p.Destroy()


def test_rejects_ids_out_of_range():
    rows = np.array([0, 1, 5], np.int32)
    cols = np.array([1, 2, 0], np.int32)
    rc, _, _ = _device(5, rows, cols)
    assert rc == N.ERROR_INVALID_VALUE


def test_problem_from_coo_searches_like_oracle():
    from back40computing_b200 import CsrGraph, BuildRmatGraph
    g = CsrGraph()
    BuildRmatGraph(1 << 14, 1 << 17, g, True, 0.57, 0.19, 0.19, seed=2, permute=True)
    rows = np.repeat(np.arange(g.nodes, dtype=np.int32), np.diff(g.row_offsets))
    perm = np.random.default_rng(0).permutation(rows.size)
    r, c = rows[perm], g.column_indices[perm]
    p = CsrProblem.from_coo(r, c, g.nodes)
    want_ro, want_ci = _host_csr(g.nodes, r, c)
    for s in (0, 17, 4242):
        got = search(p, s, strategy=DIRECTION_OPTIMIZING)
        want, _ = oracle.bfs(want_ro, want_ci, s)
        assert oracle.compare_labels(got, want) == -1
    with pytest.raises(B40cError):
        CsrProblem.from_coo(np.array([0, 3]), np.array([1, 1]), 3)
