"""A wait inside a one-kernel solve that runs out: an error status, the caller's
data as they were, and the next solve as if nothing had happened.  The limit of
one cycle makes the first waits run out; every block then leaves the kernel."""
import contextlib
import ctypes as C

import numpy as np
import pytest

import _cases as K
from test_gpu_team import controls
from test_gpu_team_csr import matrix

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def limit(name, cycles):
    import chuanflow_b200 as cf
    assert getattr(cf.lib(), name)(C.c_int64(cycles)) == 0
    try:
        yield
    finally:
        getattr(cf.lib(), name)(C.c_int64(0))


def wait_limit(cycles):
    return limit("cfg_solver_wait_limit", cycles)


def static_solve(n, width, seed, max_iter=2000):
    """cfg_pcg_solve_static as a function of nothing: (status, x, report, the exact solution)."""
    import torch
    import chuanflow_b200 as cf
    rs, cols, vals, sol, b = matrix(n, width, np.random.default_rng(seed), True)
    dev = [torch.from_numpy(a).cuda() for a in (rs.astype(np.int32), cols.astype(np.int32), vals, b)]

    def solve():
        out = torch.full((n,), 0.25, dtype=torch.float64, device="cuda")
        rep = cf._capi._Report()
        torch.cuda.synchronize()
        rc = cf.lib().cfg_pcg_solve_static(C.c_int32(0), C.c_int64(n), *[C.c_void_p(t.data_ptr()) for t in dev],
                                           C.c_void_p(out.data_ptr()), C.c_double(1e-12), C.c_int32(max_iter), None,
                                           C.byref(rep))
        return rc, out.cpu().numpy(), rep

    return solve, sol


@pytest.mark.parametrize("p", ["Jacobi", "DIC"])
@pytest.mark.parametrize("dims", [(60, 40, 37), (106, 31, 32)])  # a grid per component; one grid for three
def test_context_reports_once_and_solves_again(dims, p):
    import chuanflow_b200 as cf
    ctl = controls(p, max_iterations=1, linear_max_iter=5)
    _, fresh = K.channel_product(*dims, L=(2.0, 0.1, 0.1))
    start = fresh.download()
    fresh.solve(ctl)
    _, case = K.channel_product(*dims, L=(2.0, 0.1, 0.1))
    with wait_limit(1), pytest.raises(cf.CfgError, match="ran out"):
        case.solve(ctl)
    case.upload(*start)
    r = case.solve(ctl)
    assert not r.diverged
    assert all(np.array_equal(a, b) for a, b in zip(case.download(), fresh.download()))


@pytest.mark.parametrize("method", [0, 1])
def test_host_csr_leaves_x(method):
    import chuanflow_b200 as cf
    n = 75000
    rs, cols, vals, sol, b = matrix(n, 7, np.random.default_rng(3), method == 0)
    x = np.full(n, 3.5)
    rep = cf._capi._Report()

    def solve():
        return cf.lib().cfg_sparse_solve(None, C.c_int32(0), C.c_int64(n), *[a.ctypes.data_as(C.c_void_p) for a in
                                         (rs, cols, vals, b, x)], C.c_double(1e-12), C.c_int32(500),
                                         C.c_int32(method), C.byref(rep))

    with wait_limit(1):
        assert solve() == 2 and np.all(x == 3.5)
    assert solve() == 0 and rep.converged
    assert np.linalg.norm(x - sol) < 1e-9 * np.linalg.norm(sol)


@pytest.mark.parametrize("n", [32769, 75000, 200000, 262144])
def test_static_pcg_without_all_its_blocks(n):
    """Blocks that are not all there in time leave, and the per-iteration
    kernels give the same bits."""
    solve, sol = static_solve(n, 7, 5)
    rc, x, rep = solve()
    assert rc == 0 and rep.converged and np.linalg.norm(x - sol) < 1e-9 * np.linalg.norm(sol)
    with limit("cfg_solver_start_limit", 1):
        rc, y, other = solve()
    assert rc == 0 and other.iterations == rep.iterations and np.array_equal(x, y)
    rc, y, _ = solve()
    assert rc == 0 and np.array_equal(x, y)


@pytest.mark.parametrize("n", [32769, 262144])
def test_static_pcg_wait(n):
    solve, sol = static_solve(n, 7, 6)
    with wait_limit(1):
        assert solve()[0] == 2
    rc, x, rep = solve()
    assert rc == 0 and rep.converged and np.linalg.norm(x - sol) < 1e-9 * np.linalg.norm(sol)


@pytest.mark.parametrize("n", [2, 300, 513, 32768, 32769, 262144])
def test_static_pcg_one_long_row(n):
    """A single row of more than seven entries anywhere sends the whole system
    to the per-iteration kernels."""
    import scipy.sparse as sp
    import torch
    import chuanflow_b200 as cf
    for at in {0, n // 2, n - 1}:
        k = [j for j in range(max(0, at - 6), min(n, at + 7)) if j != at]
        d = np.full(n, 20.0)
        w = np.full(len(k), -1.0)
        A = sp.csr_matrix((np.r_[d, w, w], (np.r_[np.arange(n), np.full(len(k), at), k],
                                            np.r_[np.arange(n), k, np.full(len(k), at)])), (n, n))
        sol = np.random.default_rng(at).standard_normal(n)
        dev = [torch.from_numpy(a).cuda() for a in (A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data, A @ sol)]
        out = torch.zeros(n, dtype=torch.float64, device="cuda")
        rep = cf._capi._Report()
        torch.cuda.synchronize()
        rc = cf.lib().cfg_pcg_solve_static(C.c_int32(0), C.c_int64(n), *[C.c_void_p(t.data_ptr()) for t in dev],
                                           C.c_void_p(out.data_ptr()), C.c_double(1e-12), C.c_int32(200), None,
                                           C.byref(rep))
        assert rc == 0 and rep.converged and np.linalg.norm(out.cpu().numpy() - sol) < 1e-9 * np.linalg.norm(sol)
