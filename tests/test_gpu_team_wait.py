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
def wait_limit(cycles):
    import chuanflow_b200 as cf
    assert cf.lib().cfg_solver_wait_limit(C.c_int64(cycles)) == 0
    try:
        yield
    finally:
        cf.lib().cfg_solver_wait_limit(C.c_int64(0))


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
