"""An infinity reaches only the rows coupled to it, also in the one-kernel
solves, whose rows all have the same number of slots: the initial residual of a
start with one infinite value is infinite, not a NaN (every row meets it once,
so no row subtracts infinities)."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_team_csr import matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 300, 600, 5000, 40000])
@pytest.mark.parametrize("at", ["first", "last"])
def test_infinite_start(n, at):
    import torch
    import chuanflow_b200 as cf
    rs, cols, vals, sol, b = matrix(n, 5, np.random.default_rng(n), True)
    x0 = np.zeros(n)
    x0[0 if at == "first" else n - 1] = np.inf
    for solve in (cf.solve_cg, cf.solve_bicgstab):
        x, rep = solve(rs, cols, vals, b, x0, 1e-10, 0)
        assert rep.initial_residual == np.inf and rep.iterations == 0 and np.array_equal(x, x0)
        _, rep = solve(rs, cols, vals, b, x0, 1e-10, 20)
        assert rep.initial_residual == np.inf and not rep.converged
    dev = [torch.from_numpy(a).cuda() for a in (rs.astype(np.int32), cols.astype(np.int32), vals, b)]
    out, rep = torch.from_numpy(x0).cuda(), cf._capi._Report()
    torch.cuda.synchronize()
    assert cf.lib().cfg_pcg_solve_static(C.c_int32(0), C.c_int64(n), *[C.c_void_p(t.data_ptr()) for t in dev],
                                         C.c_void_p(out.data_ptr()), C.c_double(1e-10), C.c_int32(0), None,
                                         C.byref(rep)) == 0
    assert rep.initial_residual == np.inf
