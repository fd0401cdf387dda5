"""The V-cycle that the solvers apply -- several weighted sweeps on the coarse
levels -- against its numpy restatement, for one vector and for three, in every
class of sweeps: ends in the dense solve after level kernels (last aggregated
level above 1,024 rows), in the one-block and in the clustered last level, and
first coarse levels on either side of the SELL-32 and three-sweep rule and of the four-sweep one
(the largest system).

Tolerance, from the restatement alone: the device and the FP32 restatement add
in different orders with the same operators, so each is off the same cycle in
FP64 by rounding of about the same size; the device may be off by eight times
the most that the restatement is in any class (one near-singular operator, whose
slowest mode carries the rounding of all three)."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

import _amg_cycle_ref as W
import _amg_ref as R
import _cases as K
from test_gpu_amg import _system, rel

pytestmark = pytest.mark.gpu

KERNEL_ROWS, CLUSTER_ENTRIES = 1024, 2048


def tets(n):
    _, case, A, _ = _system(n=n, seed=6)
    return case, A


def channel(cells):
    mesh, case = K.channel_product(*cells, jitter=0.1, seed=7, L=(2.0, 0.1, 0.1))
    case.poisson_setup()
    rs, cols, vals = K.channel_case(*cells, jitter=0.1, seed=7, L=(2.0, 0.1, 0.1)).pressure_csr(np.ones(mesh.n_faces))
    return case, sp.csr_matrix((vals, cols, rs), shape=(mesh.n_cells, mesh.n_cells))


def cycle(case, r, skew_class):
    import chuanflow_b200 as cf
    r = np.ascontiguousarray(r, np.float64)
    z = np.zeros_like(r)
    rc = cf.lib().cfg_poisson_amg_cycle(case._h, r.ctypes.data_as(C.c_void_p), z.ctypes.data_as(C.c_void_p),
                                        C.c_int32(1 if r.ndim == 1 else 3), C.c_int32(skew_class))
    assert rc == 0
    return z


# system, how it ends, whether the first coarse level is large
SYSTEMS = [(tets, 3, "dense", False), (tets, 5, "block", False), (tets, 8, "cluster", False), (tets, 10, "dense", False),
           (tets, 13, "block", False), (tets, 20, "cluster", False), (tets, 40, "block", True),
           (channel, (68, 66, 65), "dense", True), (channel, (80, 78, 76), "dense", True),
           (channel, (100, 92, 92), "cluster", True)]


@pytest.mark.parametrize("make,size,end,large", SYSTEMS, ids=lambda v: getattr(v, "__name__", str(v)))
def test_solver_cycle_matches_restatement(make, size, end, large):
    case, A = make(size)
    H = R.Hierarchy(A)
    last = H.levels[-1]["A"]
    held = len(H.levels) > 1 and last.shape[0] <= KERNEL_ROWS
    assert (("cluster" if last.nnz > CLUSTER_ENTRIES else "block") if held else "dense") == end
    assert (H.rows[1] >= W.SELL_MIN_ROWS) == large
    r = np.random.default_rng(12).standard_normal((3, A.shape[0]))
    r -= r.mean(axis=1, keepdims=True)
    exact = [W.Cycle(H, c, np.float64)(r[0]) for c in range(3)]
    tol = 8 * max(rel(W.Cycle(H, c, np.float32)(r[0]).astype(np.float64), exact[c]) for c in range(3))
    assert tol < 5e-3  # the classes' cycles differ by 0.2 and more
    for skew_class in range(3):
        z3 = cycle(case, r, skew_class)
        assert rel(z3[0], exact[skew_class]) < tol, (skew_class, tol)
        for q in range(3):
            assert np.array_equal(cycle(case, r[q], skew_class), z3[q])
    assert np.array_equal(z3[0], case.poisson_amg_apply(r[0]))  # class 2
