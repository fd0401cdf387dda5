"""Sweeps of the pressure V-cycle on a hierarchy aggregated by strength: weighted
while the couplings left out still count, single ones when they are hardly any
(cells ten and twenty times longer than wide), by the iterations of the same
flexible CG in numpy, which differ between the two.  One iteration may go
either way with the rounding of an FP32 cycle."""
import numpy as np
import pytest
import scipy.sparse as sp

import _amg_cycle_ref as W
import _amg_ref as R
import _cases as K
from test_amg_ref import fcg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length,theta,skew_class", [(0.1, 0.25, 0), (0.5, 0.25, 0), (2.0, 0.25, 2)])
def test_iterations_tell_the_sweeps(length, theta, skew_class):
    cells, L = (20, 18, 17), (length, 0.1, 0.1)
    mesh, case = K.channel_product(*cells, jitter=0.1, seed=7, L=L)
    if theta:
        case.amg_strength(theta)
    case.poisson_setup()
    rs, cols, vals = K.channel_case(*cells, jitter=0.1, seed=7, L=L).pressure_csr(np.ones(mesh.n_faces))
    A = sp.csr_matrix((vals, cols, rs), shape=(mesh.n_cells, mesh.n_cells))
    H = R.Hierarchy(A, theta)
    b = np.random.default_rng(1).standard_normal(mesh.n_cells)
    want = {c: fcg(A, b, W.Cycle(H, c, np.float32), 1e-10)[1] for c in (0, 2)}
    assert want[2] > want[0] + 2
    _, rep = case.poisson_solve(b, "fcg_amg", tol=1e-10)
    assert abs(rep["inner_iterations"] - want[skew_class]) <= 1
