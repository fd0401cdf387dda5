"""The last aggregated level and the coarsest solve, one block per vector for
small levels and one cluster per vector above 2,048 entries, against the numpy
restatement, on either side of that line (rows that eight blocks do not
divide among them, too).

Tolerance, derived before the first run: the FP32 conditioning of one V-cycle
grows as the cells' number to the 2/3; 5.9e-4 at 444k tets gives 1.5e-4 at
55k, taken as 3e-4, and under 6e-5 at 12k and less, taken as 1e-4.  The three
vectors of a three-component cycle equal single cycles bit for bit."""
import numpy as np
import pytest

import _amg_ref as R
from test_gpu_amg import _system, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,tol,large", [(5, 1e-4, False), (8, 1e-4, True), (12, 1e-4, False), (20, 3e-4, True)])
def test_last_level_matches_restatement(n, tol, large):
    mesh, case, A, _ = _system(n=n, seed=6)
    case.poisson_amg_setup()
    H = R.Hierarchy(A)
    assert (H.levels[-1]["A"].nnz > 2048) == large
    r3 = np.random.default_rng(8).standard_normal((3, mesh.n_cells))
    r3 -= r3.mean(axis=1, keepdims=True)
    z3 = case.poisson_amg_apply3(r3)
    for q in range(3):
        assert np.array_equal(z3[q], case.poisson_amg_apply(r3[q]))
        assert rel(z3[q], H.apply(r3[q]).astype(np.float64)) < tol
