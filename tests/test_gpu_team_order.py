"""A one-kernel solve adds its sums in the order of the per-iteration kernels
that run one row per thread, so both give the same bits -- also where a thread
of the final sum holds four partials (more than 768 groups of 256 rows)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(58, 58, 58), (64, 56, 55), (64, 64, 64)])  # 763, 770 and 1,024 groups
def test_jacobi_cg_same_bits(monkeypatch, dims):
    import chuanflow_b200 as cf
    monkeypatch.setenv("CHUANFLOW_ROW_BLOCKS_PER_SM", "7")  # a thread for every row
    out = []
    for timed in (False, True):  # event timing selects the per-iteration kernels
        mesh = cf.PolyMesh.block((0, 0, 0), (1, 1, 1), dims)
        mesh.jitter_interior(0.1, 3)
        case = cf.SimpleCase(mesh)
        case.poisson_setup(ref_cell=0)
        case.kernel_timing(timed)
        b = np.random.default_rng(4).standard_normal(mesh.n_cells)
        x, rep = case.poisson_solve(b - b.mean(), "jacobi64", tol=1e-30, max_iter=25)
        assert rep["inner_iterations"] == 25
        out.append(x)
    assert np.array_equal(*out)
