"""The V-cycles of the solvers, whose coarse levels take several weighted
sweeps: hierarchies that end in the dense solve alone, in the fused last
level, and with a first coarse level on either side of the SELL-32 rule; the
momentum solve at operators from nearly symmetric to convection alone (each
class of sweeps).

Tolerance, derived before the first run: both solvers stop at |r|inf <= 1e-11
|b|inf; the solutions follow within the conditioning of these meshes, about
1e4 at most, so they agree within 1e-7."""
import numpy as np
import pytest

import _cases as K

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("dims", [(7, 6, 5), (11, 10, 9), (24, 21, 20), (64, 61, 60), (66, 64, 63)])
def test_poisson_amg_matches_dic(dims):
    """From one coarse (dense) level to a SELL first coarse level."""
    import chuanflow_b200 as cf
    mesh = cf.PolyMesh.block((0, 0, 0), (1, 1, 1), dims)
    mesh.jitter_interior(0.1, 3)
    case = cf.SimpleCase(mesh)
    case.poisson_setup(ref_cell=0)
    b = np.random.default_rng(2).standard_normal(mesh.n_cells)
    b -= b.mean()
    x, rep = case.poisson_solve(b, "fcg_amg", tol=1e-11)
    y, _ = case.poisson_solve(b, "dic64", tol=1e-11)
    assert rep["outer_iterations"] == 1 and rep["inner_iterations"] < 120
    assert rel(x, y) < 1e-7


@pytest.mark.parametrize("nu", [1e-3, 3e-5, 6e-6])
@pytest.mark.parametrize("theta", [0.0, 0.25])
def test_momentum_amg_matches_jacobi(nu, theta):
    import chuanflow_b200 as cf
    out = []
    for u in ("Jacobi", "AMG"):
        mesh, case = K.channel_product(48, 14, 13, L=(2.0, 0.1, 0.1))
        case.init_flux((0.1, 0.0, 0.0))
        if theta:
            case.amg_strength(theta)
        r = case.solve(cf.SimpleControls(max_iterations=2, relax_u=0.9, relax_p=0.03, p_relax_start=0.002,
                                         non_orth_correctors=1, linear_tol=1e-11, linear_max_iter=4000, nu=nu,
                                         p_preconditioner="AMG", u_preconditioner=u))
        assert not r.diverged
        out.append((case.download(), r.u_inner_iterations))
    assert out[1][1] < out[0][1]
    for x, y in zip(out[1][0], out[0][0]):
        assert rel(x, y) < 1e-7
