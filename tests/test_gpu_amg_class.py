"""The class of the momentum operator that chooses the sweeps of its V-cycles:
from nearly symmetric to convection alone, and a NaN anywhere counts as the
worst, also in a row that its thread follows with others (systems above one
wave of the row grid); the coarsest inverse then refuses the operator."""
import ctypes as C

import numpy as np
import pytest

import _cases as K

pytestmark = pytest.mark.gpu


def momentum_class(dims, nu, spoil=None, L=(2.0, 0.1, 0.1), **mesh_args):
    import chuanflow_b200 as cf
    mesh, case = K.channel_product(*dims, L=L, **mesh_args)
    case.init_flux((0.1, 0.0, 0.0))
    if spoil is not None:
        U, p, phi = case.download()
        phi[spoil] = np.nan
        case.upload(U, p, phi)
    ctl = cf.SimpleControls(max_iterations=1, relax_u=1.0, relax_p=0.03, p_relax_start=0.002, linear_tol=1e-8,
                            linear_max_iter=4, nu=nu, p_preconditioner="AMG", u_preconditioner="AMG")
    if spoil is None:
        case.solve(ctl)
    else:
        with pytest.raises(cf.CfgError, match="singular coarsest operator"):
            case.solve(ctl)
    out = C.c_int32(-1)
    assert cf.lib().cfg_amg_momentum_class(case._h, C.byref(out)) == 0
    return out.value


def test_class_follows_the_convection():
    got = [momentum_class((48, 14, 13), nu) for nu in (1e-2, 1e-6)]
    assert got == [0, 2]


@pytest.mark.parametrize("theta,skew_class", [(0.45, 0), (0.55, 1), (0.65, 1), (0.75, 2), (0.85, 2)])
def test_class_of_a_known_theta(theta, skew_class):
    """Uniform flow u through cubes of side h: an interior row has two faces
    with |a_ij - a_ji| = u h^2 and the diagonal 6 nu h + u h^2; the other rows
    less flux or more diffusion."""
    u, h = 0.1, 0.1
    nu = u * h * (1 - theta) / (6 * theta)
    assert momentum_class((20, 10, 10), nu, L=(2.0, 1.0, 1.0), jitter=0) == skew_class


@pytest.mark.parametrize("face", [0, 1000])
@pytest.mark.parametrize("dims", [(48, 14, 13), (120, 37, 36)])
def test_nan_is_the_worst_class(dims, face):
    assert momentum_class(dims, 1e-2) == 0
    assert momentum_class(dims, 1e-2, face) == 2
