"""Programmatic dependent launch of the AMG loops changes when kernels start,
not what they compute: with it off, on by size and on at every size the same
bits.  Sizes on either side of the fused flexible-CG passes' line are left to
CHUANFLOW_PDL=1, which takes every size."""
import numpy as np
import pytest

import _cases as K

pytestmark = pytest.mark.gpu


def runs(monkeypatch, once):
    out = []
    for v in ("0", None, "1"):
        if v is None:
            monkeypatch.delenv("CHUANFLOW_PDL", raising=False)
        else:
            monkeypatch.setenv("CHUANFLOW_PDL", v)
        out.append(once())
    for got in out[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(got, out[0]))


@pytest.mark.parametrize("dims", [(11, 10, 9), (33, 32, 31), (62, 60, 58)])
def test_poisson(monkeypatch, dims):
    import chuanflow_b200 as cf

    def once():
        mesh = cf.PolyMesh.block((0, 0, 0), (1, 1, 1), dims)
        mesh.jitter_interior(0.1, 3)
        case = cf.SimpleCase(mesh)
        case.poisson_setup(ref_cell=0)
        b = np.random.default_rng(2).standard_normal(mesh.n_cells)
        b -= b.mean()
        x, rep = case.poisson_solve(b, "fcg_amg", tol=1e-11)
        assert rep["converged"]
        return x, rep["inner_iterations"]

    runs(monkeypatch, once)


@pytest.mark.parametrize("dims", [(48, 14, 13), (110, 44, 43)])
def test_momentum_and_pressure(monkeypatch, dims):
    import chuanflow_b200 as cf

    def once():
        mesh, case = K.channel_product(*dims, L=(2.0, 0.1, 0.1))
        case.init_flux((0.1, 0.0, 0.0))
        r = case.solve(cf.SimpleControls(max_iterations=2, relax_u=0.9, relax_p=0.03, p_relax_start=0.002,
                                         non_orth_correctors=1, linear_tol=1e-11, linear_max_iter=2000, nu=1e-3,
                                         p_preconditioner="AMG", u_preconditioner="AMG"))
        return (*case.download(), r.u_inner_iterations, r.p_inner_iterations)

    runs(monkeypatch, once)


def test_piso(monkeypatch):
    import chuanflow_b200 as cf

    def once():
        mesh, case = K.channel_product(40, 20, 20, L=(2.0, 0.1, 0.1))
        case.init_flux((0.1, 0.0, 0.0))
        case.piso_step(cf.PisoControls(dt=1e-3, nu=1e-3, linear_tol=1e-10, p_preconditioner="AMG"))
        return case.download()

    runs(monkeypatch, once)
