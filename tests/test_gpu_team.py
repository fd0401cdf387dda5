"""The Krylov solves that run as one resident kernel against the
per-iteration kernels (which event timing selects): the same systems at the
edges of the teams' ranges -- one block, a partly filled last block, 16-block
clusters, the first sizes of a grid per component and of one grid for three.

Tolerances, derived before the first run: with three inner iterations both
paths do the same arithmetic per element and differ by the rounding of the
reductions only (about 1e-16 times the square root of the terms, through three
iterations: 1e-12); solved to 1e-12 both satisfy |r| <= 1e-12 |b|, and the
fields follow within a condition-number factor of about 1e3: 1e-9."""
import dataclasses

import numpy as np
import pytest

import _cases as K

pytestmark = pytest.mark.gpu

# cells: 1 block; 513 rows (2 blocks); a ragged 4-block cluster; full and ragged 16-block clusters at 1, 2, 3 and 4
# rows per thread; the first grid per component; three rows per thread of it; one grid for three components
SMALL = [(4, 3, 2), (8, 8, 8), (27, 19, 1), (20, 10, 7), (32, 16, 16), (41, 20, 10), (40, 20, 20), (45, 20, 20)]
LARGE = [(50, 30, 20), (64, 32, 16), (33, 32, 32), (60, 40, 37), (106, 31, 32)]


def rel(a, b):
    n = np.linalg.norm(b)
    return np.linalg.norm(a - b) / (n if n > 0 else 1.0)


def both(dims, ctl, upload=None):
    got = []
    for timed in (False, True):
        mesh, case = K.channel_product(*dims, L=(2.0, 0.1, 0.1))
        if upload:
            upload(case, mesh)
        case.kernel_timing(timed)
        r = case.solve(ctl)
        got.append((case.download(), r, case.last_timing()[1]))
    return got


def controls(p, **over):
    import chuanflow_b200 as cf
    return cf.SimpleControls(**{**dict(max_iterations=2, relax_u=0.9, relax_p=0.03, p_relax_start=0.002,
                                       non_orth_correctors=1, linear_tol=1e-12, linear_max_iter=3000, nu=1e-3,
                                       p_preconditioner=p), **over})


@pytest.mark.parametrize("p", ["Jacobi", "DIC"])
@pytest.mark.parametrize("dims", SMALL + LARGE)
def test_three_iterations_agree(dims, p):
    (a, ra, na), (b, rb, nb) = both(dims, controls(p, linear_max_iter=3, max_iterations=1))
    assert ra.u_inner_iterations == rb.u_inner_iterations and ra.p_inner_iterations == rb.p_inner_iterations
    assert na < nb  # the solves were single kernels
    for x, y in zip(a, b):
        assert rel(x, y) < 1e-12


@pytest.mark.parametrize("p", ["Jacobi", "DIC"])
@pytest.mark.parametrize("dims", [SMALL[0], SMALL[2], SMALL[4], SMALL[6], LARGE[0], LARGE[2]])
def test_converged_fields_agree(dims, p):
    (a, _, _), (b, _, _) = both(dims, controls(p))
    for x, y in zip(a, b):
        assert rel(x, y) < 1e-9


def test_no_iterations_and_converged_start():
    for ctl in (controls("Jacobi", linear_max_iter=0, max_iterations=1), controls("DIC", linear_tol=1e30)):
        (a, ra, _), (b, rb, _) = both((20, 10, 7), ctl)
        assert ra.u_inner_iterations == rb.u_inner_iterations == 0 and ra.p_inner_iterations == rb.p_inner_iterations == 0
        for x, y in zip(a, b):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("dims", [(20, 10, 7), (40, 20, 20), (33, 32, 32)])
def test_nan_ends_the_solves_as_before(dims):
    def spoil(case, mesh):
        U, p, phi = case.download()
        p[mesh.n_cells // 2] = np.nan
        case.upload(U, p, phi)

    (a, ra, _), (b, rb, _) = both(dims, controls("Jacobi", max_iterations=1, linear_max_iter=40), spoil)
    assert ra.diverged and rb.diverged
    assert ra.u_inner_iterations == rb.u_inner_iterations and ra.p_inner_iterations == rb.p_inner_iterations
    for x, y in zip(a, b):
        assert np.array_equal(np.isnan(x), np.isnan(y))


def test_teams_are_reproducible_and_independent_of_the_schedule():
    """The same solve twice gives the same bits, and a detail block gives them
    under every schedule of a batch."""
    import chuanflow_b200 as cf
    from chuanflow_b200 import meshgen
    runs = [both((40, 20, 20), controls("DIC", max_iterations=1))[0][0] for _ in range(2)]
    for x, y in zip(*runs):
        assert np.array_equal(x, y)
    out = []
    for sched in ((1, 0), (2, 1), (0, -1)):
        cases = []
        for cells, aspect in ((700, 6.0), (18000, 8.0)):
            c = cf.SimpleCase(meshgen.channel_block(cells, aspect))
            c.detail_setup("parabolic")
            cases.append(c)
        b = cf.Batch(cases)
        b.set_schedule(*sched)
        ctl = dataclasses.replace(controls("DIC", max_iterations=1), nu=1e-4)
        r, _ = b.loss([0.002, 0.001], ctl)
        out.append(([x["dp_pa"] for x in r], [c.download() for c in cases]))
    for dp, fields in out[1:]:
        assert dp == out[0][0]
        for f, g in zip(fields, out[0][1]):
            assert all(np.array_equal(x, y) for x, y in zip(f, g))
