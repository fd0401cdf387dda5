"""Systems that take a grid of blocks when they solve alone, and kernels per
iteration when other contexts solve on the device too: the same bits either
way, by the limit that forces the kernels, and with contexts at once on several
threads."""
import ctypes as C
import threading

import numpy as np
import pytest

import _cases as K
from test_gpu_team import controls

pytestmark = pytest.mark.gpu

# a grid per component at 1, 2 and 4 rows per thread; one grid for three; the largest of it
SIZES = [(33, 32, 32), (60, 40, 37), (70, 38, 37), (106, 31, 32), (64, 48, 49)]


def grid_solves(n):
    import chuanflow_b200 as cf
    assert cf.lib().cfg_solver_grid_solves(C.c_int32(n)) == 0


@pytest.fixture(autouse=True)
def restore():
    yield
    grid_solves(-1)


def channel(dims, ctl):
    _, case = K.channel_product(*dims, L=(2.0, 0.1, 0.1))
    case.solve(ctl)
    return (*case.download(), case.last_timing()[1])


@pytest.mark.parametrize("p", ["Jacobi", "DIC"])
@pytest.mark.parametrize("dims", SIZES)
def test_channel_same_bits(dims, p):
    ctl = controls(p, max_iterations=1, linear_max_iter=60)
    *alone, few = channel(dims, ctl)
    grid_solves(0)
    *shared, many = channel(dims, ctl)
    assert few < many
    assert all(np.array_equal(a, b) for a, b in zip(alone, shared))


@pytest.mark.parametrize("method", ["jacobi64", "dic64"])
@pytest.mark.parametrize("dims", [(33, 32, 32), (64, 56, 55), (64, 64, 64)])
def test_poisson_same_bits(dims, method):
    import chuanflow_b200 as cf
    out = []
    for n in (-1, 0):
        grid_solves(n)
        mesh = cf.PolyMesh.block((0, 0, 0), (1, 1, 1), dims)
        mesh.jitter_interior(0.1, 3)
        case = cf.SimpleCase(mesh)
        case.poisson_setup(ref_cell=0)
        b = np.random.default_rng(4).standard_normal(mesh.n_cells)
        out.append(case.poisson_solve(b - b.mean(), method, tol=1e-30, max_iter=25)[0])
    assert np.array_equal(*out)


def test_contexts_at_once_same_bits():
    dims, ctl = (45, 28, 28), controls("DIC", max_iterations=2, linear_max_iter=60)
    *alone, _ = channel(dims, ctl)
    got = [None] * 4
    threads = [threading.Thread(target=lambda i=i: got.__setitem__(i, channel(dims, ctl))) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for *fields, _ in got:
        assert all(np.array_equal(a, b) for a, b in zip(alone, fields))
