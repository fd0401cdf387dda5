"""The CSR entry points as one resident kernel, against a dense solve in
NumPy: sizes around the teams' edges, rows of one entry, rows too long for the
resident layout (the per-iteration kernels then run), a missing diagonal entry
order and unsorted columns.

Tolerance, derived before the first run: the matrices have condition numbers
below 1e3 and both solvers stop at |r|inf <= 1e-12 |b|inf: 1e-9."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def matrix(n, width, rng, symmetric):
    """Banded with `width` entries per interior row, columns in random order."""
    off = [k for k in (1, 2, 5, 11, 23) if k < n][:max(0, (width - 1) // 2)]
    rows, cols, vals = [np.arange(n)], [np.arange(n)], [np.full(n, 1.0 + 2.2 * len(off))]
    for k in off:
        i = np.arange(n - k)
        w = -rng.uniform(0.5, 1.0, n - k)
        rows += [i, i + k]
        cols += [i + k, i]
        vals += [w, w if symmetric else w * rng.uniform(0.4, 1.0, n - k)]
    rows, cols, vals = (np.concatenate(a) for a in (rows, cols, vals))
    order = np.lexsort((rng.random(rows.size), rows))
    rows, cols, vals = rows[order], cols[order], vals[order]
    rs = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(rows, minlength=n), out=rs[1:])
    x = rng.standard_normal(n)
    return rs, cols.astype(np.int64), vals, x, np.bincount(rows, vals * x[cols], n)


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


SIZES = [1, 2, 255, 257, 513, 4097, 32768, 32769, 75000]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("width", [1, 7, 11])
def test_host_csr(n, width):
    import chuanflow_b200 as cf
    rng = np.random.default_rng(n + width)
    for solve, sym in ((cf.solve_cg, True), (cf.solve_bicgstab, False)):
        rs, cols, vals, x, b = matrix(n, width, rng, sym)
        got, rep = solve(rs, cols, vals, b, np.zeros(n), 1e-12, 2000)
        assert rep.converged and rel(got, x) < 1e-9
        again, rep2 = solve(rs, cols, vals, b, got, 1e-6, 2000)
        assert rep2.converged and rep2.iterations == 0 and np.array_equal(again, got)


@pytest.mark.parametrize("n", SIZES + [262144])
@pytest.mark.parametrize("width", [3, 7, 11])
def test_device_csr(n, width):
    import torch
    import chuanflow_b200 as cf
    rng = np.random.default_rng(7 * n + width)
    rs, cols, vals, x, b = matrix(n, width, rng, True)
    dev = [torch.from_numpy(a).cuda() for a in (rs.astype(np.int32), cols.astype(np.int32), vals, b)]
    out = torch.zeros(n, dtype=torch.float64, device="cuda")
    rep = cf._capi._Report()
    torch.cuda.synchronize()
    for _ in range(2):  # the static scratch serves one call after another
        out.zero_()
        torch.cuda.synchronize()
        rc = cf.lib().cfg_pcg_solve_static(C.c_int32(0), C.c_int64(n), *[C.c_void_p(t.data_ptr()) for t in dev],
                                           C.c_void_p(out.data_ptr()), C.c_double(1e-12), C.c_int32(2000), None,
                                           C.byref(rep))
        assert rc == 0 and rep.converged
        assert rel(out.cpu().numpy(), x) < 1e-9
