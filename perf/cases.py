"""The work users of this library have it do, as timed cases.

Every case goes through the public entry points from host data to host
results, as the library is called: fields and right-hand sides are uploaded,
the solve runs on the device, the fields come back.  `listed()` holds the
named cases, `draw(rng)` one more of the same ranges, `prepare` what a program
has in hand before the call (mesh, context, boundary conditions, pinned host
fields), `run` one pass, `work` the bytes and operations one pass cannot do
without and `exact` the 64-bit results where plain numpy gives them.

The linear solves run to tolerances one or two digits below the tests' 1e-10:
the fields are then those of the equations, not of the iterate a looser test
happens to stop at.  The starting fields are a developed flow with a seeded
disturbance, the meshes are jittered from the seed.
"""
import ctypes as C
import math

import numpy as np
import torch

import chuanflow_b200 as cf
from chuanflow_b200 import meshgen

SIDES = ["xmin", "xmax", "ymin", "ymax", "zmin", "zmax"]
CHANNEL = dict(zip(SIDES, zip(["inlet", "outlet", "bottom", "top", "front", "back"],
                              ["inlet", "outlet", "wall", "wall", "wall", "wall"])))
CAVITY = dict(zip(SIDES, zip(["left", "right", "bottom", "lid", "front", "back"], ["wall"] * 6)))
TOL = 1e-12  # |r|inf / |b|inf of the flow solvers' linear solves and of the CSR solves (the Poisson ones: 3e-12, |r|2 / |b|2)
TET_SEED = 3  # the number of tetrahedra depends on their points: their mesh is fixed, the solutions are seeded


def listed():
    return [
        # the smallest flow solve the tests and smoke runs make: a jittered lid-driven cavity, the reference's own
        # solvers and a pinned pressure cell; launches and latency are all there is
        dict(name="cavity 1.3k", kind="simple", case="cavity", nx=12, ny=11, nz=10, u="Jacobi", p="Jacobi",
             div="upwind", grad="corrected", non_orth=1, iters=4, theta=0.0),
        # the reference's verification channel (40 x 20 x 20) with its default solvers and corrector count
        dict(name="channel 16k", kind="simple", case="channel", nx=40, ny=20, nz=20, u="Jacobi", p="Jacobi",
             div="upwind", grad="corrected", non_orth=2, iters=3, theta=0.0),
        # an everyday ragged mesh with the second-order convection and least-squares gradients, FP64 throughout
        # (Jacobi momentum, multicolour DIC pressure)
        dict(name="channel 131k DIC", kind="simple", case="channel", nx=203, ny=27, nz=24, u="Jacobi", p="DIC",
             div="linearUpwind", grad="leastSquares", non_orth=1, iters=1, theta=0.0),
        # the same family with both multigrid preconditioners, blended convection
        dict(name="channel 262k AMG", kind="simple", case="channel", nx=256, ny=32, nz=32, u="AMG", p="AMG",
             div="blend", grad="corrected", non_orth=1, iters=1, theta=0.25),
        # the headline workload of the benchmark, one outer iteration
        dict(name="channel 2M AMG", kind="simple", case="channel", nx=512, ny=64, nz=64, u="AMG", p="AMG",
             div="upwind", grad="corrected", non_orth=1, iters=1, theta=0.25),
        # a k-epsilon channel: the model's two scalar equations beside the flow, one outer iteration from saved fields
        dict(name="k-epsilon 23k", kind="rans", nx=63, ny=19, nz=19, model="kEpsilon", p="DIC", iters=1),
        # one implicit-Euler PISO step of a transient run (two correctors, multigrid pressure)
        dict(name="piso 158k AMG", kind="piso", nx=397, ny=99, nz=4, p="AMG"),
        # the pressure-Poisson system on Delaunay tetrahedra, mixed-precision multigrid solve
        dict(name="poisson 55k tets", kind="poisson", mesh="tets", n=20, method="fcg_amg"),
        # the same solve on a 1.2M-cell jittered block
        dict(name="poisson 1.2M hex", kind="poisson", mesh="hex", n=107, method="fcg_amg"),
        # the reference's BiCGStab on a host CSR matrix (upwind convection-diffusion): copies in and out included
        dict(name="csr bicgstab 30k", kind="csr", method="bicgstab", nx=37, ny=29, nz=28),
        # the allocation-free CG on a caller's device matrix, near its 262,144-row limit
        dict(name="device cg 250k", kind="static", nx=63, ny=63, nz=63),
        # one coupling pass over 16 detail blocks (ducts of 2k to 60k cells, the odd small ones k-epsilon) as one graph
        dict(name="16 detail blocks", kind="blocks", n=16, cells_min=2000, cells_max=60000, spec=2024),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["simple", "simple", "simple", "simple", "rans", "piso", "poisson", "poisson", "csr", "static",
                       "blocks"])
    if kind == "simple":
        n = _log_int(rng, 1300, 2_000_000)
        c = dict(kind="simple", div=rng.choice(["upwind", "blend", "linearUpwind"]),
                 grad=rng.choice(["corrected", "leastSquares", "linear"]), non_orth=rng.choice([1, 2]),
                 iters=4 if n < 10_000 else 2 if n < 100_000 else 1)
        if n < 20_000 and rng.random() < 0.3:
            s = n ** (1 / 3)
            return dict(c, case="cavity", nx=int(s) + rng.randint(0, 2), ny=int(s) + rng.randint(0, 1),
                        nz=max(9, int(s) - rng.randint(0, 2)), u="Jacobi", p=rng.choice(["Jacobi", "DIC"]), theta=0.0)
        ny = max(5, int(round((n / 8) ** (1 / 3))) + rng.randint(-1, 1))
        nz = max(5, ny + rng.randint(-1, 1))
        big = n > 150_000
        return dict(c, case="channel", nx=max(8, int(round(n / (ny * nz)))), ny=ny, nz=nz,
                    u="AMG" if big else rng.choice(["Jacobi", "AMG"]),
                    p="AMG" if big else rng.choice(["Jacobi", "DIC", "AMG"]), theta=rng.choice([0.0, 0.25]))
    if kind == "rans":
        ny = _log_int(rng, 5, 24)
        return dict(kind="rans", nx=ny * rng.randint(2, 5) + rng.randint(0, 3), ny=ny, nz=max(4, ny - rng.randint(0, 2)),
                    model=rng.choice(["kEpsilon", "kOmegaSST"]), p=rng.choice(["Jacobi", "DIC"]), iters=1)
    if kind == "piso":
        ny = _log_int(rng, 12, 160)
        return dict(kind="piso", nx=4 * ny + rng.randint(-3, 3), ny=ny, nz=rng.choice([2, 4, 5]),
                    p=rng.choice(["AMG", "AMG", "DIC"]))
    if kind == "poisson":
        if rng.random() < 0.5:
            return dict(kind="poisson", mesh="tets", n=rng.randint(8, 24), method=rng.choice(["fcg_amg", "dic64"]))
        return dict(kind="poisson", mesh="hex", n=_log_int(rng, 16, 107), method=rng.choice(["fcg_amg", "fcg_amg",
                                                                                          "jacobi64"]))
    if kind == "csr":
        n = _log_int(rng, 8, 55)
        return dict(kind="csr", method=rng.choice(["bicgstab", "cg"]), nx=n + rng.randint(0, 3), ny=n,
                    nz=max(3, n - rng.randint(0, 3)))
    if kind == "static":
        n = _log_int(rng, 8, 62)
        return dict(kind="static", nx=n + rng.randint(0, 1), ny=n, nz=max(3, n - rng.randint(0, 2)))
    return dict(kind="blocks", n=rng.randint(3, 16), cells_min=2000, cells_max=_log_int(rng, 8000, 60000),
                spec=rng.randint(1, 10_000))


# ---- inputs -----------------------------------------------------------------

def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


def _modes(xyz, rng, count, kmax):
    """A smooth seeded field on points in the unit box: `count` waves."""
    v = np.zeros(xyz[0].shape)
    for _ in range(count):
        k = rng.uniform(0.5, kmax, 3) * math.pi
        ph = rng.uniform(0, 2 * math.pi, 3)
        v += np.sin(k[0] * xyz[0] + ph[0]) * np.sin(k[1] * xyz[1] + ph[1]) * np.sin(k[2] * xyz[2] + ph[2])
    return v / count


def _lattice(nx, ny, nz):
    """Cell centres of the unjittered block in the unit box, x fastest."""
    z, y, x = np.meshgrid((np.arange(nz) + 0.5) / nz, (np.arange(ny) + 0.5) / ny, (np.arange(nx) + 0.5) / nx,
                          indexing="ij")
    return x.ravel(), y.ravel(), z.ravel()


def _start_fields(case, mesh, dims, lengths, speed, p_drop, rng, cavity=False):
    """Pinned host U, p, phi to start from: the inlet's own profile carried
    through the channel (or the cavity's vortex) and seeded eddies.  The flux
    is a curl on the unjittered lattice, so every cell's net flux is zero, as
    a running solver's nearly is; its boundary part comes from the
    conditions.  U is the lattice cells' mean flux and 0.1% of noise."""
    nx, ny, nz = dims
    h = [lengths[a] / dims[a] for a in range(3)]
    n, ni = mesh.n_cells, mesh.n_internal_faces
    U, p, phi = _pinned(n, 3), _pinned(n), _pinned(mesh.n_faces)
    for f in (U, p, phi):
        f[:] = 0.0
    case.upload(U, p, phi)
    case.init_flux()
    case.download(U, p, phi)
    adr = mesh.addressing()
    owner, nbr = adr["owner"], adr["neighbour"]
    fx, fy, fz = np.zeros((nz, ny, nx + 1)), np.zeros((nz, ny + 1, nx)), np.zeros((nz + 1, ny, nx))
    xn, yn, zn = (np.arange(m + 1) / m for m in dims)           # lattice planes
    xc, yc, zc = ((np.arange(m) + 0.5) / m for m in dims)       # and cell centres
    if cavity:
        psi = 0.2 * speed * lengths[1] / math.pi * np.outer(np.sin(math.pi * yn) ** 2, np.sin(math.pi * xn) ** 2)
        amp, ramp = 0.05, np.sin(math.pi * xn) ** 2
    else:
        start, size = next((q[2], q[3]) for q in mesh.patches if q[0] == "inlet")
        profile = np.zeros((nz, ny))
        cells = owner[start:start + size]
        profile[cells // (nx * ny), (cells // nx) % ny] = -phi[start:start + size]
        fx += profile[:, :, None]
        psi = np.zeros((ny + 1, nx + 1))
        amp, ramp = 0.02, 1.0 - np.exp(-20.0 * xn)
    # two families of eddies, in planes of constant z and of constant y, zero on the walls and at the inlet
    wave = sum(np.sin(rng.uniform(2, 12) * xn + rng.uniform(0, 6.28)) for _ in range(3)) / 3.0
    psi = psi + amp * speed * lengths[1] * np.outer(np.sin(math.pi * yn) ** 2, ramp * wave)
    g = h[2] * (np.sin(math.pi * zc) ** 2 if cavity else 4 * zc * (1 - zc))
    fx += g[:, None, None] * np.diff(psi, axis=0)[None]
    fy -= g[:, None, None] * np.diff(psi, axis=1)[None]
    wave = sum(np.sin(rng.uniform(2, 12) * xn + rng.uniform(0, 6.28)) for _ in range(3)) / 3.0
    chi = amp * speed * lengths[2] * np.outer(np.sin(math.pi * zn) ** 2, ramp * wave)
    g = h[1] * 4 * yc * (1 - yc)
    fx += g[None, :, None] * np.diff(chi, axis=0)[:, None, :]
    fz -= g[None, :, None] * np.diff(chi, axis=1)[:, None, :]
    own = owner[:ni]
    i, j, k = own % nx, (own // nx) % ny, own // (nx * ny)
    step = nbr - own
    phi[:ni] = np.where(step == 1, fx[k, j, i + 1], np.where(step == nx, fy[k, np.minimum(j + 1, ny), i],
                                                             fz[np.minimum(k + 1, nz), j, i]))
    U[:, 0] = ((fx[:, :, 1:] + fx[:, :, :-1]) / (2 * h[1] * h[2])).ravel()
    U[:, 1] = ((fy[:, 1:] + fy[:, :-1]) / (2 * h[0] * h[2])).ravel()
    U[:, 2] = ((fz[1:] + fz[:-1]) / (2 * h[0] * h[1])).ravel()
    U += 0.001 * speed * rng.standard_normal((n, 3))
    x, y, z = _lattice(nx, ny, nz)
    p[:] = p_drop * ((x - 0.5) * (y - 0.5) if cavity else 1.0 - x) + 0.02 * p_drop * _modes((x, y, z), rng, 3, 4.0)
    case.upload(U, p, phi)
    case.init_flux()
    case.download(U, p, phi)
    return U, p, phi


def _channel_bcs(case, mesh, speed):
    for name, _, _, _ in mesh.patches:
        case.set_patch_bc("U", name, "zeroGradient" if name == "outlet" else "fixedValue",
                          (speed, 0, 0) if name == "inlet" else (0, 0, 0))
        case.set_patch_bc("p", name, "fixedValue" if name == "outlet" else "zeroGradient", 0.0)


def _out_fields(mesh):
    return _pinned(mesh.n_cells, 3), _pinned(mesh.n_cells), _pinned(mesh.n_faces)


def _prepare_simple(c, seed):
    rng = np.random.default_rng(seed)
    dims = (c["nx"], c["ny"], c["nz"])
    cavity = c["case"] == "cavity"
    lengths = (1.0, 1.0, 1.0) if cavity else (2.0, 0.1, 0.1)
    mesh = cf.PolyMesh.block((0, 0, 0), lengths, dims, CAVITY if cavity else CHANNEL)
    mesh.jitter_interior(0.1, seed)
    case = cf.SimpleCase(mesh, 0, cf.Schemes(div=c["div"], grad=c["grad"], blend_coeff=0.5))
    if c["theta"]:
        case.amg_strength(c["theta"])
    if cavity:
        for name, _, _, _ in mesh.patches:
            case.set_patch_bc("U", name, "fixedValue", (1.0, 0, 0) if name == "lid" else (0, 0, 0))
            case.set_patch_bc("p", name, "zeroGradient", 0.0)
        ctl = dict(relax_u=0.7, relax_p=0.3, p_relax_start=0.02, nu=0.0025, p_ref_cell=0)
        speed, drop = 1.0, 0.1
    else:
        speed, drop = 0.1 * rng.uniform(0.9, 1.1), 0.007
        _channel_bcs(case, mesh, speed)
        ctl = dict(relax_u=0.9, relax_p=0.03, p_relax_start=0.002, nu=1e-4)
    fields = _start_fields(case, mesh, dims, lengths, speed, drop, rng, cavity)
    controls = cf.SimpleControls(max_iterations=c["iters"], non_orth_correctors=c["non_orth"], linear_tol=TOL,
                                 linear_max_iter=4000, p_preconditioner=c["p"], u_preconditioner=c["u"], **ctl)
    return dict(kind="simple", case=case, fields=fields, controls=controls, out=_out_fields(mesh))


def _run_simple(s):
    s["case"].upload(*s["fields"])
    s["case"].solve(s["controls"])
    U, p, phi = s["case"].download(*s["out"])
    return {"U": U, "p": p, "phi": phi}


def _prepare_rans(c, seed):
    rng = np.random.default_rng(seed)
    dims, lengths = (c["nx"], c["ny"], c["nz"]), (1.0, 0.1, 0.1)
    mesh = cf.PolyMesh.block((0, 0, 0), lengths, dims, CHANNEL)  # orthogonal, as the tests' RANS channel
    case = cf.SimpleCase(mesh)
    speed, nu = 0.5 * rng.uniform(0.9, 1.1), 2.5e-6
    _channel_bcs(case, mesh, speed)
    case.init_flux()
    case.turbulence_setup(c["model"], intensity=0.05, length_scale=-1.0, relaxation=0.7, nu=nu)
    _start_fields(case, mesh, dims, lengths, speed, 0.05, rng)
    saved = cf.Batch([case])
    saved.save()
    controls = cf.SimpleControls(max_iterations=c["iters"], relax_u=0.9, relax_p=0.03, p_relax_start=0.002,
                                 non_orth_correctors=1, linear_tol=TOL, linear_max_iter=4000, nu=nu,
                                 p_preconditioner=c["p"])
    return dict(kind="rans", case=case, saved=saved, controls=controls, out=_out_fields(mesh))


def _run_rans(s):
    s["saved"].restore()
    s["case"].solve(s["controls"])
    U, p, phi = s["case"].download(*s["out"])
    t = s["case"].turbulence_fields()
    return {"U": U, "p": p, "phi": phi, "k": t["k"], "eps": t["eps"], "nut": t["nut"], "nuEff": t["nuEffFace"]}


def _prepare_piso(c, seed):
    rng = np.random.default_rng(seed)
    dims = (c["nx"], c["ny"], c["nz"])
    h = 1.0 / c["ny"]
    lengths = (dims[0] * h, 1.0, dims[2] * h)
    mesh = cf.PolyMesh.block((0, 0, 0), lengths, dims, CHANNEL)
    mesh.jitter_interior(0.1, seed)
    case = cf.SimpleCase(mesh)
    _channel_bcs(case, mesh, 1.0)
    for name in ("front", "back"):  # the extruded sides of a two-dimensional run
        case.set_patch_bc("U", name, "zeroGradient", 0.0)
    fields = _start_fields(case, mesh, dims, lengths, 1.0, 0.5, rng)
    controls = cf.PisoControls(dt=0.5 * h / 2.5, correctors=2, continuity_tol=0.0, linear_tol=TOL, linear_max_iter=8000,
                               non_orth_correctors=0, nu=0.25 / 200, p_preconditioner=c["p"])
    return dict(kind="piso", case=case, fields=fields, controls=controls, out=_out_fields(mesh))


def _run_piso(s):
    s["case"].upload(*s["fields"])
    s["case"].piso_step(s["controls"])
    U, p, phi = s["case"].download(*s["out"])
    return {"U": U, "p": p, "phi": phi}


def _solution(xyz, seed):
    """A smooth field on cell centres in the unit box with a little grid-scale
    noise: a right-hand side formed from it has a solution known exactly."""
    rng = np.random.default_rng(seed + 1)
    return _modes(xyz, rng, 6, 6.0) + 1e-4 * rng.standard_normal(xyz[0].size)


def _poisson_solution(c, seed):
    """On a block's lattice, or on the tetrahedra's centroids (the input
    mesh's points and cells, which the generator gives as plain arrays)."""
    if c["mesh"] == "hex":
        return _solution(_lattice(c["n"] + 1, c["n"], c["n"] - 1), seed)
    pts = meshgen.jittered_lattice(c["n"], 0.1, TET_SEED)
    return _solution(tuple(pts[meshgen.delaunay_tets(pts)].mean(axis=1).T), seed)


def _poisson_mesh(c, seed):
    if c["mesh"] == "tets":
        return meshgen.tet_mesh(c["n"], 0.1, TET_SEED)[0]
    n = c["n"]
    mesh = cf.PolyMesh.block((0, 0, 0), (1, 1, 1), (n + 1, n, n - 1), CAVITY)
    mesh.jitter_interior(0.1, seed)
    return mesh


def _prepare_poisson(c, seed):
    mesh = _poisson_mesh(c, seed)
    case = cf.SimpleCase(mesh)
    case.poisson_setup(ref_cell=0)
    if c["method"] == "fcg_amg":
        case.poisson_amg_setup()
    # b = A x of the orthogonal Laplacian with unit face coefficient, zero-gradient sides, the reference cell's
    # diagonal doubled
    adr, g, ni, n = mesh.addressing(), mesh.geometry(), mesh.n_internal_faces, mesh.n_cells
    own, nbr = adr["owner"][:ni], adr["neighbour"]
    d, sf = g["d"][:ni], g["Sf"][:ni]
    a = np.einsum("ij,ij->i", sf, d) / np.einsum("ij,ij->i", d, d)
    x = _poisson_solution(c, seed)
    f = a * (x[own] - x[nbr])
    b = np.bincount(own, f, n) - np.bincount(nbr, f, n)
    diag0 = a[own == 0].sum() + a[nbr == 0].sum()
    b[0] += diag0 * x[0]
    hb = _pinned(n)
    hb[:] = b
    return dict(kind="poisson", case=case, b=hb, method=c["method"])


def _run_poisson(s):
    return {"x": s["case"].poisson_solve(s["b"], s["method"], tol=3e-12, max_iter=20000)[0]}


def _stencil_csr(dims, conv, rng):
    """A 7-point matrix on a block, rows sorted by column: diffusion with
    coefficients varying by 30% and, with conv, an upwind flow along x and a
    swirl; strictly dominant by a small time term."""
    nx, ny, nz = dims
    n = nx * ny * nz
    i = np.arange(n)
    ix, iy, iz = i % nx, (i // nx) % ny, i // (nx * ny)
    rows, cols, vals = [], [], []
    diag = np.full(n, 0.01)
    for step, ok, vel in ((1, ix < nx - 1, 1.0), (nx, iy < ny - 1, 0.3), (nx * ny, iz < nz - 1, -0.2)):
        o = i[ok]
        w = rng.uniform(0.7, 1.3, o.size)
        f = vel * conv * rng.uniform(0.5, 1.5, o.size)
        lo, up = -w - np.maximum(f, 0), -w - np.maximum(-f, 0)  # neighbour's row, owner's row
        rows += [o, o + step]
        cols += [o + step, o]
        vals += [up, lo]
        diag[o] -= up
        diag[o + step] -= lo
    rows, cols, vals = np.concatenate(rows + [i]), np.concatenate(cols + [i]), np.concatenate(vals + [diag])
    order = np.lexsort((cols, rows))
    start = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(rows, minlength=n), out=start[1:])
    return start, cols[order].astype(np.int64), vals[order], rows[order]


def _prepare_csr(c, seed):
    rng = np.random.default_rng(seed)
    dims = (c["nx"], c["ny"], c["nz"])
    start, cols, vals, rows = _stencil_csr(dims, 2.0 if c.get("method") == "bicgstab" else 0.0, rng)
    n = start.size - 1
    b = np.bincount(rows, vals * _solution(_lattice(*dims), seed)[cols], n)
    if c["kind"] == "csr":
        return dict(kind="csr", method=c["method"], a=(start, cols, vals), b=b, x0=np.zeros(n))
    dev = [torch.from_numpy(a).cuda() for a in (start.astype(np.int32), cols.astype(np.int32), vals, b)]
    return dict(kind="static", n=n, dev=dev, x=torch.zeros(n, dtype=torch.float64, device="cuda"))


def _run_csr(s):
    solve = cf.solve_bicgstab if s["method"] == "bicgstab" else cf.solve_cg
    x, _ = solve(*s["a"], s["b"], s["x0"], TOL, 4000)
    return {"x": x}


def _run_static(s):
    s["x"].zero_()
    rep = cf._capi._Report()
    a = [C.c_void_p(t.data_ptr()) for t in s["dev"]]
    rc = cf.lib().cfg_pcg_solve_static(C.c_int32(0), C.c_int64(s["n"]), a[0], a[1], a[2], a[3],
                                       C.c_void_p(s["x"].data_ptr()), C.c_double(TOL), C.c_int32(4000), None,
                                       C.byref(rep))
    if rc:
        raise cf.CfgError(rc, cf._capi._err())
    return {"x": s["x"]}


def _prepare_blocks(c, seed):
    rng = np.random.default_rng(seed)
    cases, qs, ctls = [], [], []
    for s in meshgen.detail_block_set(c["n"], c["spec"], c["cells_min"], c["cells_max"]):
        s["laminar"] = s["laminar"] or s["cells"] > 6000  # a large block's first k-epsilon pass may not converge
        mesh = meshgen.channel_block(s["cells"], s["aspect"])
        case = cf.SimpleCase(mesh)
        case.detail_setup(s["shape"], rho=998.0)
        speed = s["speed"] * rng.uniform(0.95, 1.05)
        nu = 1e-4 if s["laminar"] else s["speed"] * 0.1 / 2e4
        if not s["laminar"]:
            case.detail_turbulence("kEpsilon", intensity=0.05, length_scale=-1.0, relaxation=0.7, nu=nu)
        cases.append(case)
        qs.append(speed * 0.01)
        ctls.append(cf.SimpleControls(max_iterations=1, relax_u=0.7, relax_p=0.3, p_relax_start=0.002,
                                      non_orth_correctors=1, linear_tol=0.1 * TOL, linear_max_iter=4000, nu=nu,
                                      p_preconditioner="DIC"))
    batch = cf.Batch(cases)
    batch.set_schedule(0, -1)  # the pass as one CUDA-graph launch
    batch.loss(qs, ctls)       # the conditions, the RANS models and the graph
    out = []
    for case, q, ctl in zip(cases, qs, ctls):
        mesh = case.mesh
        ny = int(round(math.sqrt(next(p[3] for p in mesh.patches if p[0] == "inlet"))))
        dims = (mesh.n_cells // (ny * ny), ny, ny)
        v = q / 0.01
        _start_fields(case, mesh, dims, (0.1 * dims[0] / ny, 0.1, 0.1), v, 0.5 * v * v, rng)
        out.append(_out_fields(mesh))
    batch.save()
    return dict(kind="blocks", cases=cases, batch=batch, q=qs, controls=ctls, out=out)


def _run_blocks(s):
    s["batch"].restore()
    m, _ = s["batch"].loss(s["q"], s["controls"])
    got = {"dp": np.array([x["dp_pa"] for x in m]), "flux_out": np.array([x["flux_out"] for x in m])}
    for i, (case, out) in enumerate(zip(s["cases"], s["out"])):
        got["U%d" % i], got["p%d" % i], got["phi%d" % i] = case.download(*out)
    return got


_PREPARE = {"simple": _prepare_simple, "rans": _prepare_rans, "piso": _prepare_piso, "poisson": _prepare_poisson,
            "csr": _prepare_csr, "static": _prepare_csr, "blocks": _prepare_blocks}
_RUN = {"simple": _run_simple, "rans": _run_rans, "piso": _run_piso, "poisson": _run_poisson, "csr": _run_csr,
        "static": _run_static, "blocks": _run_blocks}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, int(seed) % (1 << 31))


def run(state):
    return _RUN[state["kind"]](state)


# ---- what a pass cannot do without -------------------------------------------

def _block_counts(nx, ny, nz):
    n = nx * ny * nz
    return n, 3 * n - nx * ny - ny * nz - nx * nz, 2 * (nx * ny + ny * nz + nx * nz)


def _flow_bytes(n, f, fb, outer):
    """Per outer iteration the face geometry (14 reals, 2 indices), the cell
    volumes and the fields in and out; both assembled matrices written and
    read once."""
    fields = 8 * (4 * n + f + fb)
    return outer * ((f + fb) * (14 * 8 + 8) + 8 * n + 2 * fields + 2 * 2 * (8 * n + 16 * f))


def work(case):
    k = case["kind"]
    if k in ("simple", "rans", "piso"):
        n, f, fb = _block_counts(case["nx"], case["ny"], case["nz"])
        outer = case.get("iters", 1)
        fields = {"simple": 4, "rans": 6, "piso": 4}[k]
        return {"bytes": _flow_bytes(n, f, fb, outer) + 2 * 8 * (fields * n + f + fb), "flops": outer * 300 * (n + f)}
    if k == "poisson":
        n, f, _ = _block_counts(case["n"] + 1, case["n"], case["n"] - 1)
        if case["mesh"] == "tets":
            n, f = 6.9 * case["n"] ** 3, 13.5 * case["n"] ** 3
        return {"bytes": 24 * n + 8 * n + 16 * f, "flops": 2 * n + 4 * f}
    if k in ("csr", "static"):
        n, f, _ = _block_counts(case["nx"], case["ny"], case["nz"])
        nnz = n + 2 * f
        per = 16 if k == "csr" else 12
        return {"bytes": per * nnz + (8 if k == "csr" else 4) * (n + 1) + 24 * n, "flops": 2 * nnz}
    total = 0.0
    for s in meshgen.detail_block_set(case["n"], case["spec"], case["cells_min"], case["cells_max"]):
        n = s["cells"]
        total += _flow_bytes(n, 3 * n, 0.3 * n, 1) + 2 * 8 * (4 * n + 3.3 * n)
    return {"bytes": total, "flops": total}


# ---- the results in 64 bits ---------------------------------------------------

def exact(case, seed):
    """The linear systems' right-hand sides are made from their solutions.  A
    flow solve's result has no short plain form: an outer iteration is several
    large nested solves and a whole discretisation."""
    seed = int(seed) % (1 << 31)
    if case["kind"] in ("csr", "static"):
        return {"x": _solution(_lattice(case["nx"], case["ny"], case["nz"]), seed)}
    if case["kind"] == "poisson":
        return {"x": _poisson_solution(case, seed)}
    return None
