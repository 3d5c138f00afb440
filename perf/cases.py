"""Performance cases of the solver: what its users have it do, through the
public entry points of the package (the Python classes and the C ABI they bind).

Families (field "family" of a case):

  step   the implicit solver on one of the four benchmark flows.  A pass loads a
         state from pinned host memory, advances it (Newton steps, the steady
         loop, or dual time steps) and reads the state back, which is what
         the end-to-end leg of bench.py does each step.
  bsr    the linear algebra on a caller's own block matrix with device vectors
         (the seam the reference adapters use): SGS set-up, product, SGS
         application, BiCGSTAB.
  recon  gradient and limiter on caller-owned device fields.
  mlp    the learned initial guess: inference on device features and one
         training epoch over a dataset.

Sizes are those of the benchmark flows and of the tests (4 thousand to 4.1
million cells).  The mesh, the solver handle (connectivity, orderings, device
storage) and the frozen limiter values belong to the case and are kept between
states, as a program that advances many states on one mesh keeps them; states,
matrix values, fields and samples come from the seed.
"""
from __future__ import annotations

import ctypes as C
import importlib.util
import math
import sys
from collections import OrderedDict
from pathlib import Path

import numpy as np
import torch

PKG = Path(__file__).resolve().parent.parent / "distributed-cfd-solver_b200"


def _package():
    if "cfd_b200" not in sys.modules:
        spec = importlib.util.spec_from_file_location("cfd_b200", PKG / "__init__.py",
                                                      submodule_search_locations=[str(PKG)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["cfd_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["cfd_b200"]


cb = _package()

L2_BYTES = 126e6
TETS = 6  # tetrahedra per hex of the bump mesh


# ------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest solver call: the supersonic ramp, ten iterations of the
        # steady loop (launch- and latency-bound)
        dict(name="ramp_steady_4k", family="step", flow="ramp", nx=64, ny=32, nz=2, mixed=False, sgs="color",
             operator="picard", guess=False, mode="steady", steps=10, its=30, rtol=1e-3),
        # the laminar plate at 1/8 size, the linear tolerance of the
        # time-to-convergence runs
        dict(name="plate_131k_rtol01", family="step", flow="plate", nx=128, ny=64, nz=16, mixed=False, sgs="color",
             operator="picard", guess=False, mode="newton", steps=1, its=30, rtol=1e-1),
        # the laminar plate at full size, plain FP64
        dict(name="plate_1m", family="step", flow="plate", nx=256, ny=128, nz=32, mixed=False, sgs="color",
             operator="picard", guess=False, mode="newton", steps=1, its=30, rtol=1e-3),
        # Spalart-Allmaras plate, mixed precision, 1/8 size
        dict(name="sa_516k_mixed", family="step", flow="sa_plate", nx=192, ny=96, nz=28, mixed=True, sgs="color",
             operator="picard", guess=False, mode="newton", steps=1, its=30, rtol=1e-3),
        # the headline workload: the 4.1M-cell Spalart-Allmaras plate in FP64,
        # with about half of the benchmark's 30 linear iterations (the solve
        # ends at the cap either way, and rounding grows with every one)
        dict(name="sa_4m", family="step", flow="sa_plate", nx=384, ny=192, nz=56, mixed=False, sgs="color",
             operator="picard", guess=False, mode="newton", steps=1, its=16, rtol=1e-3),
        # tetrahedra, mixed precision: the transonic bump at 1/8 size
        dict(name="bump_768k_mixed", family="step", flow="bump", nx=80, ny=40, nz=40, mixed=True, sgs="color",
             operator="picard", guess=False, mode="newton", steps=1, its=30, rtol=1e-3),
        # the learned initial guess: a step that makes a previous update and a
        # step that starts from the network's prediction
        dict(name="bump_guess_96k", family="step", flow="bump", nx=40, ny=20, nz=20, mixed=True, sgs="color",
             operator="picard", guess=True, mode="newton", steps=2, its=30, rtol=1e-3),
        # the reference's own (sequential) sweep order, level-scheduled
        dict(name="plate_level_16k", family="step", flow="plate", nx=64, ny=32, nz=8, mixed=False, sgs="level",
             operator="picard", guess=False, mode="newton", steps=1, its=10, rtol=1e-3),
        # Jacobian-free Newton-Krylov: every GMRES product is a residual
        # evaluation
        dict(name="plate_jfnk_131k", family="step", flow="plate", nx=128, ny=64, nz=16, mixed=False, sgs="color",
             operator="jfnk", guess=False, mode="newton", steps=1, its=20, rtol=1e-2),
        # a caller's own matrix of odd size, natural cell order
        dict(name="bsr_219k_bs5", family="bsr", nx=97, ny=61, nz=37, bs=5, mixed=False, sgs="color", order="natural",
             its=12),
        # reconstruction operators on a caller's fields, odd-sized tet mesh
        dict(name="recon_393k", family="recon", nx=61, ny=37, nz=29, nvars=5, limiter=1, gradient=3),
        # the network alone: inference and one training epoch
        dict(name="mlp_600k", family="mlp", rows=600_011, nvars=6, batch=8192),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, cells, aspect):
    """Three extents of about `cells` cells with the proportions `aspect`, odd ones among them."""
    f = (cells / (aspect[0] * aspect[1] * aspect[2])) ** (1.0 / 3.0)
    return [max(2, int(round(a * f * rng.uniform(0.85, 1.15)))) for a in aspect]


def draw(rng):
    family = rng.choices(("step", "bsr", "recon", "mlp"), (6, 2, 1, 1))[0]
    if family == "bsr":
        nx, ny, nz = _box(rng, _logint(rng, 4_000, 400_000), (3.0, 2.0, 1.0))
        return dict(family="bsr", nx=nx, ny=ny, nz=nz, bs=rng.choice((1, 3, 4, 5, 6)), mixed=rng.random() < 0.5,
                    sgs=rng.choice(("color", "color", "level")), order=rng.choice(("natural", "colour")),
                    its=rng.randint(4, 14))
    if family == "recon":
        nx, ny, nz = _box(rng, _logint(rng, 600, 100_000), (2.0, 1.0, 1.0))
        return dict(family="recon", nx=nx, ny=ny, nz=nz, nvars=rng.choice((1, 3, 5, 6)), limiter=rng.choice((1, 2, 3)),
                    gradient=rng.choice((2, 3)))
    if family == "mlp":
        return dict(family="mlp", rows=_logint(rng, 2_000, 1_500_000), nvars=rng.choice((5, 6)),
                    batch=rng.choice((2048, 4096, 8192)))
    flow = rng.choice(("ramp", "plate", "plate", "sa_plate", "sa_plate", "bump", "bump"))
    case = dict(family="step", flow=flow, mixed=rng.random() < 0.5, sgs="color", operator="picard", guess=False,
                mode="newton", steps=1, its=rng.randint(6, 20), rtol=1e-3)
    if flow == "ramp":
        nx, ny, nz = _box(rng, _logint(rng, 500, 30_000), (8.0, 4.0, 1.0))
        case.update(mode=rng.choice(("newton", "steady", "unsteady")), steps=rng.randint(2, 6))
    elif flow == "bump":
        nx, ny, nz = _box(rng, _logint(rng, 600, 130_000), (2.0, 1.0, 1.0))
        if rng.random() < 0.3:
            case.update(guess=True, steps=2)
    else:
        nx, ny, nz = _box(rng, _logint(rng, 8_000, 1_000_000), (8.0, 4.0, 1.0))
        kind = rng.random()
        if kind < 0.2 and nx * ny * nz < 60_000:
            case.update(sgs="level", its=rng.randint(3, 10))
        elif kind < 0.4 and nx * ny * nz < 300_000:
            case.update(operator="jfnk", its=rng.randint(5, 20), rtol=1e-2)
    case.update(nx=nx, ny=ny, nz=nz)
    return case


def _key(case):
    return tuple(sorted((k, v) for k, v in case.items() if k != "name"))


_KEPT: OrderedDict = OrderedDict()
KEEP_CELLS = 14_000_000


def _kept(case, make):
    """The case's mesh and handle, built once; the oldest go when many cells are held."""
    key = _key(case)
    if key not in _KEPT:
        _KEPT[key] = make()
        while len(_KEPT) > 1 and sum(h["cells"] for h in _KEPT.values()) > KEEP_CELLS:
            _KEPT.popitem(last=False)
    _KEPT.move_to_end(key)
    return _KEPT[key]


def _pinned_ptr(t):
    return C.cast(t.data_ptr(), C.POINTER(C.c_double))


def _centroids(mesh):
    v = mesh.view
    return torch.from_numpy(np.stack([np.ctypeslib.as_array(p, shape=(v.n_cells,)) for p in (
        v.cell_centroid_x, v.cell_centroid_y, v.cell_centroid_z)])).cuda()


def _waves(xyz, rng):
    """Three smooth waves through the box, values in about [-1, 1]."""
    lo = xyz.amin(dim=1, keepdim=True)
    t = (xyz - lo) / (xyz.amax(dim=1, keepdim=True) - lo).clamp_min(1e-30)
    out = torch.zeros_like(t[0])
    for _ in range(3):
        k = rng.integers(1, 6, size=3) * 2.0 * math.pi
        out += torch.sin(k[0] * t[0] + k[1] * t[1] + k[2] * t[2] + rng.uniform(0, 2 * math.pi)) / 3.0
    return out


# -------------------------------------------------------------------- step
def _flow(case):
    flow, nx, ny, nz = case["flow"], case["nx"], case["ny"], case["nz"]
    if flow == "ramp":
        c = cb.cases.ramp()
        c.spec.lz = nz * c.spec.lx / nx
    elif flow == "plate":
        c = cb.cases.plate(mixed=case["mixed"])
        f = 128.0 / ny  # the wall-normal growth covers the same height with ny cells
        c.spec.first_spacing, c.spec.stretch = 1.0e-5 * f, 1.08 ** f
    elif flow == "sa_plate":
        c = cb.cases.sa_plate(mixed=case["mixed"])
        f = 192.0 / ny
        c.spec.first_spacing, c.spec.stretch, c.spec.cap_spacing = 1.0e-6 * f, 1.1 ** f, 0.01 * f
    else:
        c = cb.cases.bump(mixed=case["mixed"])
    c.spec.nx, c.spec.ny, c.spec.nz = nx, ny, nz
    cfg = c.cfg
    cfg.precision = cb.PREC_MIXED if case["mixed"] else cb.PREC_FP64
    cfg.sgs_ordering = cb.SGS_LEVEL if case["sgs"] == "level" else cb.SGS_COLOR
    cfg.lin_max_iterations, cfg.lin_rel_tol = case["its"], case["rtol"]
    cfg.residual_tolerance = 0.0
    if case["operator"] == "jfnk":
        cfg.newton_operator = cb.NEWTON_JACOBIAN_FREE
        cfg.jf_max_iterations, cfg.jf_rel_tol, cfg.jf_accept = case["its"], case["rtol"], 1.0
    if case["mode"] == "steady":
        cfg.max_iterations = case["steps"]
    elif case["mode"] == "unsteady":
        cfg.time_mode, cfg.bdf_order, cfg.dt_physical = cb.TIME_UNSTEADY, 2, 2.0e-5
        cfg.max_time_steps, cfg.max_iterations = 2, case["steps"]
        cfg.cfl = cfg.cfl_max = 20.0
    return c


def _state(c, xyz, seed, out):
    """A smooth flow of the case around its free stream (a wall layer on the plates) into `out`."""
    rng = np.random.default_rng(seed)
    cfg = c.cfg
    rho0, p0, u0 = cfg.init_rho, cfg.init_p, cfg.init_velocity[0]
    g1 = cfg.gamma - 1.0
    rho = rho0 * (1.0 + 0.02 * _waves(xyz, rng))
    p = p0 * (1.0 + 0.02 * _waves(xyz, rng))
    u = u0 * (1.0 + 0.02 * _waves(xyz, rng))
    v = 0.02 * u0 * _waves(xyz, rng)
    w = 0.02 * u0 * _waves(xyz, rng)
    rows = [rho]
    if cfg.viscous:
        y = (xyz[1] / 0.01).clamp_max(50.0)
        on = torch.sigmoid((xyz[0] - c.spec.plate_x0) / 0.05)
        wall = 1.0 - on * torch.exp(-y)
        u, v, w = u * wall, v * wall, w * wall
    rows += [rho * u, rho * v, rho * w, p / g1 + 0.5 * rho * (u * u + v * v + w * w)]
    if cfg.turbulence:
        nu = c.extra["nu_inf"] * (1.0 + 20.0 * on * y * torch.exp(-y)) * (1.0 + 0.02 * _waves(xyz, rng))
        rows.append(rho * nu)
    for k, row in enumerate(rows):
        out[k].copy_(row)
    torch.cuda.synchronize()


def _damped_update_net(nvars):
    """A network that predicts a fraction of the previous update (its third group of features)."""
    net = cb.Mlp(nvars, seed=11)
    sizes = [(64, 48), (64,), (64, 64), (64,), (16, 64), (16,)]
    w1, b1, w2, b2, w3, b3 = [np.zeros(s, dtype=np.float32) for s in sizes]
    for v in range(nvars):
        w1[2 * v, 2 * nvars + v], w1[2 * v + 1, 2 * nvars + v] = 1.0, -1.0
        w2[2 * v, 2 * v] = w2[2 * v + 1, 2 * v + 1] = 1.0
        w3[v, 2 * v], w3[v, 2 * v + 1] = 0.25, -0.25
    net.set_params(np.concatenate([a.ravel() for a in (w1, b1, w2, b2, w3, b3)]))
    return net


def _step_handle(case):
    c = _flow(case)
    mesh = cb.HostMesh(c.spec)
    solver = cb.Solver(mesh, c.cfg, c.bcs)
    h = dict(case=c, mesh=mesh, solver=solver, cells=mesh.n_cells, xyz=_centroids(mesh))
    if case["guess"]:
        h["net"] = _damped_update_net(solver.nvars)
        solver.attach_guess(h["net"])
    if case["mode"] == "newton":
        # the limiter as it stands after the CFL ramp: frozen, here at the
        # values of a state of its own
        U = torch.empty(solver.nvars, mesh.n_cells, dtype=torch.float64, pin_memory=True)
        _state(c, h["xyz"], 987654321, U)
        cb.check(cb.lib().cfdg_solver_set_state(solver._h, _pinned_ptr(U), mesh.n_cells))
        solver.evaluate_residual()
        solver.freeze_limiter(True)
    return h


def _step_prepare(case, seed):
    h = _kept(case, lambda: _step_handle(case))
    n, nv = h["solver"].n_cells, h["solver"].nvars
    U = torch.empty(nv, n, dtype=torch.float64, pin_memory=True)
    _state(h["case"], h["xyz"], seed, U)
    return dict(family="step", mode=case["mode"], steps=case["steps"], solver=h["solver"], keep=h, U=U,
                cfl=h["case"].cfg.cfl_max, out=torch.empty(nv, n, dtype=torch.float64, pin_memory=True))


def _step_run(s):
    solver, lib = s["solver"], cb.lib()
    cb.check(lib.cfdg_solver_set_state(solver._h, _pinned_ptr(s["U"]), solver.n_cells))
    if s["mode"] == "steady":
        norms = solver.run_steady().l2_last
    elif s["mode"] == "unsteady":
        solver.reset_time_levels()
        norms = solver.run_unsteady().l2_last
    else:
        for _ in range(s["steps"]):
            norms = solver.newton_step(s["cfl"]).l2
    cb.check(lib.cfdg_solver_get_field(solver._h, cb.FIELD_U, _pinned_ptr(s["out"]), s["out"].numel()))
    return {"U": list(s["out"].unbind(0)), "norms": [float(norms[v]) for v in range(solver.nvars)]}


def _step_counts(case):
    hexes = case["nx"] * case["ny"] * case["nz"]
    n = hexes * (TETS if case["flow"] == "bump" else 1)
    inner = 2 * n if case["flow"] == "bump" else 3 * n
    bs = 6 if case["flow"] == "sa_plate" else 5
    return n, inner, n + 2 * inner, bs


def _step_work(case):
    """The state in and out, per iteration the mesh and the matrix written once, and the matrix read for
    the two products of each BiCGSTAB iteration when it does not stay on the chip."""
    n, faces, blocks, bs = _step_counts(case)
    size = 4 if case["mixed"] else 8
    steps = case["steps"] * (2 if case["mode"] == "unsteady" else 1)
    matrix = blocks * bs * bs * size
    fits = matrix < L2_BYTES
    mesh = faces * (8 * 8) + n * (4 * 8)
    vector = n * bs * 8
    if case["operator"] == "jfnk":
        its = case["its"]
        solve = its * (mesh + 2 * vector) + its * (0 if fits else matrix) + its * its // 2 * vector
        flops = its * (2 * blocks * bs * bs + 1200 * faces)
    else:
        its = case["its"]
        solve = (1 if fits else 2 * its) * matrix + 2 * vector
        flops = 2 * its * 2 * blocks * bs * bs
    one = mesh + 2 * vector + matrix + solve
    return {"bytes": float(2 * vector + steps * one), "flops": float(steps * (flops + 3000 * faces))}


# --------------------------------------------------------------------- bsr
def _box_rows(case):
    """Natural-order indices of the box, colours (i + j + k) % 2, and row numbers in the chosen order."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    k, j, i = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    parity = ((i + j + k) % 2).ravel()
    n = parity.size
    if case["order"] == "colour":
        cell = np.argsort(parity, kind="stable")  # row -> cell
    else:
        cell = np.arange(n)
    row = np.empty(n, dtype=np.int64)
    row[cell] = np.arange(n)
    return (nx, ny, nz), parity, cell, row


def _bsr_structure(case):
    (nx, ny, nz), parity, cell, row = _box_rows(case)
    n = parity.size
    cols = np.full((n, 7), np.iinfo(np.int64).max, dtype=np.int64)
    c = np.arange(n).reshape(nz, ny, nx)
    cols[:, 3] = row
    for slot, (axis, step) in enumerate(((0, -1), (1, -1), (2, -1), (2, 1), (1, 1), (0, 1))):
        s = slot if slot < 3 else slot + 1
        here = [slice(None)] * 3
        there = [slice(None)] * 3
        here[axis], there[axis] = (slice(1, None), slice(0, -1)) if step < 0 else (slice(0, -1), slice(1, None))
        cols[c[tuple(here)].ravel(), s] = row[c[tuple(there)].ravel()]
    cols = np.sort(cols[cell], axis=1)  # rows in the chosen order, missing neighbours last
    have = cols < n
    row_ptr = np.zeros(n + 1, dtype=np.int32)
    row_ptr[1:] = np.cumsum(have.sum(axis=1))
    flat = cols[have].astype(np.int32)
    rows = np.repeat(np.arange(n), have.sum(axis=1))
    return row_ptr, flat, rows, parity[cell], cell


def _bsr_handle(case):
    row_ptr, cols, rows, colour, cell = _bsr_structure(case)
    a = cb.Bsr(row_ptr, cols, case["bs"], cb.PREC_MIXED if case["mixed"] else cb.PREC_FP64)
    return dict(a=a, cells=len(colour), row_ptr=row_ptr, cols=torch.from_numpy(cols).cuda().long(),
                rows=torch.from_numpy(rows).cuda(), colour=torch.from_numpy(colour).cuda(), cell=cell)


def _bsr_values(h, case, seed):
    """An implicit time step's matrix: a transport-like coupling between neighbours, a dominant diagonal."""
    g = torch.Generator("cuda").manual_seed(seed)
    bs, nnz = case["bs"], h["cols"].numel()
    eye = torch.eye(bs, dtype=torch.float64, device="cuda")
    v = 0.25 / bs * torch.randn(nnz, bs, bs, generator=g, dtype=torch.float64, device="cuda") - eye
    diag = torch.nonzero(h["rows"] == h["cols"]).ravel()
    v[diag] = 6.2 * eye + 0.5 / bs * torch.randn(diag.numel(), bs, bs, generator=g, dtype=torch.float64, device="cuda")
    n = h["cells"] * bs
    x = torch.randn(n, generator=g, dtype=torch.float64, device="cuda")
    b = torch.randn(n, generator=g, dtype=torch.float64, device="cuda")
    return v, x, b


def _bsr_prepare(case, seed):
    # the values belong to the state: a handle of its own on the case's structure
    h = _kept(case, lambda: _bsr_handle(case))
    v, x, b = _bsr_values(h, case, seed)
    a = cb.Bsr(h["row_ptr"], h["a"].cols, case["bs"], cb.PREC_MIXED if case["mixed"] else cb.PREC_FP64)
    a.set_values(v.cpu().numpy())
    new = lambda: torch.zeros_like(x)  # noqa: E731
    torch.cuda.synchronize()
    return dict(family="bsr", a=a, x=x, b=b, y=new(), z=new(), sol=new(), its=case["its"],
                ordering=cb.SGS_LEVEL if case["sgs"] == "level" else cb.SGS_COLOR)


def _bsr_run(s):
    lib, a = cb.lib(), s["a"]
    s["sol"].zero_()
    torch.cuda.current_stream().synchronize()  # the library works on a stream of its own
    a.sgs_setup(s["ordering"], 1)
    cb.check(lib.cfdg_bsr_spmv(a._h, s["x"].data_ptr(), s["y"].data_ptr(), 1.0, 0.0))
    cb.check(lib.cfdg_sgs_apply(a._h, s["b"].data_ptr(), s["z"].data_ptr()))
    r = cb.KrylovResult()
    cb.check(lib.cfdg_bicgstab(a._h, cb.PC_SGS, 1e-14, 1e-300, s["its"], s["sol"].data_ptr(), s["b"].data_ptr(),
                               C.byref(r)))
    return {"y": s["y"], "z": s["z"], "x": s["sol"]}


def _bsr_exact(case, seed):
    h = _kept(case, lambda: _bsr_handle(case))
    v, x, b = _bsr_values(h, case, seed)
    n, bs = h["cells"], case["bs"]
    rows, cols = h["rows"], h["cols"]

    def product(u, pick=None):
        r, c, m = (rows, cols, v) if pick is None else (rows[pick], cols[pick], v[pick])
        t = torch.bmm(m, u.view(n, bs)[c].unsqueeze(2)).squeeze(2)
        return torch.zeros(n, bs, dtype=torch.float64, device="cuda").index_add_(0, r, t).view(-1)

    inv = torch.linalg.inv(v[torch.nonzero(rows == cols).ravel()])
    if case["sgs"] == "level":  # the sequential sweep in row order
        cell = torch.from_numpy(h["cell"]).cuda()
        nx, ny = case["nx"], case["ny"]
        plane = cell % nx + (cell // nx) % ny + cell // (nx * ny)
        key = plane + (h["colour"] * 10_000_000 if case["order"] == "colour" else 0)
    else:
        key = h["colour"]
    # groups of rows without neighbours among them, in sweep order, and each group's blocks
    _, group = torch.unique(key, return_inverse=True)
    ng = int(group.max()) + 1
    if case["sgs"] == "level" and case["order"] == "colour":
        group, ng = h["colour"], 2  # rows of a colour are independent and the colours follow each other
    off = rows != cols
    by_row = [torch.nonzero(group == q).ravel() for q in range(ng)]
    order = torch.argsort(group[rows[off]], stable=True)
    entries = torch.nonzero(off).ravel()[order]
    ends = torch.bincount(group[rows[entries]], minlength=ng).cumsum(0).tolist()
    by_entry = [entries[(ends[q - 1] if q else 0):ends[q]] for q in range(ng)]

    def sgs(r):
        z = torch.zeros(n, bs, dtype=torch.float64, device="cuda")
        r = r.view(n, bs)
        for q in list(range(ng)) + list(range(ng - 1, -1, -1)):
            e = by_entry[q]
            t = torch.bmm(v[e], z[cols[e]].unsqueeze(2)).squeeze(2)
            s = r.clone() if ng == 2 else None
            if s is None:
                s = torch.zeros(n, bs, dtype=torch.float64, device="cuda")
                s[by_row[q]] = r[by_row[q]]
            s.index_add_(0, rows[e], t, alpha=-1.0)
            z[by_row[q]] = torch.bmm(inv[by_row[q]], s[by_row[q]].unsqueeze(2)).squeeze(2)
        return z.view(-1)

    y, z = product(x), sgs(b)
    if ng > 2 and n > 60_000:  # hundreds of levels, two sweeps an iteration
        return {"y": y, "z": z, "x": None}
    xs = torch.zeros_like(b)
    r = b.clone()
    r0, p = r.clone(), r.clone()
    rho = r0 @ r
    for _ in range(case["its"]):
        ph = sgs(p)
        vv = product(ph)
        alpha = rho / (r0 @ vv)
        s = r - alpha * vv
        sh = sgs(s)
        t = product(sh)
        omega = (t @ s) / (t @ t)
        xs += alpha * ph + omega * sh
        r = s - omega * t
        rho_new = r0 @ r
        p = r + (rho_new / rho) * (alpha / omega) * (p - omega * vv)
        rho = rho_new
    return {"y": y, "z": z, "x": xs}


def _bsr_work(case):
    n = case["nx"] * case["ny"] * case["nz"]
    blocks = 7 * n - 2 * (n // case["nx"] + n // case["ny"] + n // case["nz"])
    matrix = blocks * (case["bs"] ** 2 * (4 if case["mixed"] else 8) + 4)
    vec = n * case["bs"] * 8
    reads = 1 if matrix < L2_BYTES else 2 + 2 * case["its"]
    return {"bytes": float(reads * matrix + 7 * vec), "flops": float((3 + 2 * case["its"]) * 2 * blocks * case["bs"] ** 2)}


# ------------------------------------------------------------------- recon
def _recon_handle(case):
    c = cb.cases.bump(mixed=False)
    c.spec.nx, c.spec.ny, c.spec.nz = case["nx"], case["ny"], case["nz"]
    mesh = cb.HostMesh(c.spec)
    op = cb.Recon(mesh, gradient=case["gradient"], limiter=case["limiter"])
    return dict(mesh=mesh, op=op, cells=mesh.n_cells, xyz=_centroids(mesh))


def _recon_fields(h, case, seed):
    """Smooth fields with a jump across a plane, as a flow with a shock has."""
    rng = np.random.default_rng(seed)
    xyz = h["xyz"]
    q = torch.empty(case["nvars"], h["cells"], dtype=torch.float64, device="cuda")
    for v in range(case["nvars"]):
        shock = torch.sigmoid((xyz[0] - rng.uniform(1.2, 1.8)) / 0.02)
        q[v] = 1.0 + v + 0.1 * _waves(xyz, rng) + 0.3 * shock
    return q


def _recon_prepare(case, seed):
    h = _kept(case, lambda: _recon_handle(case))
    q = _recon_fields(h, case, seed)
    grad = torch.zeros(3, case["nvars"], h["cells"], dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    return dict(family="recon", op=h["op"], keep=h, q=q, grad=grad, phi=torch.zeros_like(q))


def _recon_run(s):
    ptrs = lambda t: [r.data_ptr() for r in t]  # noqa: E731
    q, g, phi, st = ptrs(s["q"]), [ptrs(d) for d in s["grad"]], ptrs(s["phi"]), torch.cuda.current_stream().cuda_stream
    s["op"].gradient(q, *g, stream=st)
    s["op"].limiter(q, *g, phi, stream=st)
    return {"gx": s["grad"][0], "gy": s["grad"][1], "gz": s["grad"][2], "phi": s["phi"]}


def _recon_exact(case, seed):
    h = _kept(case, lambda: _recon_handle(case))
    q, xyz, m = _recon_fields(h, case, seed), h["xyz"], h["mesh"].arrays()
    n, ni = h["cells"], h["mesh"].n_inner
    own = torch.from_numpy(m["face_owner"]).cuda().long()
    nei = torch.from_numpy(m["face_neigh"][:ni]).cuda().long()
    pairs = torch.cat([own[:ni] * n + nei, nei * n + own[:ni]]).sort().values
    face_pairs = pairs
    if case["gradient"] == cb.GRAD_LSQ_NODE:  # cells that share a node
        nodes = torch.from_numpy(m["cell_nodes"]).cuda().long()
        of = torch.repeat_interleave(torch.arange(n, device="cuda"),
                                     torch.from_numpy(np.diff(m["cell_nodes_offsets"])).cuda().long())
        order = torch.argsort(nodes, stable=True)
        nodes, of = nodes[order], of[order]
        found = []
        for shift in range(1, int(torch.bincount(nodes).max())):
            same = nodes[shift:] == nodes[:-shift]
            a, b = of[shift:][same], of[:-shift][same]
            found += [a * n + b, b * n + a]
        pairs = torch.unique(torch.cat(found))
    i, j = pairs // n, pairs % n
    dr = xyz[:, j] - xyz[:, i]
    w = 1.0 / (dr * dr).sum(0).clamp_min(1e-30)
    A = torch.zeros(n, 3, 3, dtype=torch.float64, device="cuda")
    for a in range(3):
        for b in range(3):
            A[:, a, b].index_add_(0, i, w * dr[a] * dr[b])
        A[:, a, a] += 1e-14
    # cells whose neighbours do not span space keep a zero gradient
    flat = torch.linalg.det(A).abs() <= 1e-14
    A[flat] = torch.eye(3, dtype=torch.float64, device="cuda")
    inv = torch.linalg.inv(A) * (~flat).view(-1, 1, 1)
    grad = torch.empty(3, case["nvars"], n, dtype=torch.float64, device="cuda")
    for v in range(case["nvars"]):
        rhs = torch.zeros(n, 3, dtype=torch.float64, device="cuda")
        for a in range(3):
            rhs[:, a].index_add_(0, i, w * dr[a] * (q[v, j] - q[v, i]))
        grad[:, v] = torch.bmm(inv, rhs.unsqueeze(2)).squeeze(2).T
    # limiter: face-neighbour extrema, then the smallest value over the cell's faces
    fi, fj = face_pairs // n, face_pairs % n
    fc = torch.from_numpy(np.stack([m[k] for k in ("face_centroid_x", "face_centroid_y", "face_centroid_z")])).cuda()
    cell = torch.cat([own, nei])
    e = torch.cat([fc, fc[:, :ni]], dim=1) - xyz[:, cell]
    eps2 = 0.5 ** 3 * torch.from_numpy(m["cell_volume"]).cuda()[cell]
    phi = torch.ones_like(q)
    for v in range(case["nvars"]):
        hi = q[v].clone().scatter_reduce_(0, fi, q[v, fj], "amax") - q[v]
        lo = q[v].clone().scatter_reduce_(0, fi, q[v, fj], "amin") - q[v]
        df = (grad[:, v, cell] * e).sum(0)
        d = torch.where(df > 0, hi[cell], lo[cell])
        prod = d * df
        if case["limiter"] == cb.LIM_BARTH_JESPERSEN:
            f = (d / df).clamp(0.0, 1.0)
        else:
            if case["limiter"] == cb.LIM_VAN_ALBADA:
                f = (d * d + prod) / (d * d + df * df + eps2)
            else:
                f = (d * d + eps2 + 2 * prod) / (d * d + eps2 + 2 * df * df + prod)
            f = torch.where(prod <= 0, torch.zeros_like(f), f)
        f = torch.where(df == 0, torch.ones_like(f), f)
        phi[v].scatter_reduce_(0, cell, f, "amin")
    return {"gx": grad[0], "gy": grad[1], "gz": grad[2], "phi": phi}


def _recon_work(case):
    n = case["nx"] * case["ny"] * case["nz"] * TETS
    entries = n * (66 if case["gradient"] == cb.GRAD_LSQ_NODE else 4)
    # fields in, gradient and limiter out; centroids and the stencil's columns define the weights
    return {"bytes": float(n * 8 * case["nvars"] * 5 + n * 8 * 4 + 2 * n * 8 * 3 + entries * 4),
            "flops": float(entries * 7 * case["nvars"] + 4 * n * 20 * case["nvars"])}


# --------------------------------------------------------------------- mlp
def _mlp_samples(case, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    x = torch.randn(case["rows"], cb.MLP_IN, generator=g, device="cuda").to(torch.bfloat16)
    t = torch.zeros(case["rows"], cb.MLP_OUT, device="cuda")
    mix = torch.randn(cb.MLP_IN, case["nvars"], generator=g, device="cuda") / cb.MLP_IN ** 0.5
    t[:, :case["nvars"]] = torch.tanh(x.float() @ mix)
    scale = torch.rand(8, generator=g, dtype=torch.float64, device="cuda") + 0.5
    return x, t, scale


def _mlp_prepare(case, seed):
    x, t, scale = _mlp_samples(case, seed)
    net = cb.Mlp(case["nvars"], seed=3)
    ds = cb.Dataset(case["nvars"], case["rows"])
    ds.append(x.view(torch.int16).cpu().numpy().view(np.uint16), t.cpu().numpy())
    out = torch.zeros(case["rows"], case["nvars"], dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    return dict(family="mlp", net=net, ds=ds, x=x, scale=scale, out=out, start=net.get_params(), batch=case["batch"])


def _mlp_run(s):
    net = s["net"]
    net.set_params(s["start"])
    cb.check(cb.lib().cfdg_mlp_forward(net._h, C.c_void_p(s["x"].data_ptr()), s["x"].shape[0],
                                       C.c_void_p(s["scale"].data_ptr()), C.c_void_p(s["out"].data_ptr())))
    loss = net.train(s["ds"], epochs=1, batch=s["batch"], lr=1e-3)
    return {"y": s["out"], "loss": loss, "params": net.get_params()}


def _mlp_exact(case, seed):
    x, _, scale = _mlp_samples(case, seed)
    p = torch.from_numpy(cb.Mlp(case["nvars"], seed=3).get_params()).cuda().double()
    sizes = [(64, 48), (64,), (64, 64), (64,), (16, 64), (16,)]
    w1, b1, w2, b2, w3, b3 = [t.view(s) for t, s in zip(p.split([math.prod(s) for s in sizes]), sizes)]
    y = torch.relu(torch.relu(x.double() @ w1.T + b1) @ w2.T + b2) @ w3.T + b3
    # the trained parameters follow the batches' order and 16-bit gradients: no 64-bit value of their own
    return {"y": y[:, :case["nvars"]] * scale[:case["nvars"]], "loss": None, "params": None}


def _mlp_work(case):
    macs = 48 * 64 + 64 * 64 + 64 * 16
    return {"bytes": float(case["rows"] * (2 * cb.MLP_IN * 2 + 4 * cb.MLP_OUT + 8 * case["nvars"])),
            "flops": float(case["rows"] * 2 * macs * 4)}


# --------------------------------------------------------------- interface
def prepare(case, seed):
    return {"step": _step_prepare, "bsr": _bsr_prepare, "recon": _recon_prepare,
            "mlp": _mlp_prepare}[case["family"]](case, seed)


def run(state):
    return {"step": _step_run, "bsr": _bsr_run, "recon": _recon_run, "mlp": _mlp_run}[state["family"]](state)


def work(case):
    return {"step": _step_work, "bsr": _bsr_work, "recon": _recon_work, "mlp": _mlp_work}[case["family"]](case)


def exact(case, seed):
    """The linear algebra, the reconstruction and the network in 64 bits; the solver's steps compute in
    64 bits themselves (FP32 enters only through the linear solve that the bsr family pins)."""
    if case["family"] == "step":
        return None
    return {"bsr": _bsr_exact, "recon": _recon_exact, "mlp": _mlp_exact}[case["family"]](case, seed)


def tolerance(case):
    """About four times the differences seen between runs whose input differs by one unit in the last place
    (FP64) or between FP32 and FP64 matrices (mixed): the wall spacing and the unconverged linear solves
    amplify rounding, most on the Spalart-Allmaras plate."""
    family = case["family"]
    if family == "mlp":
        return {"rel": 1e-2, "max": 0.2}  # bf16 weights and activations
    if family == "recon":
        return {"rel": 1e-12, "max": 1e-9}
    if family == "bsr":
        return {"rel": 5e-7, "max": 1e-5} if case["mixed"] else {"rel": 1e-12, "max": 1e-10}
    if case["operator"] == "jfnk":
        return {"rel": 3e-4, "max": 2e-3}  # finite-difference products
    if case["flow"] == "sa_plate":
        return {"rel": 1e-5, "max": 3e-4}
    if case["guess"]:
        return {"rel": 5e-5, "max": 4e-4}
    if case["mixed"] and case["flow"] != "ramp":
        return {"rel": 1e-6, "max": 1e-5}
    return {"rel": 1e-8, "max": 1e-7}
