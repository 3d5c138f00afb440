"""Benchmark of the implicit hot path on B200: Mcell-iter/s of full Newton
iterations (residual -> 6x6 BSR Jacobian -> BiCGSTAB + SGS -> update) on the
Spalart-Allmaras flat plate (384x192x56 hex, 4,128,768 cells), plain FP64
for `value`, with mixed precision and mixed precision + learned initial
guess measured on the same iterations beside it; and time to a 1e-8
residual drop, FP64 vs mixed vs mixed + learned guess.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
                  [--case sa_plate|plate|bump|ramp] [--scale S]

One step = one nonlinear iteration over the whole mesh at the operating
point after the CFL ramp: every leg first runs the case's 50-iteration CFL
ramp (CFL 1 -> 100; the limiter freezes at its end, and the iterations
before the freeze use the FP64 matrix in every leg), untimed, then W warm-up
and K timed iterations at CFL 100.  `value` is timed with CUDA events on
the solver stream with the state resident in HBM (the 8.3 GB Jacobian and
the fields exceed the 126 MB L2, so no flush is needed); `e2e` replays the
same K iterations from the same state through the C ABI with the state
copied in from pinned host memory and back out every step.  Under torchrun
each rank runs an independent replica on its own GPU (no data-path
collective); value is the sum over ranks of cells x steps over the maximum
rank time, and the mixed / learned legs and the time-to-1e-8 runs are
single-GPU only.

time_to_1e8 (single GPU): the transonic Euler bump (M = 0.85; the
160x80x80x6-tet mesh divided by --converge-scale per direction, 2 by
default: 768,000 cells) run to a 1e-8 residual drop as plain FP64, mixed
precision and mixed precision with the learned initial guess, each its own
run from the free stream; converged fields are compared with the FP64 run.
time_to_1e8_plate: the laminar plate (256x128x32 hex divided by
--plate-converge-scale, 2 by default: 131,072 cells) to 1e-8, FP64 and mixed.
The Spalart-Allmaras plate needs tens of thousands of Newton iterations at
full size; `--converge-only --converge-case sa_plate` runs its comparison
(FP64, mixed, mixed + learned) at --converge-scale.

`--impl reference` times the reference's CPU implementation on a bounded
sample of the same workload (see run_reference).
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import tempfile
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

METRIC = "time to 1e-8 residual drop & Mcell-iter/s: FP64 plain vs mixed+learned, 1 B200"
UNIT = "Mcell-iter/s"


def _peaks():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return float(d.get("hbm_gbs", 6650.0)), "measured"
    return 6650.0, "fallback"


def _dist():
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return world, rank, local


class Clocks:
    """nvidia-smi samples (every 200 ms) during the timed region."""

    def __init__(self, index: int):
        self.index = index
        self.proc = None
        self.path = None

    def __enter__(self):
        fd, self.path = tempfile.mkstemp(suffix=".csv")
        os.close(fd)
        q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
             "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
             "clocks_event_reasons.sw_power_cap")
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.index}", f"--query-gpu={q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except FileNotFoundError:
            self.proc = None
        time.sleep(0.3)
        return self

    def __exit__(self, *a):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        try:
            for line in Path(self.path).read_text().splitlines():
                f = [x.strip() for x in line.split(",")]
                if len(f) < 9:
                    continue
                try:
                    sm.append(float(f[1]))
                    mx.append(float(f[2]))
                except ValueError:
                    continue
                for name, val in zip(names, f[5:9]):
                    if val.lower() == "active":
                        reasons.add(name)
        finally:
            try:
                os.unlink(self.path)
            except OSError:
                pass
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": [], "samples": 0}
        return {"sm_mhz": float(np.median(sm)), "sm_max_mhz": float(max(mx)), "reasons": sorted(reasons),
                "samples": len(sm)}


_SGS_CHOICE = "color"  # --sgs
_NEWTON_CHOICE = "picard"  # --newton


def _case(cb, name: str, precision: str, scale: int = 1):
    mixed = precision == "mixed"
    if name == "plate":
        case = cb.cases.plate(scale=scale, mixed=mixed)
    elif name == "ramp":
        case = cb.cases.ramp(scale=scale)
        case.cfg.precision = 1 if mixed else 0
    elif name == "sa_plate":
        case = cb.cases.sa_plate(scale=scale, mixed=mixed)
    else:
        case = cb.cases.bump(scale=scale, mixed=mixed)
    if scale != 1:
        case.description += f" (each dimension divided by {scale})"
    if _SGS_CHOICE == "level":
        case.cfg.sgs_ordering = cb.SGS_LEVEL
        case.description += ", level-scheduled SGS (the reference's sweep order)"
    if _NEWTON_CHOICE == "jf":
        case.cfg.newton_operator = cb.NEWTON_JACOBIAN_FREE
        case.description += ", Jacobian-free Newton-Krylov (GMRES) after the limiter freeze"
    return case


def _cfl(cb, case, it):
    return cb.cases.cfl_at(case.cfg, it)


def _prepare(cb, solver, case):
    """The case's CFL ramp from the free stream (iterations 1..R, limiter
    frozen at R): the operating point every timed window starts from."""
    R = max(case.cfg.cfl_ramp_iterations, case.cfg.limiter_freeze, 1)
    for it in range(1, R + 1):
        if it == case.cfg.limiter_freeze:
            solver.freeze_limiter(True)
        solver.newton_step(_cfl(cb, case, it))
    return R


def _config(case, n, faces, nnzb, args, world, kry=None):
    """The workload description both arms print (the driver pairs the arms
    by it)."""
    R = max(case.cfg.cfl_ramp_iterations, case.cfg.limiter_freeze, 1)
    return {"workload": case.description, "case": case.name, "cells": int(n), "faces": int(faces),
            "nnzb": int(nnzb), "block": 6 if case.cfg.turbulence else 5, "precision": "fp64",
            "sgs": "multicolour (GPU) / sequential (CPU reference)", "krylov": "BiCGSTAB rtol 1e-3 max 30",
            "cfl_schedule": f"1->{case.cfg.cfl_max:g} geometric over {case.cfg.cfl_ramp_iterations} iterations, "
                            f"limiter frozen at {case.cfg.limiter_freeze}",
            "iterations_timed": f"{R + args.warmup + 1}..{R + args.warmup + args.steps}",
            "l2": "inputs larger than L2 (Jacobian and fields, no flush)",
            "parallelism": "replicas" if world > 1 else "single GPU"}


# DRAM bytes (read + write) per algorithmic byte of a kernel family from ncu
# captures of the same kernels on smaller meshes, scaled to a full launch by
# the rows it processes: 6x6 FP64 blocks on the SA plate divided by 2 per
# direction (profiles/kernels_sa_plate_scale2_fp64.md), 5x5 on the laminar
# plate divided by 2 (profiles/kernels_plate_scale2_fp64.md).
TRAFFIC_PER_ALG_BYTE = {"sgs": 262.8 / 236.8, "spmv": 103.1 / 102.0}
TRAFFIC_PER_ALG_BYTE_SA = {"sgs": 1.016}


def _roofline(prof: dict, peak: float, peak_kind: str, traffic_table: dict | None = None):
    table_ratio = TRAFFIC_PER_ALG_BYTE if traffic_table is None else traffic_table
    fams = {k: v for k, v in prof.items() if v["launches"] > 0}
    total = sum(v["ms"] for v in fams.values())
    dom = max(fams, key=lambda k: fams[k]["ms"])
    d = fams[dom]
    per_launch_ms = d["ms"] / d["launches"]
    per_launch_bytes = d["bytes"] / d["launches"]
    achieved = per_launch_bytes / (per_launch_ms * 1e-3) / 1e9
    table = {k: {"ms_per_step_share": round(v["ms"] / total, 4), "launches": v["launches"],
                 "gbs": round(v["bytes"] / (v["ms"] * 1e-3) / 1e9, 1) if v["ms"] > 0 else None,
                 "frac": round(v["bytes"] / (v["ms"] * 1e-3) / 1e9 / peak, 3) if v["ms"] > 0 else None}
             for k, v in sorted(fams.items(), key=lambda kv: -kv[1]["ms"])}
    return {"bound": "hbm", "kernel": dom, "achieved": round(achieved, 1), "peak": peak, "unit": "GB/s",
            "frac": round(achieved / peak, 4),
            "peak_source": f"{peak_kind} (MEASURED_PEAKS.json hbm_gbs)" if peak_kind == "measured" else "fallback",
            "bytes_per_launch": per_launch_bytes, "avg_launch_ms": per_launch_ms,
            "traffic": (round(per_launch_bytes * table_ratio[dom]) if dom in table_ratio else None),
            "families": table}


def max_over_ranks(ms: float, dist_mod, device: str) -> float:
    """The slowest rank's time (all ranks take part; dist_mod None: one rank)."""
    if dist_mod is None:
        return ms
    import torch
    t = torch.tensor([ms], dtype=torch.float64, device=device)
    dist_mod.all_reduce(t, op=dist_mod.ReduceOp.MAX)
    return float(t.item())


def replica_throughput(world: int, cells: int, steps: int, t_max_ms: float) -> float:
    """Whole-job Mcell-iter/s of `world` independent replicas of `cells`
    cells that each ran `steps` iterations, timed by the slowest rank."""
    return world * cells * steps / (t_max_ms * 1e-3) / 1e6


# ------------------------------------------------------------------ CPU side
def _reference_built() -> bool:
    """Whether the reference's CPU build, which the CPU samples run, is here."""
    import __graft_entry__ as ge
    refh, _ = ge.load_oracle()
    return refh.available()


def _cpu_sample(case_name: str, scale: int, warmup: int, steps: int, step_cb=None):
    """The reference's CPU implementation on a bounded sample of the
    workload: the same case with each mesh dimension divided by `scale`,
    built by the reference's own preprocessing (oracle refh.RefMesh), run
    through the case's CFL ramp to the same operating point, then `warmup`
    and `steps` timed Newton iterations.  The reference solver is used where
    the reference has the physics (Euler, laminar Navier-Stokes); its
    Spalart-Allmaras module does not compile (a header it includes is not in
    the repository), so the turbulent case runs the oracle's C restatement
    of it.  Single-threaded: the reference solver has no threading and its
    only parallelism, MPI domain decomposition, is not available here.
    Returns (seconds per step list, description, kind, mesh cells)."""
    import __graft_entry__ as ge
    cb = ge.load_package()  # configurations only: the product library is not loaded
    refh, port = ge.load_oracle()
    case = _case(cb, case_name, "fp64", scale)
    mesh = refh.RefMesh(case.spec)
    if case.cfg.turbulence:
        solver, kind = port.PortSolver(mesh, case.cfg, case.bcs), "port"
    else:
        solver, kind = refh.RefSolver(mesh, case.cfg, case.bcs), "reference"
    solver.set_state(cb.cases.freestream_state(case, mesh.n_cells))
    R = _prepare(cb, solver, case)
    it = R
    for _ in range(warmup):
        it += 1
        solver.newton_step(_cfl(cb, case, it))
    times = []
    for _ in range(steps):
        it += 1
        t0 = time.perf_counter()
        solver.newton_step(_cfl(cb, case, it))
        times.append(time.perf_counter() - t0)
        if step_cb:
            step_cb(times[-1])
    desc = (f"iterations {R + warmup + 1}..{R + warmup + steps} (after the CFL ramp) of the same case on its mesh "
            f"divided by {scale} per direction ({mesh.n_cells} cells, built by the reference's preprocessing), "
            f"{'the C restatement of the reference solver with the Spalart-Allmaras terms' if kind == 'port' else 'the reference solver built from its sources'}, "
            f"one core")
    return times, desc, kind, mesh.n_cells


def run_reference(args):
    """The reference arm: no product library is loaded.  Each step is one
    Newton iteration of the bounded sample (_cpu_sample: the workload's
    case at 1/`ref_scale` per direction, CFL ramp to the same operating
    point); Mcell-iter/s is intensive, so the sample's rate stands for the
    workload's."""
    world, rank, local = _dist()
    if rank != 0:
        return
    import __graft_entry__ as ge
    refh, port = ge.load_oracle()
    if not refh.available() or not port.available():
        print(json.dumps({"impl": "reference", "unavailable": "oracle/_ref libraries were not built"}))
        return
    cb = ge.load_package()
    times, desc, kind, n_sample = _cpu_sample(args.case, args.ref_scale * args.scale, args.warmup, args.steps)
    dt = float(sum(times))
    value = n_sample * args.steps / dt / 1e6
    case = _case(cb, args.case, "fp64", args.scale)
    cells, faces, nnzb = _workload_sizes(cb, case)
    line = {"impl": "reference", "metric": METRIC, "value": round(value, 5), "unit": UNIT, "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(dt / args.steps * 1e3, 3),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": _config(case, cells, faces, nnzb, args, world),
            "cpu_baseline": {"value": round(value, 5), "unit": UNIT, "cores": 1, "kind": kind, "sample": desc},
            "e2e": {"value": round(value, 5), "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line))


def _workload_sizes(cb, case):
    """Cells, faces and BSR blocks of a case without building its mesh:
    hex blocks have n = nx ny nz cells, 2(nx ny + ny nz + nx nz) boundary
    faces and (6n - boundary) / 2 interior faces; the tet meshes split each
    hex into 6 (4 faces per cell, two triangles per boundary quad); one
    block row per cell plus two blocks per interior face."""
    s = case.spec
    nx, ny, nz = s.nx, s.ny, s.nz
    fb = 2 * (nx * ny + ny * nz + nx * nz)
    if s.kind == 2:
        n = 6 * nx * ny * nz
        fb *= 2
        fi = (4 * n - fb) // 2
    else:
        n = nx * ny * nz
        fi = (6 * n - fb) // 2
    return n, fi + fb, n + 2 * fi


# ------------------------------------------------------------------ GPU side
def _train_sa_network(cb, device):
    """The learned guess for the SA plate, trained on the GPU by the
    library's own tcgen05 kernels on (features, dU) samples the solver writes
    while running the training flows (cases.sa_training_flows: SA on the
    laminar plate's mesh over M x Re_L); untimed."""
    t0 = time.perf_counter()
    flows = cb.cases.sa_training_flows()
    ds = cb.Dataset(6, 3_000_000, device=device)
    runs = []
    for case in flows:
        mesh = cb.HostMesh(case.spec)
        stride = max(1, (mesh.n_cells * case.iterations) // 300_000)
        with cb.Solver(mesh, case.cfg, case.bcs, device=device) as s:
            s.init_fields()
            s.attach_dataset(ds, stride)
            r = s.run_steady()
        runs.append({"mach": round(case.extra["mach"], 3), "Re": case.extra["Re"], "iterations": int(r.iterations)})
    t_collect = time.perf_counter() - t0
    net = cb.Mlp(6, seed=5, device=device)
    t1 = time.perf_counter()
    net.train(ds, epochs=40, batch=8192, lr=1e-3)
    loss = net.train(ds, epochs=20, batch=8192, lr=2e-4)
    info = {"samples": len(ds), "snapshots": sum(r["iterations"] for r in runs), "flows": len(runs),
            "mesh": f"laminar plate mesh / 4 per direction ({cb.HostMesh(flows[0].spec).n_cells} cells)",
            "epochs": "40 at lr 1e-3 + 20 at lr 2e-4", "final_loss": round(loss, 6),
            "collect_s": round(t_collect, 2), "train_s": round(time.perf_counter() - t1, 3)}
    ds.close()
    return net, info


def _timed_leg(cb, torch, s, case, stream, args, pg, local, it0, clocks=False):
    """W warm-up and K timed Newton iterations from iteration it0; CUDA
    events on the solver stream, barrier + synchronize on both sides."""
    it = it0
    kry = []
    for _ in range(args.warmup):
        it += 1
        s.newton_step(_cfl(cb, case, it))
    U_warm = s.get(cb.FIELD_U)

    def barrier():
        if pg is not None:
            pg.barrier()
        torch.cuda.synchronize()

    launches0 = s.launch_count()
    barrier()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    clk = Clocks(local) if clocks else None
    if clk:
        clk.__enter__()
    ev0.record(stream)
    for _ in range(args.steps):
        it += 1
        kry.append(int(s.newton_step(_cfl(cb, case, it)).krylov_iterations))
    ev1.record(stream)
    torch.cuda.synchronize()
    if clk:
        clk.__exit__()
    ms = ev0.elapsed_time(ev1)
    barrier()
    return {"ms": ms, "launches": s.launch_count() - launches0, "krylov": kry, "U_warm": U_warm,
            "it_warm": it0 + args.warmup, "clocks": clk.summary() if clk else None}


def run_ours(args):
    world, rank, local = _dist()
    import torch
    import __graft_entry__ as ge
    cb = ge.load_package()
    torch.cuda.set_device(local)
    pg = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=300))
        pg = dist
    case = _case(cb, args.case, "fp64", args.scale)
    case.cfg.krylov_loop = cb.KRYLOV_HOST_LOOP if args.krylov_loop == "host" else cb.KRYLOV_DEVICE_LOOP
    t0 = time.perf_counter()
    mesh = cb.HostMesh(case.spec)
    t_mesh = time.perf_counter() - t0
    n = mesh.n_cells
    t0 = time.perf_counter()
    s = cb.Solver(mesh, case.cfg, case.bcs, device=local)
    t_setup = time.perf_counter() - t0
    s.init_fields()
    stream = torch.cuda.ExternalStream(s.stream(), device=local)
    R = _prepare(cb, s, case)

    # ------------------------------------------------- FP64: the product path
    leg = _timed_leg(cb, torch, s, case, stream, args, pg, local, R, clocks=True)
    t_max = max_over_ranks(leg["ms"], pg, f"cuda:{local}")
    value = replica_throughput(world, n, args.steps, t_max)
    U_warm, it_warm = leg["U_warm"], leg["it_warm"]

    # ------------------------------------------------- kernel-family events
    # The timed iterations again from the same state with a CUDA event pair
    # around every kernel family on the solver's stream (the Krylov loop then
    # runs host-driven so that each launch is bracketed).
    s.set_state(U_warm)
    s.profile(True)
    kry_prof = []
    pe0, pe1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    pe0.record(stream)
    for k in range(args.steps):
        kry_prof.append(int(s.newton_step(_cfl(cb, case, it_warm + k + 1)).krylov_iterations))
    pe1.record(stream)
    torch.cuda.synchronize()
    prof = s.profile_read()
    s.profile(False)
    prof_ms = pe0.elapsed_time(pe1)
    if pg is not None:
        pg.barrier()

    # ---------------------------------------------------- end to end (C ABI)
    # The same K iterations from the same state, each with the state copied
    # in from pinned host memory and the updated state read back.
    s.set_state(U_warm)
    U_host = torch.empty(s.field_size(cb.FIELD_U), dtype=torch.float64, pin_memory=True)
    U_host.numpy()[:] = U_warm
    import ctypes as C
    lib = cb.lib()
    ptr = C.cast(U_host.data_ptr(), C.POINTER(C.c_double))
    if pg is not None:
        pg.barrier()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for k in range(args.steps):
        cb.check(lib.cfdg_solver_set_state(s._h, ptr, n))
        s.newton_step(_cfl(cb, case, it_warm + k + 1))
        cb.check(lib.cfdg_solver_get_field(s._h, cb.FIELD_U, ptr, U_host.numel()))
    e1.record(stream)
    torch.cuda.synchronize()
    e2e_ms = max_over_ranks(e0.elapsed_time(e1), pg, f"cuda:{local}")
    e2e_value = replica_throughput(world, n, args.steps, e2e_ms)
    bytes_state = U_host.numel() * 8
    nnzb, faces = s.nnzb, mesh.n_faces
    s.close()

    legs = {"fp64": {"value": round(value, 4), "ms_per_step": round(t_max / args.steps, 3),
                     "krylov_iterations_per_step": round(float(np.mean(leg["krylov"])), 2)}}
    if world == 1 and not args.no_mixed:
        # mixed precision and mixed + learned guess: each its own run from the
        # free stream (FP64 until the freeze), timed on the same iterations
        net, train_info = (None, None)
        if not args.no_learned:
            net, train_info = _train_sa_network(cb, local) if case.cfg.turbulence else (None, None)
        for name, learned in (("mixed", False), ("mixed_learned", True)):
            if learned and net is None:
                continue
            c = _case(cb, args.case, "mixed", args.scale)
            with cb.Solver(mesh, c.cfg, c.bcs, device=local) as sm:
                sm.init_fields()
                if learned:
                    sm.attach_guess(net)
                st = torch.cuda.ExternalStream(sm.stream(), device=local)
                Rm = _prepare(cb, sm, c)
                lg = _timed_leg(cb, torch, sm, c, st, args, None, local, Rm)
                legs[name] = {"value": round(replica_throughput(1, n, args.steps, lg["ms"]), 4),
                              "ms_per_step": round(lg["ms"] / args.steps, 3),
                              "krylov_iterations_per_step": round(float(np.mean(lg["krylov"])), 2)}
        if train_info:
            legs["mixed_learned"]["training"] = train_info
        if net is not None:
            net.close()

    if rank == 0:
        peak, peak_kind = _peaks()
        roof = _roofline(prof, peak, peak_kind, TRAFFIC_PER_ALG_BYTE_SA if case.cfg.turbulence else None)
        roof["measured_in"] = (f"iterations {it_warm + 1}..{it_warm + args.steps} replayed from the same state with "
                               f"CUDA events around each kernel family and a host-driven Krylov loop "
                               f"({prof_ms / args.steps:.3f} ms per step, {float(np.mean(kry_prof)):.2f} Krylov "
                               f"iterations per step)")
        sizes = _workload_sizes(cb, case)
        assert sizes == (n, faces, nnzb), (sizes, (n, faces, nnzb))
        cfg_out = _config(case, n, faces, nnzb, args, world)
        line = {"metric": METRIC, "value": round(value, 4), "unit": UNIT, "n_gpus": world, "steps": args.steps,
                "warmup": args.warmup, "ms_per_step": round(t_max / args.steps, 3), "higher_is_better": True,
                "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
                "config": cfg_out, "clocks": leg["clocks"], "gpu_launches": int(leg["launches"]),
                "krylov_iterations_per_step": legs["fp64"]["krylov_iterations_per_step"],
                "legs": legs,
                "e2e": {"value": round(e2e_value, 4), "unit": UNIT, "h2d_bytes_per_step": bytes_state,
                        "d2h_bytes_per_step": bytes_state, "steps": args.steps,
                        "iterations": f"{it_warm + 1}..{it_warm + args.steps}"},
                "roofline": roof,
                "setup_s": {"mesh": round(t_mesh, 2), "solver": round(t_setup, 2)}}
        cpu = not args.no_cpu_baseline and _reference_built()
        if not cpu and not args.no_cpu_baseline:
            line["cpu_baseline"] = {"unavailable": "the reference's CPU build is not here"}
        if cpu and world == 1:
            times, desc, kind, n_s = _cpu_sample(args.case, args.cpu_scale * args.scale, 1, args.cpu_steps)
            v = n_s * len(times) / sum(times) / 1e6
            line["cpu_baseline"] = {"value": round(v, 5), "unit": UNIT, "cores": 1, "kind": kind, "sample": desc}
        if not args.no_converge and world == 1:
            line["time_to_1e8"] = _time_to_converge(cb, args.converge_scale, cpu)
            line["time_to_1e8_plate"] = _time_to_converge_plate(cb, args.plate_converge_scale, cpu)
        print(json.dumps(line))
    if pg is not None:
        pg.destroy_process_group()


def _time_to_converge(cb, scale: int, cpu: bool = True):
    """Wall time of run_steady to a 1e-8 residual drop on the bump: FP64,
    mixed, mixed + learned guess (network trained first on other flows),
    each its own run from the free stream; the limiter freezes at the end of
    the CFL ramp and the mixed runs use the FP64 matrix until then, so all
    three solve the same frozen problem and their converged fields are
    compared directly.  With `cpu`, the reference CPU solver's seconds per
    iteration on the same mesh times the FP64 run's iteration count (same
    algorithm and schedule: an extrapolated time to 1e-8)."""
    t0 = time.perf_counter()
    ds = cb.Dataset(5, 6_000_000)
    collect = []
    for mach in (0.8, 0.9):
        case = cb.cases.bump(scale=2 * scale, mixed=True, mach=mach, iterations=2000)
        mesh = cb.HostMesh(case.spec)
        stride = max(1, (mesh.n_cells * 1000) // 3_000_000)
        with cb.Solver(mesh, case.cfg, case.bcs) as s:
            s.init_fields()
            s.attach_dataset(ds, stride)
            r = s.run_steady()
            collect.append({"mach": mach, "cells": mesh.n_cells, "iterations": int(r.iterations),
                            "converged": bool(r.converged)})
    t_collect = time.perf_counter() - t0
    net = cb.Mlp(5, seed=5)
    t1 = time.perf_counter()
    # Adam at lr 1e-3, then a lower-rate phase (the Adam moments carry over)
    net.train(ds, epochs=40, batch=8192, lr=1e-3)
    loss = net.train(ds, epochs=20, batch=8192, lr=2e-4)
    t_train = time.perf_counter() - t1
    n_samples = len(ds)
    ds.close()
    case = cb.cases.bump(scale=scale, iterations=4000)
    mesh = cb.HostMesh(case.spec)
    out = {"workload": f"transonic Euler bump M=0.85, {mesh.n_cells} tets (160x80x80x6 / {scale}^3), "
                       f"run_steady to a 1e-8 drop of max(mass, |momentum|, energy) L2 vs its running maximum",
           "training": {"samples": n_samples, "epochs": "40 at lr 1e-3 + 20 at lr 2e-4",
                        "final_loss": round(loss, 6), "collect_s": round(t_collect, 2), "train_s": round(t_train, 3),
                        "runs": collect}}
    fields = {}
    for name, prec, learned in (("fp64", 0, False), ("mixed", 1, False), ("mixed_learned", 1, True)):
        c = cb.cases.bump(scale=scale, iterations=4000)
        c.cfg.precision = prec
        with cb.Solver(mesh, c.cfg, c.bcs) as s:
            s.init_fields()
            if learned:
                s.attach_guess(net)
            r = s.run_steady()
            fields[name] = s.get(cb.FIELD_U).reshape(5, -1)
        out[name] = {"seconds": round(r.seconds, 3), "iterations": int(r.iterations), "converged": bool(r.converged),
                     "rel": float(r.rel), "krylov_iterations": int(r.krylov_iterations_total)}
    net.close()
    ref = fields["fp64"]
    for name in ("mixed", "mixed_learned"):
        out[name]["field_rel_l2_vs_fp64"] = [
            float("%.3g" % (np.linalg.norm(fields[name][v] - ref[v]) / max(np.linalg.norm(ref[v]), 1e-300)))
            for v in (0, 1, 2, 4)]
    out["field_components"] = "rho, rho u, rho v, rho E"
    out["speedup_mixed_learned_vs_fp64"] = round(out["fp64"]["seconds"] / out["mixed_learned"]["seconds"], 3)
    if cpu:
        import __graft_entry__ as ge
        refh, _ = ge.load_oracle()
        if refh.available():
            c = cb.cases.bump(scale=scale, iterations=4000, mixed=False)
            rsol = refh.RefSolver(mesh, c.cfg, c.bcs)
            rsol.set_state(cb.cases.freestream_state(c, mesh.n_cells))
            rsol.newton_step(cb.cases.cfl_at(c.cfg, 1))  # first iteration outside the sample
            t_r = time.perf_counter()
            for k in range(2):
                rsol.newton_step(cb.cases.cfl_at(c.cfg, k + 2))
            del rsol
            spi = (time.perf_counter() - t_r) / 2
            out["reference_cpu"] = {"seconds_per_iteration": round(spi, 3), "cores": 1,
                                    "sample": "iterations 2-3 of the same mesh, single-threaded reference build",
                                    "extrapolated_seconds": round(spi * out["fp64"]["iterations"], 1),
                                    "speedup_mixed_learned_vs_reference": round(
                                        spi * out["fp64"]["iterations"] / out["mixed_learned"]["seconds"], 1)}
    return out


# Linear tolerance of the plates' time-to-1e-8 runs.  Their Newton rate is
# set by a slow mass (pressure) mode, not by the accuracy of the linear
# solves: on the SA plate at 1/4 size, rtol 1e-3 / 1e-2 / 1e-1 reached 1e-8
# in 18,871 / 18,874 / 19,487 Newton iterations and 57 / 40 / 25 s (23, 15
# and 8 Krylov iterations per step).  The converged state does not depend
# on it.
PLATE_LIN_RTOL = 0.1


def _time_to_converge_plate(cb, scale: int, cpu: bool = True, ser: float = 1000.0):
    """Wall time of run_steady to a 1e-8 residual drop on the laminar plate
    (256x128x32 hex divided by `scale` per direction): FP64 and mixed
    precision, each from the free stream with the Picard operator and the
    multicolour SGS (BiCGSTAB rtol PLATE_LIN_RTOL), the limiter frozen at the
    end of the CFL ramp and the CFL raised after it by switched evolution
    relaxation up to `ser`; with `cpu`, the reference CPU solver's seconds
    per iteration on the same mesh (its own linear settings) times the FP64
    run's iteration count (an extrapolated time)."""
    case = cb.cases.plate(scale=scale, iterations=40000)
    mesh = cb.HostMesh(case.spec)
    out = {"workload": f"laminar flat plate M=0.5 Re_L=1e5, {mesh.n_cells} hex (256x128x32 / {scale}^3), "
                       f"run_steady to a 1e-8 drop of max(mass, |momentum|, energy) L2 vs its running maximum",
           "schedule": f"CFL 1->100 over 50 iterations, then switched evolution relaxation up to {ser:g}; "
                       f"limiter frozen at iteration 50; Picard operator, multicolour SGS, BiCGSTAB rtol "
                       f"{PLATE_LIN_RTOL:g} max 30"}
    fields = {}
    for name, prec in (("fp64", 0), ("mixed", 1)):
        c = cb.cases.plate(scale=scale, iterations=40000)
        c.cfg.precision = prec
        c.cfg.cfl_ser_max = ser
        c.cfg.lin_rel_tol = PLATE_LIN_RTOL
        with cb.Solver(mesh, c.cfg, c.bcs) as s:
            s.init_fields()
            r = s.run_steady()
            fields[name] = s.get(cb.FIELD_U).reshape(5, -1)
        out[name] = {"seconds": round(r.seconds, 3), "iterations": int(r.iterations), "converged": bool(r.converged),
                     "rel": float(r.rel), "krylov_iterations": int(r.krylov_iterations_total)}
    ref = fields["fp64"]
    out["mixed"]["field_rel_l2_vs_fp64"] = [
        float("%.3g" % (np.linalg.norm(fields["mixed"][v] - ref[v]) / max(np.linalg.norm(ref[v]), 1e-300)))
        for v in (0, 1, 2, 4)]
    out["field_components"] = "rho, rho u, rho v, rho E"
    if cpu:
        import __graft_entry__ as ge
        refh, _ = ge.load_oracle()
        if refh.available():
            c = cb.cases.plate(scale=scale, iterations=40000)
            rsol = refh.RefSolver(mesh, c.cfg, c.bcs)
            rsol.set_state(cb.cases.freestream_state(c, mesh.n_cells))
            rsol.newton_step(cb.cases.cfl_at(c.cfg, 1))  # first iteration outside the sample
            t_r = time.perf_counter()
            for k in range(2):
                rsol.newton_step(cb.cases.cfl_at(c.cfg, k + 2))
            del rsol
            spi = (time.perf_counter() - t_r) / 2
            out["reference_cpu"] = {"seconds_per_iteration": round(spi, 3), "cores": 1,
                                    "sample": "iterations 2-3 of the same mesh, single-threaded reference build",
                                    "extrapolated_seconds": round(spi * out["fp64"]["iterations"], 1)}
    return out


def _time_to_converge_sa(cb, scale: int, device: int = 0):
    """Wall time of run_steady to a 1e-8 residual drop on the
    Spalart-Allmaras plate (384x192x56 hex divided by `scale` per direction):
    plain FP64, mixed precision and mixed precision + learned guess (the
    network trained first on the SA training flows), each from the free
    stream with the Picard operator, the multicolour SGS (BiCGSTAB rtol
    PLATE_LIN_RTOL), CFL 1->100 and the limiter frozen at the ramp's end;
    converged rho, u, p and nu_tilde are compared with the FP64 run's."""
    net, train = _train_sa_network(cb, device)
    case = cb.cases.sa_plate(scale=scale, iterations=60000)
    mesh = cb.HostMesh(case.spec)
    out = {"workload": f"Spalart-Allmaras flat plate M=0.2 Re_L=5e6, {mesh.n_cells} hex (384x192x56 / {scale}^3), "
                       f"run_steady to a 1e-8 drop of max(mass, |momentum|, energy, nu_tilde) L2 vs its running "
                       f"maximum",
           "schedule": f"CFL 1->100 over 50 iterations; limiter frozen at iteration 50; Picard operator, "
                       f"multicolour SGS, BiCGSTAB rtol {PLATE_LIN_RTOL:g} max 30",
           "training": train}
    fields = {}
    for name, prec, learned in (("fp64", 0, False), ("mixed", 1, False), ("mixed_learned", 1, True)):
        c = cb.cases.sa_plate(scale=scale, iterations=60000, mixed=bool(prec))
        c.cfg.lin_rel_tol = PLATE_LIN_RTOL
        with cb.Solver(mesh, c.cfg, c.bcs, device=device) as s:
            s.init_fields()
            if learned:
                s.attach_guess(net)
            r = s.run_steady()
            fields[name] = s.get(cb.FIELD_U).reshape(6, -1)
        out[name] = {"seconds": round(r.seconds, 3), "iterations": int(r.iterations), "converged": bool(r.converged),
                     "rel": float(r.rel), "krylov_iterations": int(r.krylov_iterations_total)}
    net.close()

    def prim(U):
        rho = U[0]
        return {"rho": rho, "u": U[1] / rho, "p": 0.4 * (U[4] - 0.5 * (U[1] ** 2 + U[2] ** 2 + U[3] ** 2) / rho),
                "nu_tilde": U[5] / rho}
    ref = prim(fields["fp64"])
    for name in ("mixed", "mixed_learned"):
        q = prim(fields[name])
        out[name]["field_rel_l2_vs_fp64"] = {
            k: float("%.3g" % (np.linalg.norm(q[k] - ref[k]) / max(np.linalg.norm(ref[k]), 1e-300))) for k in q}
    out["speedup_mixed_learned_vs_fp64"] = round(out["fp64"]["seconds"] / out["mixed_learned"]["seconds"], 3)
    return out


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--case", default="sa_plate", choices=["sa_plate", "plate", "ramp", "bump"])
    ap.add_argument("--scale", type=int, default=1, help="divide each mesh dimension (profiling runs)")
    ap.add_argument("--ref-scale", type=int, default=4,
                    help="mesh divisor per direction of the reference arm's bounded sample")
    ap.add_argument("--cpu-scale", type=int, default=8, help="mesh divisor of the cpu_baseline sample")
    ap.add_argument("--cpu-steps", type=int, default=3)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-mixed", action="store_true", help="skip the mixed and mixed + learned legs")
    ap.add_argument("--no-learned", action="store_true", help="skip the learned-guess leg")
    ap.add_argument("--no-converge", action="store_true", help="skip the time-to-1e-8 runs")
    ap.add_argument("--converge-scale", type=int, default=2, help="bump mesh divisor of the time-to-1e-8 runs")
    ap.add_argument("--converge-only", action="store_true",
                    help="run only the time-to-1e-8 comparison (one JSON line with time_to_1e8); with "
                         "--converge-scale 1 the full 6,144,000-tet bump")
    ap.add_argument("--converge-case", default="bump", choices=["bump", "plate", "sa_plate"],
                    help="workload of --converge-only: the tet bump (FP64, mixed, mixed + learned), the "
                         "laminar plate (FP64, mixed; --converge-scale 1 = 1,048,576 cells) or the SA plate "
                         "(FP64, mixed, mixed + learned)")
    ap.add_argument("--plate-converge-scale", type=int, default=2,
                    help="laminar plate mesh divisor of the default run's time-to-1e-8 leg")
    ap.add_argument("--krylov-loop", default="device", choices=["device", "host"],
                    help="BiCGSTAB driver of the timed steps (host: one launch sequence per iteration, "
                         "e.g. for a profiler that does not see kernels inside conditional graph nodes)")
    ap.add_argument("--sgs", default="color", choices=["color", "level"],
                    help="SGS ordering of the measured legs: multicolour (default) or level-scheduled (the "
                         "reference's sequential order, one cooperative launch per sweep)")
    ap.add_argument("--newton", default="picard", choices=["picard", "jf"],
                    help="Newton operator of the measured legs: the assembled Picard matrix (the reference's) "
                         "or the Jacobian-free product (profiling its kernels)")
    args = ap.parse_args()
    global _SGS_CHOICE, _NEWTON_CHOICE
    _SGS_CHOICE = args.sgs
    _NEWTON_CHOICE = args.newton
    if args.impl == "reference":
        run_reference(args)
    elif args.converge_only:
        import __graft_entry__ as ge
        cb = ge.load_package()
        t0 = time.perf_counter()
        if args.converge_case == "plate":
            out = _time_to_converge_plate(cb, args.converge_scale, not args.no_cpu_baseline)
            key = "time_to_1e8_plate"
        elif args.converge_case == "sa_plate":
            out = _time_to_converge_sa(cb, args.converge_scale)
            key = "time_to_1e8_sa_plate"
        else:
            out = _time_to_converge(cb, args.converge_scale, not args.no_cpu_baseline)
            key = "time_to_1e8"
        print(json.dumps({"metric": METRIC, key: out, "wall_s": round(time.perf_counter() - t0, 1)}))
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
