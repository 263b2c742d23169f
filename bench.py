#!/usr/bin/env python3
"""Benchmark of the projection time step (cell-steps/s at Poisson residual 1e-8).

Workload (default "c2"): the 512x256x64 uniform MAC grid over [0,32]x[0,16]x[0,4],
cylinder D=1 at (8,8), Re 200, dt 0.002, the reference's own boundary conditions and
initial state (u=1, v=w=0), Jacobi-scaled BiCGSTAB to relative residual 1e-8, FP64.
A step is one projection step (convection-diffusion, Poisson solve, correction + DFIB
forcing + drag, ghost fill).  Inputs (~1.5 GB of fields and Krylov vectors) are far
larger than the 129 MB L2, so no flush is needed between steps.

One JSON line on rank 0.  value: FP64 cell-steps/s over exactly --steps steps after
--warmup steps, CUDA events on the library's stream, max over ranks (replicas: the
path does not shard).  Beside it: the FP32+FP64-refined mode and red-black SOR on the
same workload, e2e through the C ABI with host buffers, per-kernel live timing for the
roofline, the CPU baseline (the reference's own OpenMP build, bounded sample) and SM
clocks sampled during the timed region.

--impl reference times the reference's own CPU implementation (oracle/_ref, built
from the reference sources) on the host cores for the same workload and metric.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import threading
import time
from pathlib import Path

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

WORKLOADS = {
    # plain FP64 on the GPU at scale (8.4M cells)
    "c2": dict(nx=512, ny=256, nz=64, lx=32.0, ly=16.0, lz=4.0, cx=8.0, cy=8.0, Re=200.0, dt=0.002),
    # the reference's CPU-runnable case
    "c1": dict(nx=96, ny=48, nz=4, lx=24.0, ly=12.0, lz=1.0, cx=6.0, cy=6.0, Re=100.0, dt=0.005),
    # mixed-precision scale case (67M cells)
    "c3": dict(nx=1024, ny=512, nz=128, lx=32.0, ly=16.0, lz=4.0, cx=8.0, cy=8.0, Re=300.0, dt=0.001),
    # adjoint case (1M cells)
    "c4": dict(nx=256, ny=128, nz=32, lx=24.0, ly=12.0, lz=2.0, cx=6.0, cy=6.0, Re=100.0, dt=0.004),
    # combined stress case (113M cells)
    "c5": dict(nx=1536, ny=768, nz=96, lx=48.0, ly=24.0, lz=3.0, cx=12.0, cy=12.0, Re=300.0, dt=0.001),
    # the reference's own default case (src/CFD_MX.cpp:23-27, structureGrid.hpp:20-40,
    # setEta.hpp:145, 0_1_SimulationVariable.hpp:61): its stretched SML grid of 190x210x40,
    # SPE BiCGSTAB to its default 1e-3
    "ref": dict(nx=190, ny=210, nz=40, lx=17.0, ly=12.0, lz=3.0, cx=6.5, cy=6.0, Re=40.0, dt=0.002, grid="sml",
                solver="bicgstab", tol=1e-3),
}


def workload(wl):
    """(Solver keyword arguments of the case, the solver of its FP64 run, its tolerance)."""
    cfg = dict(WORKLOADS[wl])
    return cfg, cfg.pop("solver", "jacobi"), cfg.pop("tol", TOL)


def l2_note(wl):
    """The state a step reads (11 padded FP64 fields, ~10 compact FP64 vectors) against L2."""
    cfg, _, _ = workload(wl)
    pad = (cfg["nx"] + 4) * (cfg["ny"] + 4) * (cfg["nz"] + 4)
    gb = (11 * pad + 10 * cfg["nx"] * cfg["ny"] * cfg["nz"]) * 8 / 1e9
    return f"state ~{gb:.2g} GB > 129 MB L2 each step, no flush"


def config_of(wl):
    cfg, solver, tol = workload(wl)
    return {"workload": wl, **cfg, "solver": {"jacobi": "jacobi_bicgstab", "bicgstab": "spe_bicgstab"}[solver],
            "tol": tol}


def metric(wl):
    _, solver, tol = workload(wl)
    if (solver, tol) == ("jacobi", TOL):
        return METRIC
    name = {"jacobi": "Jacobi-BiCGSTAB", "bicgstab": "SPE-BiCGSTAB"}[solver]
    return f"cell-steps/s @resid {tol:g} (FP64 {name} projection step)"


TOL = 1e-8
FALLBACK_HBM_GBS = 6800.0

# algorithmic bytes per interior cell and launch (one word per array read or written,
# neighbours assumed cached), FP64 = 8 B, FP32 = 4 B
KERNEL_WORDS = {
    # FP64 iteration: five kernels, 19 words per cell
    "bicg_ap64": 3,    # read p1, r0; write ap
    "bicg_s64": 3,     # read r1, ap; write s
    "bicg_as64": 2,    # read s; write as
    "bicg_xr64": 7,    # read x, p1, s, as, r0; write x, r1
    "bicg_p64": 4,     # read r1, p1, ap; write p1
    # FP32 inner iteration: three fused kernels, 17 words per cell
    "bicg_pap32": 6,   # read r1, p, ap, r0; write p', ap'
    "bicg_sas32": 4,   # read r1, ap; write s, as
    "bicg_xr32": 7,    # read x, p, s, as, r0; write x, r1
    # FP32 iteration right-preconditioned by the multigrid V-cycle: five kernels, 21 words
    # per cell beside the two V-cycles (~17 words each over all levels, timed as mg_vcycle)
    "bicgp_p32": 4,    # read r1, p, v; write p
    "bicgp_v32": 3,    # read ph, r0; write v
    "bicgp_s32": 3,    # read r1, v; write s
    "bicgp_t32": 3,    # read sh, s; write t
    "bicgp_xr32": 8,   # read x, ph, sh, s, t, r0; write x, r1
    # CG (the reference's cg.hpp method): FP64 three kernels, 11 words; FP32 sweeps two, 10
    "cg_q64": 2,       # read p; write q
    "cg_xr64": 6,      # read x, p, r, q; write x, r
    "cg_p64": 3,       # read r, p; write p
    "cg_pq32": 4,      # read r, p; write p', q
    "cg_xr32": 6,      # read x, p, r, q; write x, r
    # the same preconditioned iteration in FP64 (fp64_mg)
    "bicgp_p64": 4, "bicgp_v64": 3, "bicgp_s64": 3, "bicgp_t64": 3, "bicgp_xr64": 8,
}

# The one-launch forms of those iterations: a launch is a chunk of iterations, so words an
# iteration, those of the kernels above that they replace (the vectors of these grids live in L2, and
# cg_loop32's on chip, so the algorithmic rate may pass the HBM peak)
LOOP_WORDS = {"bicg_loop64": 19, "cg_loop64": 11, "cg_loop32": 10}


# FP64 flops per interior cell and launch of the FP64 iteration kernels (an FMA counts 2):
# SpMV 1 mul + 6 FMA, each dot 1 FMA, each axpy-like update 1 FMA per term
KERNEL_FP64_FLOPS = {"bicg_ap64": 15, "bicg_s64": 2, "bicg_as64": 17, "bicg_xr64": 10, "bicg_p64": 4,
                     "cg_q64": 15, "cg_xr64": 6, "cg_p64": 2}
LOOP_FP64_FLOPS = {"bicg_loop64": 48, "cg_loop64": 23}  # an iteration


def launch_units(prof, iters, per_launch, per_iteration):
    """Kernels of a profile that a table counts, with its entry per launch: the one-launch
    iterations' entries times the profile's Krylov iterations a launch."""
    out = {}
    for k, (ms, n) in prof.items():
        if n > 0 and ms > 0:
            if k in per_launch:
                out[k] = per_launch[k]
            elif k in per_iteration and iters:
                out[k] = per_iteration[k] * iters / n
    return out



FP_PEAK_SRC = ROOT / "bench_fp_peak.cu"
FP_PEAK_EXE = ROOT / "bench_fp_peak"


def build_fp_peak(force=False):
    """Compile the FMA throughput probe beside this script (sm_103a); returns its path."""
    if force or not FP_PEAK_EXE.exists() or FP_PEAK_EXE.stat().st_mtime < FP_PEAK_SRC.stat().st_mtime:
        from cfd_nssolver_forhpc_flowpassingcylinder_gb300.build import nvcc
        subprocess.run([nvcc(), "-gencode", "arch=compute_103a,code=sm_103a", "-O3", str(FP_PEAK_SRC), "-o",
                        str(FP_PEAK_EXE)], check=True, capture_output=True)
    return FP_PEAK_EXE


def alu_peaks():
    """FP64/FP32 FMA throughput of this GPU, measured by the probe bench_fp_peak.cu."""
    try:
        exe = build_fp_peak()
        out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60).stdout
        return json.loads(out.strip().splitlines()[-1])
    except Exception as e:  # binary missing or no GPU
        return {"error": str(e)}


def alu_roofline(prof, cells, fp_peak, iters=0):
    flops = launch_units(prof, iters, KERNEL_FP64_FLOPS, LOOP_FP64_FLOPS)
    if not flops or not fp_peak.get("fp64_tflops"):
        return None
    dom = max(flops, key=lambda k: prof[k][0])
    ms, n = prof[dom]
    achieved = flops[dom] * cells / (ms / n / 1e3) / 1e12
    return {"kernel": dom, "bound": "fp64", "achieved": round(achieved, 4), "peak": fp_peak["fp64_tflops"],
            "unit": "TFLOP/s", "frac": round(achieved / fp_peak["fp64_tflops"], 4),
            "peak_kind": "measured (bench_fp_peak FMA chains)"}


# The MIXED step's kernels beside the Krylov sweeps: algorithmic bytes per interior cell
# and launch (one word per array read or written, neighbours cached) and the FP64
# instructions per cell counted in their source (an FMA is one instruction).  Each is set
# against the HBM peak and the measured FP64 instruction rate; the larger fraction names
# its bound.  correct64 pairs two launches (the correction's mean, then x += e).
STEP_KERNELS = {
    "convection_diffusion": (60, 3),  # read u32, v32, w32 (FP32) and u, v, w; write us, vs, ws; 3 DADD
    "update_uf": (64, 6),             # read eta, p, us, vs, ws; write u, v, w; 3 DADD + 3 DFMA (uniform grid)
    "rhs": (32, 7),                   # read us, vs, ws; write b
    "residual64": (20, 3),            # read b, x; write r (FP32); A x in integers: its conversion, the subtraction,
                                      # the norm's DFMA (a solve's first one also the norm of b: 4)
    "correct64": (24, 1),             # read e (mean), then x, e; write x; 1 DADD (the scaling in integers)
    "mirror32": (36, 0),              # read u, v, w; write u32, v32, w32 (integer rounding; padded fields)
}


def step_roofline(prof, cells, npad, hbm_peak, fp_peak):
    """Per MIXED step kernel: average launch, achieved GB/s and FP64 instruction rate, each
    as a fraction of its peak, and the bound the larger one names."""
    f64 = (fp_peak or {}).get("fp64_tflops")
    inst_peak = f64 * 1e12 / 2 if f64 else None  # FMA instructions per second
    out = {}
    for k, (bpc, fpc) in STEP_KERNELS.items():
        ms, n = prof.get(k, (0.0, 0))
        if not n or ms <= 0:
            continue
        n = n / 2 if k == "correct64" else n
        per = ms / n / 1e3
        units = npad if k == "mirror32" else cells
        gbs = bpc * units / per / 1e9
        hf = gbs / hbm_peak
        ff = fpc * cells / per / inst_peak if inst_peak else None
        out[k] = {"avg_launch_us": round(per * 1e6, 2), "launches": n, "achieved_gbs": round(gbs, 1),
                  "hbm_frac": round(hf, 4), "fp64_inst_per_cell": fpc,
                  "fp64_frac": round(ff, 4) if ff is not None else None,
                  "bound": "fp64" if ff is not None and ff > hf else "hbm"}
    return out


def peaks():
    f = ROOT / "MEASURED_PEAKS.json"
    if f.exists():
        d = json.loads(f.read_text())
        return float(d["hbm_gbs"]), "measured"
    return FALLBACK_HBM_GBS, "fallback"


class Clocks:
    """nvidia-smi sampling of SM clocks and throttle reasons during the timed region."""
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device: int):
        self.device = device
        self.rows = []
        self.proc = None

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.device), f"--query-gpu={self.Q}", "--format=csv,noheader,nounits",
                 "-lms", "200"], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except FileNotFoundError:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.rows.append([x.strip() for x in line.split(",")])

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self):
        if not self.rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        sm = [float(r[1]) for r in self.rows if len(r) > 2 and r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in self.rows if len(r) > 2 and r[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[q] for r in self.rows if len(r) >= 9 for q in range(4)
                          if r[5 + q].lower() == "active"})
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(self.rows)}


def _dist():
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return world, rank, local


class Dist:
    def __init__(self):
        self.world, self.rank, self.local = _dist()
        self.pg = None
        if self.world > 1:
            import torch.distributed as tdist
            tdist.init_process_group("nccl" if os.environ.get("BENCH_GLOO") is None else "gloo")
            self.pg = tdist

    def barrier(self):
        if self.pg:
            self.pg.barrier()

    def max(self, x: float) -> float:
        if not self.pg:
            return x
        import torch
        dev = "cuda" if self.pg.get_backend() == "nccl" else "cpu"
        t = torch.tensor([x], dtype=torch.float64, device=dev)
        self.pg.all_reduce(t, op=self.pg.ReduceOp.MAX)
        return float(t.item())

    def close(self):
        if self.pg:
            self.pg.destroy_process_group()


def _timed_steps(s, steps, dist, torch):
    """Exactly `steps` steps between two CUDA events on the solver's stream."""
    stream = torch.cuda.ExternalStream(s.stream)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    dist.barrier()
    torch.cuda.synchronize()
    e0.record(stream)
    stats = s.step(steps, allow_noconv=True)  # a capped solve is reported in its status
    e1.record(stream)
    torch.cuda.synchronize()
    dist.barrier()
    return e0.elapsed_time(e1), stats


def run_mode(cg, torch, dist, wl, steps, warmup, solver, precision, maxit=5000, profile=True, keep_fields=False,
             precond="none", **extra):
    """solver None: the case's own FP64 solver; the case's tolerance throughout."""
    cfg, wsolver, tol = workload(wl)
    with cg.Solver(solver=solver or wsolver, precision=precision, tol=tol, maxit=maxit, precond=precond,
                   **cfg, **extra) as s:
        s.init_fields()
        s.step(warmup, allow_noconv=True)
        s.reset_counters()
        ms, stats = _timed_steps(s, steps, dist, torch)
        launches = s.launch_count()
        free, total = torch.cuda.mem_get_info()
        out = {"ms": ms, "stats": stats, "launches": launches, "cells": s.cells,
               "device_mem_gb": round((total - free) / 1e9, 2)}
        if keep_fields:
            out["fields"] = s.get_fields()
        if profile:
            # live per-kernel durations: the same number of further steps with every
            # kernel bracketed by CUDA events on the library's stream
            s.reset_counters()
            s.set_kernel_timing(True)
            out["kernel_iters"] = sum(r.iters for r in s.step(steps, allow_noconv=True))
            s.set_kernel_timing(False)
            out["kernels"] = s.kernel_stats()
        return out


def e2e_mode(cg, torch, dist, wl, steps, warmup, solver, precision, maxit=5000):
    """The public API with HOST buffers: per step, H2D of u,v,w,p from pinned memory,
    one step, D2H of u,v,w,p; all on the library's stream inside the events.  Returns the time, the
    bytes of a direction and step, and the steps' results (a capped solve is reported in its
    status, as in run_mode)."""
    cfg, wsolver, tol = workload(wl)
    with cg.Solver(solver=solver or wsolver, precision=precision, tol=tol, maxit=maxit, **cfg) as s:
        s.init_fields()
        s.step(warmup, allow_noconv=True)
        host = {k: torch.empty(s.shape, dtype=torch.float64, pin_memory=True).numpy() for k in "uvwp"}
        s.get_fields(host)
        stream = torch.cuda.ExternalStream(s.stream)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        dist.barrier()
        torch.cuda.synchronize()
        e0.record(stream)
        stats = []
        for _ in range(steps):
            s.set_fields(host["u"], host["v"], host["w"], host["p"])
            stats += s.step(1, allow_noconv=True)
            s.get_fields(host)
        e1.record(stream)
        torch.cuda.synchronize()
        dist.barrier()
        ms = e0.elapsed_time(e1)
        nbytes = 4 * int(host["u"].nbytes)
        return ms, nbytes, stats


def e2e_line(cg, torch, dist, wl, steps, warmup, maxit):
    """The line's e2e entry, with the solves that hit the cap and any that missed the tolerance."""
    _, _, tol = workload(wl)
    ms, nbytes, stats = e2e_mode(cg, torch, dist, wl, steps, warmup, None, "fp64", maxit)
    te = dist.max(ms)
    out = {"value": cells_of(wl) * steps * dist.world / (te / 1e3), "unit": "cell-steps/s",
           "h2d_bytes_per_step": nbytes, "d2h_bytes_per_step": nbytes, **solve_counts(stats, tol)}
    if out["unconverged_solves"]:
        out["failure"] = unconverged_text(out, steps, tol, maxit)
    return out


def unconverged_text(counts, steps, tol, maxit):
    """The metric names the tolerance: say plainly that some timed solves missed it."""
    return (f"{counts['unconverged_solves']} of {steps} timed solves ended at or above "
            f"relres {tol:g} ({counts['capped_solves']} at the {maxit}-iteration cap)")


def adjoint_mode(cg, torch, dist, nsteps, ckpt, wl="c4", first=0, precision="fp64", solver="jacobi",
                 precond="none"):
    """Forward run with checkpoints and the adjoint sweep (gradient of the drag averaged
    over the last third of the window, or from step `first`, w.r.t. the inlet profile and
    eta) on the adjoint case; returns both wall times (CUDA events on the library's stream)
    and their ratio.  precision/solver/precond: the forward's; the backward recomputes and
    solves as the forward does (MIXED: FP32 sweeps in FP64 refinement, the FP32 stencil's
    transpose; FP64 multigrid: the FP64 V-cycle)."""
    cfg = dict(WORKLOADS[wl])
    with cg.Solver(solver=solver, precision=precision, precond=precond, tol=TOL, **cfg) as s:
        stream = torch.cuda.ExternalStream(s.stream)
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(3)]
        s.init_fields()
        first = first or nsteps - nsteps // 3 + 1
        torch.cuda.synchronize()
        ev[0].record(stream)
        J = s.forward(nsteps, first, nsteps, ckpt)
        ev[1].record(stream)
        g_in, g_eta = s.backward()
        ev[2].record(stream)
        torch.cuda.synchronize()
        tf, tb = ev[0].elapsed_time(ev[1]), ev[1].elapsed_time(ev[2])
        free, total = torch.cuda.mem_get_info()
        import numpy as np
        return {"workload": wl, "precision": precision, "solver": solver, "precond": precond,
                "device_mem_gb": round((total - free) / 1e9, 2), "steps": nsteps,
                "objective_steps": [first, nsteps], "ckpt_every": ckpt,
                "J": J, "forward_ms": tf, "backward_ms": tb, "adjoint_over_forward": tb / tf,
                "forward_cell_steps_per_s": s.cells * nsteps / (tf / 1e3),
                "grad_inlet_norm": float(np.linalg.norm(g_in)), "grad_eta_norm": float(np.linalg.norm(g_eta))}


def adjoint_fd_mode(cg, nsteps, ckpt, ndir, eps=1e-6, tol=1e-12):
    """The adjoint gradients on the adjoint case against central finite differences of the
    forward step: ndir seeded directions (seeds 1..ndir) for the inlet profile and as many
    for eta (restricted to the DFIB band, 0 < eta < 1, interior cells), drag averaged over
    the last third of nsteps steps, Poisson solved to tol with its right-hand side's mean
    removed (with the reference's zero-gradient boundaries a perturbed inflow or body makes
    the unprojected Neumann problem inconsistent).  Returns the relative errors."""
    import numpy as np
    cfg = dict(WORKLOADS["c4"])
    first = nsteps - nsteps // 3 + 1
    with cg.Solver(tol=tol, project_rhs=1, **cfg) as s:
        eta0 = s.get_eta()

        def J(inlet=None, eta=eta0):
            s.set_inlet(inlet)
            s.set_eta(eta)
            s.init_fields()
            return s.forward(nsteps, first, nsteps, ckpt)

        J0 = J()
        g_in, g_eta = s.backward()
        one = np.ones(g_in.shape)
        band = (eta0 > 0) & (eta0 < 1)
        for a in range(3):
            sl = [slice(None)] * 3
            sl[a] = slice(0, 2)
            band[tuple(sl)] = False
            sl[a] = slice(-2, None)
            band[tuple(sl)] = False
        err_in, err_eta = [], []
        for seed in range(1, ndir + 1):
            rng = np.random.default_rng(seed)
            d = rng.standard_normal(g_in.shape)
            fd = (J(one + eps * d) - J(one - eps * d)) / (2 * eps)
            err_in.append(abs(float(np.sum(g_in * d)) - fd) / abs(fd))
            de = np.where(band, rng.standard_normal(eta0.shape), 0.0)
            fd = (J(eta=eta0 + eps * de) - J(eta=eta0 - eps * de)) / (2 * eps)
            err_eta.append(abs(float(np.sum(g_eta * de)) - fd) / abs(fd))
        s.set_inlet(None)
        s.set_eta(eta0)
    return {"workload": "c4", "steps": nsteps, "objective_steps": [first, nsteps], "ckpt_every": ckpt,
            "tol": tol, "eps": eps, "directions": ndir, "J": J0,
            "inlet_rel_err": err_in, "eta_rel_err": err_eta, "max_rel_err": max(err_in + err_eta)}


def field_errors(a, b):
    """Relative L2 errors of run a against run b after the same steps: u, v, w against the
    norm of b's whole velocity, p without its mean (the Neumann problem leaves it free),
    drag as the largest relative difference over the timed steps."""
    import numpy as np
    fa, fb = a["fields"], b["fields"]
    core = (slice(2, -2),) * 3
    scale = float(np.sqrt(sum(np.linalg.norm(fb[k][core]) ** 2 for k in "uvw")))
    out = {k: float(np.linalg.norm(fa[k][core] - fb[k][core]) / scale) for k in "uvw"}
    pa, pb = fa["p"][core], fb["p"][core]
    out["p"] = float(np.linalg.norm((pa - pa.mean()) - (pb - pb.mean())) / np.linalg.norm(pb - pb.mean()))
    cda, cdb = np.array([r.cd for r in a["stats"]]), np.array([r.cd for r in b["stats"]])
    out["cd"] = float(np.abs(cda - cdb).max() / np.abs(cdb).max())
    return out


def roofline(prof, cells, word_bytes, suffix, hbm_peak, peak_kind, traffic_file, iters=0):
    """iters: the profiled steps' Krylov iterations (for the one-launch kernels)."""
    words = launch_units(prof, iters, KERNEL_WORDS, LOOP_WORDS)
    ks = {k: prof[k] for k in words if k.endswith(suffix)}
    if not ks:
        return None, {}
    total = sum(v[0] for v in prof.values())
    dom = max(ks, key=lambda k: ks[k][0])
    ms, n = ks[dom]
    per_launch_s = ms / n / 1e3
    alg = words[dom] * word_bytes * cells
    achieved = alg / per_launch_s / 1e9
    traffic = None
    if traffic_file.exists():
        t = json.loads(traffic_file.read_text())
        traffic = t.get(dom, {}).get("bytes_per_launch")
    share = {k: round(v[0] / total, 4) for k, v in sorted(prof.items(), key=lambda kv: -kv[1][0]) if v[0] > 0}
    # every iteration kernel of this precision: average launch and algorithmic GB/s
    each = {}
    for k, (kms, kn) in sorted(ks.items(), key=lambda kv: -kv[1][0]):
        us = kms / kn * 1e3
        gbs = words[k] * word_bytes * cells / (us * 1e-6) / 1e9
        each[k] = {"avg_launch_us": round(us, 2), "achieved": round(gbs, 1), "frac": round(gbs / hbm_peak, 4)}
    r = {"kernel": dom, "bound": "hbm", "achieved": round(achieved, 1), "peak": hbm_peak,
         "unit": "GB/s", "frac": round(achieved / hbm_peak, 4), "traffic": traffic,
         "algorithmic_bytes_per_launch": alg, "avg_launch_us": round(per_launch_s * 1e6, 2),
         "peak_kind": peak_kind, "per_kernel": each}
    return r, share


# the modes beside the FP64 value: (solver (None: the case's own FP64 solver), precision,
# preconditioner, what it is).  Each
# MIXED mode has an FP64 counterpart with the same solver (PRECISION_PAIR), so that its
# speed-up over that one isolates the precision; against `value` it also includes the
# change of solver.
MODES = {
    "cg": ("cg", "fp64", "none", "cg (SPE operator), FP64"),
    "fp64_mg": (None, "fp64", "multigrid",
                "the case's bicgstab right-preconditioned by an FP64 multigrid V-cycle, FP64"),
    "mixed": (None, "mixed", "none", "the case's bicgstab, FP32 sweeps in FP64 refinement"),
    "mixed_cg": ("cg", "mixed", "none", "cg (SPE operator), FP32 sweeps in FP64 refinement"),
    "mixed_mg": (None, "mixed", "multigrid",
                 "the case's bicgstab, FP32 sweeps right-preconditioned by an FP32 multigrid V-cycle, in FP64 "
                 "refinement"),
}
PRECISION_PAIR = {"mixed": "fp64", "mixed_cg": "cg", "mixed_mg": "fp64_mg"}


FP_PEAK_CACHE = {}  # the measured FMA rates of this run (alu_peaks), for step_roofline


def measure_mode(cg, torch, dist, wl, key, steps, warmup, maxit, fp64, t64, hbm_peak, peak_kind, traffic_file,
                 keep_fields=True, profile=True):
    """One mode of MODES on the workload: its timed window, solve record, errors against the
    FP64 run (when fp64 holds its fields) and per-kernel roofline."""
    solver, prec, precond, what = MODES[key]
    _, _, tol = workload(wl)
    rm = run_mode(cg, torch, dist, wl, steps, warmup, solver, prec, maxit=maxit, keep_fields=keep_fields,
                  precond=precond, profile=profile)
    tm = dist.max(rm["ms"])
    cells = rm["cells"]
    out = {"value": cells * steps * dist.world / (tm / 1e3), "ms_per_step": tm / steps, "solver": what,
           "precision": prec, "iters_per_step": [r.iters for r in rm["stats"]],
           "outer_per_step": [r.outer for r in rm["stats"]], "relres": max(r.relres for r in rm["stats"]),
           **solve_counts(rm["stats"], tol), "speedup_vs_fp64": t64 / tm if t64 else None,
           "gpu_launches": rm["launches"], "device_mem_gb": rm["device_mem_gb"]}
    if fp64 is not None and "fields" in fp64 and "fields" in rm:
        out["error_vs_fp64"] = field_errors(rm, fp64)
    if profile:
        word, suffix = (4, "32") if prec == "mixed" else (8, "64")
        out["roofline"], out["kernel_share"] = roofline(rm["kernels"], cells, word, suffix, hbm_peak, peak_kind,
                                                        traffic_file, rm["kernel_iters"])
        if prec == "mixed":
            c = WORKLOADS[wl]
            npad = (c["nx"] + 4) * (c["ny"] + 4) * (c["nz"] + 4)
            out["step_kernels"] = step_roofline(rm["kernels"], cells, npad, hbm_peak, FP_PEAK_CACHE.get("peaks"))
    rm.pop("fields", None)
    return out, rm


def precision_speedups(line, t64, steps):
    """Each MIXED mode against the FP64 mode with the same solver (precision alone)."""
    out = {}
    for m, ref in PRECISION_PAIR.items():
        a = line.get(m) or {}
        b = {"ms_per_step": t64 / steps} if ref == "fp64" else (line.get(ref) or {})
        if a.get("ms_per_step") and b.get("ms_per_step"):
            out[m] = {"against": ref, "speedup": b["ms_per_step"] / a["ms_per_step"]}
            a["speedup_vs_fp64_same_solver"] = out[m]["speedup"]
    return out


def subline(cg, torch, dist, wl, steps, warmup, maxit, hbm_peak, peak_kind):
    """A short measurement of a second workload (the 1024x512x128 case the mixed-precision
    target is quoted on): every solver and precision pair, per-step time, iterations and,
    for the MIXED modes, the sweep kernels' fraction of the HBM bandwidth.  The FP64 modes
    are timed without the per-kernel pass (their kernels are the FP64 pipe's)."""
    traffic_file = ROOT / "profiles" / f"traffic_{wl}.json"
    base = run_mode(cg, torch, dist, wl, steps, warmup, None, "fp64", maxit=maxit, profile=False)
    t64 = dist.max(base["ms"])
    _, _, tol = workload(wl)
    out = {"workload": wl, "config": bench_config(wl, maxit, dist.world), "steps": steps, "warmup": warmup,
           "fp64": {"value": base["cells"] * steps * dist.world / (t64 / 1e3), "ms_per_step": t64 / steps,
                    "iters_per_step": [r.iters for r in base["stats"]], **solve_counts(base["stats"], tol)}}
    for key in ("cg", "fp64_mg", "mixed_cg", "mixed_mg"):
        prof = MODES[key][1] == "mixed"
        out[key], _ = measure_mode(cg, torch, dist, wl, key, steps, warmup, maxit, None, t64, hbm_peak, peak_kind,
                                   traffic_file, keep_fields=False, profile=prof)
        r = out[key].pop("roofline", None)
        if r:
            out[key]["hbm_frac"] = {k: v["frac"] for k, v in r["per_kernel"].items()}
        out[key].pop("kernel_share", None)
    out["precision_speedup"] = precision_speedups(out, t64, steps)
    return out


# The boundary set the benchmark's configurations state (uniform inflow, convective
# outflow, free-slip y walls, periodic z, seeded uniform(-1e-3, 1e-3) perturbation of u, v,
# w).  The reference has only its zero-gradient table, so the headline value (compared with
# the reference's own CPU build) runs that table; this line runs the stated set.
BSET_SEED = 2024
BSET_DOC = ("stated: uniform inflow U=1, convective outflow with the mass-flux correction, free-slip y walls, "
            "periodic z (not in the reference)")


def boundary_set_line(cg, torch, dist, wl, steps, warmup, maxit, hbm_peak, peak_kind):
    """The workload on the stated boundary set from the seeded perturbation: FP64 and MIXED
    with the case's solver, with CG and with the multigrid-preconditioned BiCGSTAB (its
    levels periodic in z); per-step time, iterations, solve record, each MIXED mode's error
    against the FP64 run and its speed-up over the same solver in FP64."""
    import numpy as np
    extra = dict(cg.BOUNDARY_SET, seed=BSET_SEED, amp=1e-3)
    _, _, tol = workload(wl)
    out = {"workload": wl, "bc": BSET_DOC,
           "data": f"synthetic: u=1, v=w=0 plus uniform(-1e-3, 1e-3) (splitmix64 seed {BSET_SEED})",
           "steps": steps, "warmup": warmup}
    runs, ms = {}, {}
    for key, solver, prec, pc in (("fp64", None, "fp64", "none"), ("mixed", None, "mixed", "none"),
                                  ("cg", "cg", "fp64", "none"), ("mixed_cg", "cg", "mixed", "none"),
                                  ("fp64_mg", None, "fp64", "multigrid"), ("mixed_mg", None, "mixed", "multigrid")):
        r = run_mode(cg, torch, dist, wl, steps, warmup, solver, prec, maxit=maxit, profile=prec == "mixed",
                     keep_fields=True, precond=pc, **extra)
        t = dist.max(r["ms"])
        o = {"value": r["cells"] * steps * dist.world / (t / 1e3), "ms_per_step": t / steps,
             "iters_per_step": [x.iters for x in r["stats"]], "outer_per_step": [x.outer for x in r["stats"]],
             "relres": max(x.relres for x in r["stats"]), **solve_counts(r["stats"], tol),
             "gpu_launches": r["launches"]}
        if prec == "mixed":
            o["error_vs_fp64"] = field_errors(r, runs["fp64"])
            roof, _ = roofline(r["kernels"], r["cells"], 4, "32", hbm_peak, peak_kind, Path("/nonexistent"),
                               r["kernel_iters"])
            if roof:
                o["hbm_frac"] = {k: v["frac"] for k, v in roof["per_kernel"].items()}
            base = PRECISION_PAIR[key]
            o["speedup_vs_fp64_same_solver"] = ms[base] / t
        else:
            # the corrected outlet carries the inlet's flux: the net boundary flux of the last state
            f = r["fields"]
            c = WORKLOADS[wl]
            a = (c["ly"] / c["ny"]) * (c["lz"] / c["nz"])
            o["net_flux"] = float(np.sum(f["u"][1, 2:-2, 2:-2] - f["u"][-3, 2:-2, 2:-2]) * a)
        ms[key] = t
        runs[key] = r if key == "fp64" else {"stats": r["stats"]}
        out[key] = o
    return out


def sor_legs(cg, torch, dist, wl, args, cells, tol):
    """Red-black SOR twice: at the optimal relaxation of the grid (omega = 0 picks it: Young's
    2 / (1 + sqrt(1 - mu^2)), mu the Jacobi spectral radius), timed to the tolerance, and at
    omega = 1.7, capped at --sor-maxit sweeps, with the sweeps the Jacobi spectral radius
    predicts it would need (its value is that of an unconverged solve, so it reports none)."""
    import math
    c = WORKLOADS[wl]
    h = [c["lx"] / c["nx"], c["ly"] / c["ny"], c["lz"] / c["nz"]]
    w = [1 / x ** 2 for x in h]
    low = min(wa * (1 - math.cos(math.pi / n)) for wa, n in zip(w, (c["nx"], c["ny"], c["nz"])) if n > 1)
    mu = 1 - low / sum(w)
    opt = 2 / (1 + math.sqrt(1 - mu * mu))
    so = run_mode(cg, torch, dist, wl, args.sor_steps, args.warmup, "rbsor", "fp64", maxit=args.sor_maxit,
                  profile=False, omega=0.0)
    ts = dist.max(so["ms"])
    out = {"value": cells * args.sor_steps * dist.world / (ts / 1e3), "ms_per_step": ts / args.sor_steps,
           "steps": args.sor_steps, "omega": opt, "sweeps_per_step": [r.iters for r in so["stats"]],
           "relres": [r.relres for r in so["stats"]], "status": [r.status for r in so["stats"]],
           **solve_counts(so["stats"], tol)}
    s17 = run_mode(cg, torch, dist, wl, 1, args.warmup, "rbsor", "fp64", maxit=args.sor_maxit, profile=False,
                   omega=1.7)
    # red-black SOR at omega below the optimum: rate from the largest root of
    # lambda - omega mu sqrt(lambda) + omega - 1 = 0 (Young), sweeps = ln(tol) / ln(rate)
    om = 1.7
    sq = (om * mu + math.sqrt(max(0.0, om * om * mu * mu - 4 * (om - 1)))) / 2
    out["omega_1_7"] = {"value": None, "omega": om, "sweeps_cap": args.sor_maxit,
                        "relres": [r.relres for r in s17["stats"]], "status": [r.status for r in s17["stats"]],
                        "predicted_sweeps_to_tol": round(math.log(tol) / math.log(sq * sq)),
                        "note": "unreachable at omega 1.7 within the cap; the leg above uses the optimal omega"}
    return out


def reference_build(wl, flavour="native"):
    """The reference's own build for a case and the harness's name of its solver."""
    from oracle import build_ref
    cfg, solver, tol = workload(wl)
    exe = build_ref.build(cfg["nx"], cfg["ny"], cfg["nz"], cfg["lx"], cfg["ly"], cfg["lz"], cfg["cx"], flavour,
                          gridder=cfg.get("grid", "uniform"))
    return exe, {"jacobi": "csr", "bicgstab": "spe"}[solver], tol


def cpu_reference_sample(wl, steps, cap, threads, iters_per_step):
    """Run the reference's own build (oracle/_ref) for `steps` steps with its BiCGSTAB
    capped at `cap` iterations; derive its time per iteration and per non-solve step
    part, and from those its cell-steps/s at the iteration counts a full solve to the
    case's tolerance needs (iters_per_step: list, one per step)."""
    cfg = WORKLOADS[wl]
    exe, hsolver, tol = reference_build(wl)
    with tempfile.TemporaryDirectory() as td:
        env = dict(os.environ, OMP_NUM_THREADS=str(threads), OMP_PROC_BIND="close", OMP_PLACES="cores")
        t0 = time.perf_counter()
        subprocess.run([str(exe), "run", str(steps), repr(cfg["Re"]), repr(cfg["dt"]), repr(tol), hsolver, "1.7",
                        "0", "0", td, str(cap)], check=True, env=env, cwd=td, stdout=subprocess.DEVNULL,
                       stderr=subprocess.DEVNULL)
        wall = time.perf_counter() - t0
        rows = [list(map(float, l.split())) for l in (Path(td) / "stats.txt").read_text().splitlines()
                if l and not l.startswith("#")]
    solve_rows = [r for r in rows if r[0] > 1 and r[2] > 0]
    t_iter = sum(r[7] for r in solve_rows) / sum(r[2] for r in solve_rows)
    t_other = statistics.median(r[6] - r[7] for r in solve_rows)
    cells = cfg["nx"] * cfg["ny"] * cfg["nz"]
    per_step = [t_other + it * t_iter for it in iters_per_step]
    value = cells * len(per_step) / sum(per_step)
    return {"value": value, "t_iter_s": t_iter, "t_other_s": t_other, "wall_s": wall, "cells": cells}


def reference_iteration_record(wl):
    f = ROOT / "tests" / "golden" / f"reference_iters_{wl}.json"
    if f.exists():
        return json.loads(f.read_text())
    return None


def reference_window_iters(rec, warmup, steps):
    """The reference's recorded iteration counts on the timed steps warmup+1 .. warmup+steps
    (1-based; the record's index 0 is step 1).  Nothing is imputed: a window that reaches
    beyond the record raises ValueError, naming how many timed steps it lacks."""
    its = rec["iters"]
    missing = warmup + steps - len(its)
    if missing > 0:
        raise ValueError(f"the recorded reference run ends at step {len(its)}; the timed window "
                         f"(steps {warmup + 1}-{warmup + steps}) lacks {missing} recorded steps")
    return [its[i] for i in range(warmup, warmup + steps)]


def window_record(rec, warmup, steps, cap, sampled_steps):
    """What the reference arm's number rests on: the recorded steps it is scored on, how
    many were imputed (always 0: a short record makes the arm unavailable), the steps the
    timing sample ran and its iteration cap."""
    return {"recorded_steps": [warmup + 1, warmup + steps], "record_length": len(rec["iters"]),
            "record_threads": rec.get("threads"), "record_host": rec.get("host"), "imputed_steps": 0,
            "sampled_steps": [1, sampled_steps], "cap": cap}


def bench_config(wl, maxit, world):
    """The config both arms print: the workload, its solver, tolerance and cap, the boundary
    set, the replica count and the L2 note."""
    return {**config_of(wl), "maxit": maxit, "bc": "reference (FLOWpassing table)",
            "parallelism": f"replicas x{world}", "l2": l2_note(wl)}


def reference_baseline(wl, warmup, steps, cap, cap1):
    """The reference's CPU throughput on the timed window: all host cores and one thread,
    each from a bounded timing sample (3 steps, BiCGSTAB capped) scored on the iteration
    counts of the recorded full reference run.  Raises when there is no record or it does
    not cover the window."""
    rec = reference_iteration_record(wl)
    if rec is None:
        raise ValueError(f"no recorded reference iteration counts for workload {wl}")
    want = reference_window_iters(rec, warmup, steps)
    threads = os.cpu_count() or 1
    cb = cpu_reference_sample(wl, 3, cap, threads, want)
    c1 = cpu_reference_sample(wl, 3, cap1, 1, want)
    out = {"value": cb["value"], "unit": "cell-steps/s", "cores": threads, "kind": "reference",
           "sample": SAMPLE_DOC.format(cap=cap, t_iter=cb["t_iter_s"], t_other=cb["t_other_s"]),
           "window": window_record(rec, warmup, steps, cap, 3),
           "single_thread": {"value": c1["value"], "unit": "cell-steps/s", "cores": 1, "cap": cap1,
                             "t_iter_s": c1["t_iter_s"], "t_other_s": c1["t_other_s"]}}
    return out


def main_reference(args):
    """--impl reference: the reference's own CPU implementation, host cores."""
    world, rank, _ = _dist()
    if rank != 0:
        return 0
    try:
        cb = reference_baseline(args.workload, args.warmup, args.steps, args.cap, args.cap1)
    except (ValueError, FileNotFoundError, subprocess.CalledProcessError) as e:
        print(json.dumps({"impl": "reference", "unavailable": str(e)}))
        return 0
    line = {"impl": "reference", "metric": metric(args.workload), "value": cb["value"], "unit": "cell-steps/s",
            "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": 1e3 * cells_of(args.workload) / cb["value"], "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic (reference initial state u=1, v=w=0)",
            "config": bench_config(args.workload, args.maxit, args.gpus),
            "cpu_baseline": cb,
            "e2e": {"value": cb["value"], "unit": "cell-steps/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line))
    return 0


def cells_of(wl):
    cfg = WORKLOADS[wl]
    return cfg["nx"] * cfg["ny"] * cfg["nz"]


def solve_record(stats, tol):
    """Per-step solve outcome of a timed window: iterations, final relative residual and
    status of every step, the solves that hit the iteration cap and the solves that ended
    at or above the tolerance (step 1 of a run has no solve and is not counted)."""
    solves = [r for r in stats if r.step > 1]
    return {"step": [r.step for r in stats], "iters": [r.iters for r in stats],
            "relres": [r.relres for r in stats], "status": [r.status for r in stats],
            "capped_solves": sum(1 for r in solves if r.status == -3),
            "unconverged_solves": sum(1 for r in solves if not (r.relres < tol))}


def solve_counts(stats, tol):
    r = solve_record(stats, tol)
    return {"capped_solves": r["capped_solves"], "unconverged_solves": r["unconverged_solves"]}


METRIC = "cell-steps/s @resid 1e-8 (FP64 Jacobi-BiCGSTAB projection step)"
SAMPLE_DOC = ("reference OpenMP build (-O3 -fopenmp -march=native) on the same grid, steps 1-3 with its "
              "BiCGSTAB capped at {cap} iterations: {t_iter:.4f} s per iteration, {t_other:.3f} s per step "
              "outside the solve; cell-steps/s at the iteration counts the reference itself needed to reach "
              "the tolerance on exactly the timed steps, recorded from a full reference run "
              "(tests/golden/reference_iters_<workload>.json; none imputed)")


def main(argv=None):
    ap = argparse.ArgumentParser(description="projection-step benchmark")
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="cfdgb", choices=["cfdgb", "reference"])
    ap.add_argument("--workload", default="c2", choices=sorted(WORKLOADS))
    ap.add_argument("--modes", default="fp64,mixed,fp64_mg,mixed_mg,cg,mixed_cg,rbsor,bcset,e2e,adjoint,cpu")
    ap.add_argument("--c3-steps", type=int, default=2,
                    help="timed steps of the 1024x512x128 sub-line (0: none)")
    ap.add_argument("--adj-steps", type=int, default=30)
    ap.add_argument("--adj-ckpt", type=int, default=10)
    ap.add_argument("--adj-workload", default="c4", choices=sorted(WORKLOADS))
    ap.add_argument("--adj-first", type=int, default=0,
                    help="first step of the drag average (0: the last third of --adj-steps)")
    ap.add_argument("--adj-precision", default="fp64", choices=["fp64", "mixed"])
    ap.add_argument("--adj-solver", default="jacobi", choices=["jacobi", "bicgstab", "cg"])
    ap.add_argument("--adj-precond", default="none", choices=["none", "multigrid"])
    ap.add_argument("--maxit", type=int, default=5000,
                    help="Krylov iteration cap per solve (the reference's 5000; MIXED: FP32 iterations)")
    ap.add_argument("--fd-steps", type=int, default=21, help="adjoint_fd mode: steps of each forward run")
    ap.add_argument("--fd-dirs", type=int, default=16, help="adjoint_fd mode: directions per gradient")
    ap.add_argument("--cap", type=int, default=10, help="reference BiCGSTAB iteration cap of the CPU sample")
    ap.add_argument("--cap1", type=int, default=4,
                    help="reference BiCGSTAB iteration cap of the single-thread CPU sample")
    ap.add_argument("--sor-steps", type=int, default=2)
    ap.add_argument("--sor-maxit", type=int, default=20000)
    args = ap.parse_args(argv)
    if args.warmup < 3:
        ap.error("--warmup must be >= 3")
    if args.impl == "reference":
        return main_reference(args)

    import torch
    import cfd_nssolver_forhpc_flowpassingcylinder_gb300 as cg
    dist = Dist()
    torch.cuda.set_device(dist.local)
    modes = set(args.modes.split(","))
    hbm_peak, peak_kind = peaks()
    wl = args.workload
    traffic_file = ROOT / "profiles" / f"traffic_{wl}.json"

    fp_peak = alu_peaks()
    FP_PEAK_CACHE["peaks"] = fp_peak
    with Clocks(dist.local) as clk:
        fp64 = run_mode(cg, torch, dist, wl, args.steps, args.warmup, None, "fp64", maxit=args.maxit,
                        keep_fields=bool(modes & set(MODES)))
    t64 = dist.max(fp64["ms"])
    cells = fp64["cells"]
    value = cells * args.steps * dist.world / (t64 / 1e3)
    roof, share = roofline(fp64["kernels"], cells, 8, "64", hbm_peak, peak_kind, traffic_file, fp64["kernel_iters"])
    iters64 = [r.iters for r in fp64["stats"]]
    _, _, tol = workload(wl)
    rec64 = solve_record(fp64["stats"], tol)
    line = {
        "metric": metric(wl), "value": value, "unit": "cell-steps/s", "n_gpus": dist.world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": t64 / args.steps, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f64", "data": "synthetic (reference initial state u=1, v=w=0)",
        "config": bench_config(wl, args.maxit, dist.world),
        "iters_per_step": iters64, "relres": max(r.relres for r in fp64["stats"]),
        "solves": rec64,
        "gpu_launches": fp64["launches"], "roofline": roof, "kernel_share": share,
        "alu_roofline": alu_roofline(fp64["kernels"], cells, fp_peak, fp64["kernel_iters"]), "fp_peaks": fp_peak,
        "clocks": clk.summary(), "device_mem_gb": fp64["device_mem_gb"],
    }
    if rec64["unconverged_solves"]:
        line["failure"] = unconverged_text(rec64, args.steps, tol, args.maxit)
    results = {"fp64": fp64}
    for key in [m for m in MODES if m in modes]:
        try:
            line[key], results[key] = measure_mode(cg, torch, dist, wl, key, args.steps, args.warmup, args.maxit,
                                                   fp64, t64, hbm_peak, peak_kind, traffic_file)
        except cg.CfdgbError as e:
            line[key] = {"value": None, "error": str(e)}
    line["precision_speedup"] = precision_speedups(line, t64, args.steps)
    if args.c3_steps > 0 and wl != "c3":
        try:
            line["c3"] = subline(cg, torch, dist, "c3", args.c3_steps, args.warmup, args.maxit, hbm_peak, peak_kind)
        except cg.CfdgbError as e:
            line["c3"] = {"error": str(e)}
    if "rbsor" in modes:
        line["rbsor"] = sor_legs(cg, torch, dist, wl, args, cells, tol)
    if "bcset" in modes:
        try:
            line["boundary_set"] = boundary_set_line(cg, torch, dist, wl, args.steps, args.warmup, args.maxit,
                                                     hbm_peak, peak_kind)
        except cg.CfdgbError as e:
            line["boundary_set"] = {"error": str(e)}
    if "e2e" in modes:
        try:
            line["e2e"] = e2e_line(cg, torch, dist, wl, args.steps, args.warmup, args.maxit)
        except cg.CfdgbError as e:
            line["e2e"] = {"value": None, "error": str(e)}
    if "adjoint" in modes:
        try:
            line["adjoint"] = adjoint_mode(cg, torch, dist, args.adj_steps, args.adj_ckpt, args.adj_workload,
                                           args.adj_first, args.adj_precision, args.adj_solver, args.adj_precond)
        except cg.CfdgbError as e:
            line["adjoint"] = {"value": None, "error": str(e)}
        if (args.adj_precision, args.adj_precond) != ("mixed", "multigrid"):
            # the 1536x768x96 case's recipe (MIXED multigrid forward, then the adjoint) on the
            # adjoint case's grid
            try:
                line["adjoint"]["mixed_multigrid"] = adjoint_mode(cg, torch, dist, args.adj_steps, args.adj_ckpt,
                                                                  args.adj_workload, args.adj_first, "mixed",
                                                                  args.adj_solver, "multigrid")
            except cg.CfdgbError as e:
                line["adjoint"]["mixed_multigrid"] = {"error": str(e)}
    if "adjoint_fd" in modes:  # not in the default modes: ~4 * fd_dirs forward runs
        try:
            line["adjoint_fd"] = adjoint_fd_mode(cg, args.fd_steps, args.adj_ckpt, args.fd_dirs)
        except cg.CfdgbError as e:
            line["adjoint_fd"] = {"value": None, "error": str(e)}
    if "cpu" in modes and dist.rank == 0:
        try:
            line["cpu_baseline"] = reference_baseline(wl, args.warmup, args.steps, args.cap, args.cap1)
        except Exception as e:  # reference binary or record unavailable on this host
            line["cpu_baseline"] = {"value": None, "unit": "cell-steps/s", "cores": os.cpu_count(),
                                    "kind": "reference", "sample": f"unavailable: {e}"}
    if dist.rank == 0:
        print(json.dumps(line))
    dist.close()
    return 0


if __name__ == "__main__":
    sys.exit(main())
