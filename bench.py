#!/usr/bin/env python
"""Throughput of the MPH-I time step on GB300 (particle-steps/s).

Workload (default): the 3D cube collapse of 100^3 fluid particles (l0 =
0.005 m) in a 3-layer wall tank around a 160x110x110 interior, gravity -9.8 in
z, dt = 5e-5 s, lambda*dt/(rho*l0^2) = 100, seeded +-0.01 l0 jitter:
1,297,696 particles.  Synthetic inputs generated here stand in for the case
files.  One step = the full reference step (sort, neighbours, explicit
physics, assembly, multigrid build, CR solve).

  value : particle-steps/s of the mixed form (FP32 CR + V-cycle, FP64 outer
          refinement to ||b - A x|| / ||b|| < 1e-10; --precision fp64 for the
          plain form) with the state resident in HBM, CUDA events on the case
          stream around K steps (the pair terms alone are ~7 GB, far above
          L2).  The line also carries the plain FP64 form's value on the same
          workload (the reference algorithm, stop test 1e-6) and the velocity
          error of one mixed step against the FP64 form solved to 1e-12 from
          the same state (the accuracy the metric names), plus the mixed form
          at the reference's 1e-6 as a labelled secondary
  e2e   : the same metric through the public API with pinned host buffers:
          every one of K steps uploads the particle state
          (mph_case_set_state) and reads back ids, types, positions and
          velocities (mph_get_fields)
  --impl reference : the CPU restatement of the reference (the oracle,
          OpenMP over all host cores) on the same workload, one full step
          per timed step
"""
from __future__ import annotations

import argparse
import json
import os
import re
import statistics
import subprocess
import sys
import tempfile
import time

import numpy as np

REPO = os.path.dirname(os.path.abspath(__file__))
sys.path[:0] = [REPO, os.path.join(REPO, "oracle")]

from mphimplicit_gb300 import casegen  # noqa: E402

METRIC = "particle-steps/sec at <=1e-6 rel. err vs FP64 (mixed/batched vs plain GPU); p50/p99 step ms"
UNIT = "particle-steps/s"


def workload(name: str):
    if name == "cube3d_100":
        p, parts = casegen.cube_collapse_3d(100, seed=0)
        return 3, p, parts, "3D cube collapse, 100^3 fluid in a 3-layer tank around 160x110x110 (config 1)"
    m = re.match(r"cube3d_(\d+)$", name)
    if m:
        n = int(m.group(1))
        p, parts = casegen.cube_collapse_3d(n, seed=0)
        return 3, p, parts, f"3D cube collapse, {n}^3 fluid (config-1 geometry scaled)"
    if name == "dam2d_100":
        p, parts = casegen.square_drop_2d(1.0, seed=0)
        return 2, p, parts, "2D dam, 100x100 fluid in a 3-layer box around 200x150 (config 0)"
    raise SystemExit(f"unknown workload {name}")


def replica_throughput(units: float, seconds: float, dist=None, device="cpu"):
    """Whole-job throughput of independent replicas: the units every rank
    processed, summed, over the slowest rank's time (max over ranks)."""
    if dist is None:
        return units / seconds, seconds
    import torch
    u = torch.tensor([float(units)], dtype=torch.float64, device=device)
    t = torch.tensor([float(seconds)], dtype=torch.float64, device=device)
    dist.all_reduce(u, op=dist.ReduceOp.SUM)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(u.item()) / float(t.item()), float(t.item())


def measured_peaks():
    path = os.path.join(REPO, "MEASURED_PEAKS.json")
    try:
        with open(path) as f:
            d = json.load(f)
        return float(d["hbm_gbs"]), "measured"
    except Exception:
        return 6800.0, "fallback"


def ncu_traffic(kernel: str, algorithmic_bytes: float):
    """DRAM bytes per launch of `kernel` on the bench workload: the ratio of
    DRAM traffic to algorithmic bytes measured by the committed ncu summary
    (profiles/, captured on a smaller case of the same kernels; traffic grows
    with the slot counts) times this launch's algorithmic bytes, or None."""
    path = os.path.join(REPO, "profiles", f"{kernel.split('+')[-1]}_cube3d_100.md")
    if not os.path.exists(path):
        return None
    m = re.search(r"dram_to_algorithmic_ratio:\s*([0-9.eE+]+)", open(path).read())
    return float(m.group(1)) * algorithmic_bytes if m else None


class Clocks:
    """nvidia-smi sampling of SM clocks and throttle reasons during a region."""
    Q = ("clocks.sm,clocks.max.sm,clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu: int):
        self.gpu = gpu
        self.proc = None
        self.f = tempfile.TemporaryFile(mode="w+")

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.gpu), f"--query-gpu={self.Q}", "--format=csv,noheader,nounits",
                                          "-lms", "200"], stdout=self.f, stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None
        return self

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self):
        self.f.seek(0)
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in self.f:
            parts = [x.strip() for x in line.split(",")]
            if len(parts) < 6:
                continue
            try:
                sm.append(float(parts[0]))
                mx.append(float(parts[1]))
            except ValueError:
                continue
            for n, v in zip(names, parts[2:6]):
                if v.lower() == "active":
                    reasons.add(n)
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": [], "samples": 0}
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": max(mx), "reasons": sorted(reasons), "samples": len(sm)}


def spmv_bytes(prof, scal, dim, vb=8):
    """Algorithmic bytes of one block SpMV: every block once (D*D values of vb
    bytes + a column index), row lengths and slice pointers, x once, y
    written once (vb = 8 for the FP64 form, 4 for the FP32 inner solve)."""
    nf = int(scal["FluidParticleEnd"])
    blocks = scal["NonzeroCountA"] / (dim * dim)
    nsl = (nf + 31) // 32
    return blocks * (dim * dim * vb + 4) + nf * 4 + (nsl + 1) * 8 + 2 * dim * nf * vb


def precond_name(args, mixed: bool) -> str:
    if not mixed:
        return "multigrid V-cycle (the reference's)"
    if args.mg_depth < 0:
        return "point Jacobi, in the CR vector update"
    return "multigrid V-cycle, " + ("every level" if args.mg_depth == 0 else f"{args.mg_depth} level(s)")


def pair_apply_bytes(prof, scal, dim, st=None, rec="pack"):
    """Algorithmic bytes of one FP32 inner operator on the sliced pair terms
    (k_ct_apply32 + k_visc_pen32).  k_ct_apply32: column + D FP32 C values per
    transposed P-list slot, entry counts and slice pointers, s gathered once,
    t written.  k_visc_pen32, per fluid slot: rec "fp16" an 8-byte record (g
    in FP16 and the neighbour's block-local index), "pack" a 4-byte packed g
    and, in a staged row block, a 2-byte block-local index, "recompute" only
    that index (g evaluated from the positions, read once: 16 bytes a
    particle); unless the row block's neighbours are staged in shared memory,
    a 4-byte column instead of the index (counted for no slot once any block
    is staged: a lower bound).  Then column + D FP32 lambda C per P-slot, the
    8-float diagonal / inertia record, row lengths, slice pointers and
    scales, s read once, t gathered once, y written; a staged block also reads
    its count and its distinct columns (4 bytes each; their s, which the block
    copies to shared memory, count as part of s read once)."""
    nf = int(scal["FluidParticleEnd"])
    n = int(scal["ParticleCount"])
    slots = scal["NonzeroCountA"] / (dim * dim)
    pslots = scal["NonzeroCountC"] / dim
    nsl, nct = (nf + 31) // 32, (n + 31) // 32
    st = st or {}
    staged = st.get("inner_local_blocks", 0) > 0
    col = 0 if staged else 4
    slot = {"fp16": 8, "pack": 4 + (2 if staged else 0), "recompute": 2 if staged else 0}[rec]
    # P-slots and transposed slots: 16-byte records (D values, zero-padded in
    # 2-D, and the column or the block-local rank), counted as D * 4 + 4
    pcol = ctcol = 4
    ct = pslots * (dim * 4 + ctcol) + n * 4 + (nct + 1) * 8 + dim * nf * 4 + n * 4
    vp = slots * (slot + col) + pslots * (dim * 4 + pcol) + nf * (32 + 8) + 2 * (nsl + 1) * 8 + nsl * 4 \
        + 2 * dim * nf * 4 + n * 4
    if rec == "recompute":
        vp += n * 16
    if staged:
        vp += st["inner_local_cols"] * 4 + (st["inner_local_blocks"] + st["inner_gather_blocks"]) * 4
    return ct + vp


def pen_apply_bytes(prof, scal, dim, st=None):
    """Algorithmic bytes of one application of the point-Jacobi mixed form's
    inner operator, inertia + C Lambda C^T from the P-lists (k_pen_t + k_pen_y,
    or an iteration's share of the resident k_pen_cr): a 2-byte rank per P-list
    slot, the lists of every particle for t and of the fluid rows for y;
    positions (16 bytes a particle) in both; s read in both, t written and
    read, y, D^-1 and q; the row blocks' distinct columns (4 bytes each)."""
    nf = int(scal["FluidParticleEnd"])
    n = int(scal["ParticleCount"])
    pslots = scal["NonzeroCountC"] / dim
    cols = 4 * (st or {}).get("inner_local_cols", 0)
    return 2 * prof["nnbP"] + 2 * pslots + 2 * 16 * n + (2 + 3) * 4 * dim * nf + 8 * n + 2 * cols


def f64_parts_bytes(prof, scal, dim):
    """Algorithmic bytes of one application of the 3-D FP64 form's operator in
    parts (k_f64_parts + k_f64_rows): a 24-byte pair record and a column per
    fluid slot, the direction's 24-byte records, C (3 doubles) and a column per
    P-slot of every particle for t and of the fluid rows for y, t, the pair
    part written and read, x and y."""
    nf = int(scal["FluidParticleEnd"])
    n = int(scal["ParticleCount"])
    slots = scal["NonzeroCountA"] / (dim * dim)
    pslots = scal["NonzeroCountC"] / dim
    return slots * 28 + nf * 24 + (prof["nnbP"] + pslots) * 28 + 16 * n + nf * (48 + 48)


def assemble_pen_bytes(prof, scal, dim):
    """Algorithmic bytes of the point-Jacobi mixed form's assembly stage: the
    P-lists and the particle state read once; C (D doubles) and a 2-byte rank
    per P-slot of every particle, b (D doubles) and D^-1 (D floats) per fluid
    row written."""
    nf = int(scal["FluidParticleEnd"])
    n = int(scal["ParticleCount"])
    return 4 * prof["nnbP"] + 64 * n + prof["nnbP"] * (8 * dim + 2) + nf * dim * 12 + 48 * n


def assemble_bytes(prof, scal, dim):
    nf = int(scal["FluidParticleEnd"])
    n = int(scal["ParticleCount"])
    blocks = scal["NonzeroCountA"] / (dim * dim)
    return (blocks * (dim * dim * 8 + 4) + 4 * prof["nnb"] + 4 * prof["nnbP"] + 64 * n
            + dim * 8 * scal["NonzeroCountC"] / dim)


def assemble_pair_bytes(prof, scal, dim, case, jacobi=False, rec_bytes=6):
    """Algorithmic bytes of the mixed form's assembly stage on the pair path
    (no blocks): the neighbour and P-neighbour lists and the particle state
    read once, and once written what the solve consumes: per fluid slot the
    inner operator's record (rec_bytes: 6 packed, 8 FP16), D FP32 g and a
    4-byte column (outer residual); per
    P-slot of a fluid row a 16-byte lambda-C record and a 16-byte transposed
    record; per fluid row b (D doubles) and a 32-byte diagonal / inertia
    record; the level-0 multigrid stencils (doubles), which the point-Jacobi
    mixed form (jacobi) does not build: it writes D^-1 (D doubles a row)
    instead."""
    nf = int(scal["FluidParticleEnd"])
    n = int(scal["ParticleCount"])
    slots = scal["NonzeroCountA"] / (dim * dim)
    pslots = scal["NonzeroCountC"] / dim
    lv0 = 0 if jacobi else case.export("MultiGridCsrCofA:0").size
    return (4 * prof["nnb"] + 4 * prof["nnbP"] + 64 * n + slots * (rec_bytes + 4 + 4 * dim) + pslots * 32
            + nf * (dim * 8 + 32) + lv0 * 8 + (nf * dim * 8 if jacobi else 0))


def cpu_sample(threads: int, steps: int = 1, fluid: int = 100, check_gpu: bool = False):
    """Time the oracle (OpenMP, `threads` threads) on the config-1 geometry
    at `fluid`^3 fluid particles (100: the workload itself), `steps` full
    steps after the untimed initial pass; optionally run the GPU engine's
    FP64 form on the same case and report the integer parity (sort
    permutation, cell ranges, both neighbour lists) and the velocity error
    against the oracle."""
    import oracle as orc
    orc.build_oracle()
    p, parts = casegen.cube_collapse_3d(fluid, seed=0)
    o = orc.Oracle(p, parts, 3, threads=threads)
    o.init()
    t0 = time.perf_counter()
    o.step(steps)
    dt = time.perf_counter() - t0
    out = {"value": parts.count * steps / dt, "unit": UNIT, "cores": threads, "kind": "port",
           "sample": f"3D cube collapse {fluid}^3 fluid ({parts.count} particles), {steps} full step(s) after the "
                     f"initial pass, {dt:.1f} s wall"}
    if check_gpu:
        from mphimplicit_gb300 import engine
        g = engine.Case(p, parts, 3)
        g.step(steps)
        nf = g.fluid_count
        exact = {}
        for name in ("ParticleIndex", "CellFluidParticleBegin", "CellFluidParticleEnd", "CellWallParticleBegin",
                     "CellWallParticleEnd", "NeighborPtr", "NeighborInd", "NeighborPtrP", "NeighborIndP"):
            exact[name] = bool(np.array_equal(g.export(name), o.array(name)))
        out["gpu_bit_exact"] = exact
        vo = o.array("Velocity").reshape(-1, 3)[:nf]
        vg = g.export("Velocity").reshape(-1, 3)[:nf]
        out["gpu_err_vs_oracle"] = float(np.linalg.norm(vg - vo) / np.linalg.norm(vo))
        out["iters_oracle_gpu"] = [o.solve_stats()["iter"], g.solve_stats()["iter"]]
        g.close()
    return out


def run_reference(args, rank, world):
    """The reference arm: the CPU restatement of the reference's OpenMP path
    (the oracle, all host threads) on the same workload as the GPU arm, W
    untimed and K timed full steps after the initial pass.  The oracle's CR
    iteration count of every timed step is reported beside the value."""
    if rank != 0:
        return 0
    threads = os.cpu_count() or 1
    import oracle as orc
    orc.build_oracle()
    if args.workload in ("ensemble2d", "serve"):
        dim, p, parts, desc = workload("dam2d_100")
        desc += " (one case of the batched workloads' 2D family)"
    elif args.ref_fluid > 0:
        dim = 3
        p, parts = casegen.cube_collapse_3d(args.ref_fluid, seed=0)
        desc = f"3D cube collapse {args.ref_fluid}^3 fluid (config-1 geometry scaled)"
    else:
        dim, p, parts, desc = workload(args.workload)
    t_init = time.perf_counter()
    o = orc.Oracle(p, parts, dim, threads=threads)
    o.init()
    t_init = time.perf_counter() - t_init
    warm, steps = min(args.warmup, 2), max(1, min(args.steps, args.ref_max_steps))
    for _ in range(warm):
        o.step(1)
    times, iters = [], []
    for _ in range(steps):
        t0 = time.perf_counter()
        o.step(1)
        times.append(time.perf_counter() - t0)
        iters.append(o.solve_stats()["iter"])
    tot = sum(times)
    value = parts.count * steps / tot
    same = args.workload not in ("ensemble2d", "serve") and args.ref_fluid <= 0
    sample = (f"{desc}: {parts.count} particles{', the full workload' if same else ''}; {steps} timed steps after {warm} "
              f"warm-up steps and the initial pass ({t_init:.1f} s, untimed); CR stop test 1e-6 (the reference's)"
              + ("" if steps == args.steps else f"; {steps} of the requested {args.steps} steps timed (bounded sample)"))
    line = {"impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": args.gpus, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": 1000 * tot / steps, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": args.workload if same else f"{args.workload} (sampled: {desc})", "description": desc,
                       "dim": dim, "particles": parts.count, "sample": sample, "threads": threads,
                       "cr_iterations": iters, "p50_step_ms": float(np.percentile(times, 50)) * 1000,
                       "p99_step_ms": float(np.percentile(times, 99)) * 1000},
            "cpu_baseline": {"value": value, "unit": UNIT, "cores": threads, "kind": "port", "sample": sample},
            "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)
    return 0


def _vel_error_vs_fp64(engine, cases, prec_mixed, prec_fp64, tol_outer, tol_ref=1e-12, extra=False, pre=0, setup=None):
    """One step of each (params, parts, dim) in the mixed form (outer
    tolerance tol_outer) and in the FP64 form solved to tol_ref (the
    reference's CR with only its stop-test constant changed) from the same
    state: relative velocity error of the mixed result over the fluid
    particles (both forms keep the same particle order).  pre > 0: the mixed
    case first takes `pre` steps (so that a step with solver history is
    measured) and every form starts from its state.  setup(case) sets the
    mixed form's options.  extra: also the mixed form at the reference's
    1e-6 and the FP64 form at 1e-6 against the same tight solve (returned as
    a dict of lists)."""
    errs, e_m6, e_f6 = [], [], []
    for params, parts, dim in cases:
        runs = [(prec_fp64, tol_ref), (prec_mixed, tol_outer)]
        if extra:
            runs += [(prec_mixed, 1e-6), (prec_fp64, 1e-6)]
        start = None
        if pre > 0:
            m = engine.Case(params, parts, dim, precision=prec_mixed)
            m.set_solver(tol_outer, 1e-3, 50)
            if setup:
                setup(m)
            m.step(pre)
            f = m.fields(("id", "type", "pos", "vel"))
            import mphimplicit_gb300.casegen as cg
            start = (cg.Particles(m.time(), parts.spacing, parts.domain_min, parts.domain_max, f["type"], f["pos"], f["vel"]),
                     f["id"], m.export("WallCenter"), m)
        out = []
        for prec, tol in runs:
            if start is not None and prec == prec_mixed and tol == tol_outer:
                g = start[3]                     # the case with its history
            else:
                g = engine.Case(params, parts, dim, precision=prec)
                if start is not None:
                    g.set_state(start[0], start[1], start[2])
            g.set_solver(tol, 1e-3, 50)
            if prec == prec_mixed and setup and g is not (start[3] if start else None):
                setup(g)
            g.step(1)
            out.append(g.fields(("id", "type", "vel")))
            g.close()
        ref = out[0]
        fl = ref["type"] < 2
        nv = max(np.linalg.norm(ref["vel"][fl]), 1e-300)
        for f in out[1:]:
            assert np.array_equal(f["id"], ref["id"])
        errs.append(float(np.linalg.norm(out[1]["vel"][fl] - ref["vel"][fl]) / nv))
        if extra:
            e_m6.append(float(np.linalg.norm(out[2]["vel"][fl] - ref["vel"][fl]) / nv))
            e_f6.append(float(np.linalg.norm(out[3]["vel"][fl] - ref["vel"][fl]) / nv))
    if extra:
        return {"mixed": errs, "mixed_1e-6": e_m6, "fp64_1e-6": e_f6}
    return errs


def _fp64_sequential_ms(engine, cases, prec_fp64):
    """Per-step time of each case run alone in the plain FP64 form (one warm-up
    step, one timed step, CUDA events on the legacy stream)."""
    import torch
    out = []
    for params, parts, dim in cases:
        g = engine.Case(params, parts, dim, precision=prec_fp64)
        g.step(1)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        e0.record(torch.cuda.default_stream())
        g.step(1)
        e1.record(torch.cuda.default_stream())
        torch.cuda.synchronize()
        out.append(e0.elapsed_time(e1))
        g.close()
    return out


def cpu_cases_sample(cases, budget_s: float = 20.0):
    """The oracle (OpenMP over all host cores) on a sample of the batched
    workload's cases, one full step each after the untimed initial pass, in
    order until about budget_s seconds of stepping: particle-steps/s."""
    import oracle as orc
    orc.build_oracle()
    threads = os.cpu_count() or 1
    psteps, secs, used = 0, 0.0, 0
    for params, parts, dim in cases:
        o = orc.Oracle(params, parts, dim, threads=threads)
        o.init()
        t0 = time.perf_counter()
        o.step(1)
        secs += time.perf_counter() - t0
        psteps += parts.count
        used += 1
        if secs >= budget_s:
            break
    return {"value": psteps / secs, "unit": UNIT, "cores": threads, "kind": "port",
            "sample": f"{used} of the workload's cases (in the listed order), one full step each after the initial pass, "
                      f"{psteps} particle-steps in {secs:.1f} s wall"}


def case_roofline(engine, params, parts, dim, args, steps: int = 3):
    """Roofline of the inner operator on one case of a batched workload run
    alone (mixed form, the bench's options, CUDA events inside the CR graph)."""
    from mphimplicit_gb300.cabi import PRECISION_MIXED
    g = engine.Case(params, parts, dim, precision=PRECISION_MIXED)
    g.set_solver(args.outer_tol, args.inner_tol, 50)
    g.set_option("extrapolate", args.extrapolate)
    g.set_option("dense_coarse", args.dense_coarse)
    g.step(2)
    g.profile(True)
    g.step(steps)
    prof = g.profile_read()
    g.profile(False)
    scal, st = g.scalars(), g.solve_stats()
    g.close()
    n = max(prof["kern_n_spmv"], 1)
    avg = prof["kern_ms_spmv"] / 1000.0 / n
    pen = st.get("inner_form") == 2
    b = pen_apply_bytes(prof, scal, dim, st) if pen else spmv_bytes(prof, scal, dim, 4)
    peak, kind = measured_peaks()
    return {"bound": "hbm", "achieved": b / avg / 1e9, "peak": peak, "unit": "GB/s", "frac": b / avg / 1e9 / peak,
            "traffic": None, "kernel": "k_pen_t+k_pen_y" if pen else "k_spmv32",
            "peak_source": kind, "algorithmic_bytes_per_launch": b, "avg_launch_ms": avg * 1000.0, "launches": n,
            "case": f"{parts.count} particles ({dim}D), run alone"}


def run_ensemble(args, line_base):
    """Batched 2D ensemble (512 cases by default): every timed step advances
    every case once, all cases concurrently (mph_batch_step)."""
    import torch
    from mphimplicit_gb300 import engine, serving
    from mphimplicit_gb300.cabi import PRECISION_FP64, PRECISION_MIXED
    prec = PRECISION_MIXED if args.precision == "mixed" else PRECISION_FP64
    ens = casegen.ensemble_2d(args.cases, seed=1)

    def setup(g):
        g.set_solver(args.outer_tol, args.inner_tol, 50)
        g.set_option("extrapolate", args.extrapolate)
        g.set_option("dense_coarse", args.dense_coarse)
        g.set_option("device_loop", args.device_loop)
        g.set_option("mg_depth", args.mg_depth)
        g.set_option("batch_solve", args.batch_solve)

    table = None
    if prec == PRECISION_MIXED and args.autotune:
        # the project autotuner: one tuning per size class (octave of the
        # fluid count), on the first case of each class
        from mphimplicit_gb300 import autotune

        def make(i):
            g = engine.Case(ens[i][0], ens[i][1], 2, precision=prec)
            setup(g)
            return g
        nfl = [int((parts.types < 2).sum()) for _, parts in ens]
        table = autotune.tune_table(((2, nfl[i], i) for i in range(len(ens))), make, steps=2, warmup=1)
    cases = []
    for params, parts in ens:
        g = engine.Case(params, parts, 2, precision=prec)
        if prec == PRECISION_MIXED:
            setup(g)
            if table:
                from mphimplicit_gb300 import autotune
                autotune.apply(g, autotune.choose(table, 2, g.fluid_count))
        cases.append(g)
    N = sum(g.count for g in cases)
    for _ in range(args.warmup):
        serving.batch_step(cases, 1, args.workers)
    torch.cuda.synchronize()
    evs = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps + 1)]
    l0 = engine.launch_count()
    with Clocks(0) as clk:
        evs[0].record(torch.cuda.default_stream())
        for k in range(args.steps):
            serving.batch_step(cases, 1, args.workers)
            evs[k + 1].record(torch.cuda.default_stream())
        torch.cuda.synchronize()
    launches = engine.launch_count() - l0
    step_ms = [evs[k].elapsed_time(evs[k + 1]) for k in range(args.steps)]
    total_s = sum(step_ms) / 1000.0
    value = N * args.steps / total_s
    # end to end: the same cases go on for K more steps, each step uploading
    # every case's state from pinned host buffers (the state continuing the
    # case's own steps) and reading it back after the batched step; the
    # per-case copies on a host thread pool (ctypes releases the GIL)
    e2e_value, e2e_bytes = None, 0
    e2e_steps = args.steps if args.e2e_steps < 0 else args.e2e_steps
    if e2e_steps > 0:
        from concurrent.futures import ThreadPoolExecutor

        def pinned(shape, dt):
            return torch.empty(shape, dtype=dt, pin_memory=True).numpy()
        bufs = []
        for g in cases:
            n = g.count
            f = {"id": pinned((n,), torch.int32), "type": pinned((n,), torch.int32), "pos": pinned((n, 3), torch.float64),
                 "vel": pinned((n, 3), torch.float64)}
            g.fields(out=f)
            if prec == PRECISION_MIXED:
                g.set_option("keep_history", 1)
            bufs.append(f)

        def up(k):
            g, f, parts = cases[k], bufs[k], ens[k][1]
            g.set_state(casegen.Particles(g.time(), parts.spacing, parts.domain_min, parts.domain_max, f["type"], f["pos"],
                                          f["vel"]), f["id"])

        def down(k):
            cases[k].fields(out=bufs[k])
        with ThreadPoolExecutor(max_workers=args.workers) as pool:
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            for _ in range(e2e_steps):
                list(pool.map(up, range(len(cases))))
                serving.batch_step(cases, 1, args.workers)
                list(pool.map(down, range(len(cases))))
            torch.cuda.synchronize()
            e2e_s = time.perf_counter() - t0
        e2e_value = N * e2e_steps / e2e_s
        e2e_bytes = N * (3 * 8 * 2 + 4 + 4)
    for g in cases:
        g.close()
    # plain FP64 form, one case after the other, on an evenly spaced sample
    idx = list(range(0, len(ens), max(1, len(ens) // args.sample)))[:args.sample]
    sample = [(ens[i][0], ens[i][1], 2) for i in idx]
    seq_ms = _fp64_sequential_ms(engine, sample, PRECISION_FP64)
    plain = sum(ens[i][1].count for i in idx) / (sum(seq_ms) / 1000.0)
    errs = _vel_error_vs_fp64(engine, sample[:4], PRECISION_MIXED, PRECISION_FP64, args.outer_tol) \
        if prec == PRECISION_MIXED else []
    mid = sorted(range(len(ens)), key=lambda i: ens[i][1].count)[len(ens) // 2]
    roof = case_roofline(engine, ens[mid][0], ens[mid][1], 2, args) if prec == PRECISION_MIXED else None
    cpu = None if args.no_cpu_baseline else cpu_cases_sample(sample)
    line = dict(line_base)
    line.update({
        "roofline": roof, "cpu_baseline": cpu,
        "value": value, "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1000.0 * total_s / args.steps,
        "dtype": "f64" if prec == PRECISION_FP64 else "f32-inner/f64-outer",
        "config": {"workload": "ensemble2d", "description": f"{len(ens)} independent 2D cases, fluid n x m, n,m ~ U[40,250] "
                   "(seed 1), mu log-uniform [0.01,1], gravity angle U[0,30], two fluid types in half (config 3); "
                   "one step = every case advanced once, all concurrently", "cases": len(ens), "particles": N,
                   "precision": args.precision, "workers": args.workers, "parallelism": "single",
                   "outer_tol": args.outer_tol if prec == PRECISION_MIXED else 1e-6,
                   "cr_start": "quadratic extrapolation" if args.extrapolate == 2 and prec == PRECISION_MIXED else "v_n",
                   "preconditioner": precond_name(args, prec == PRECISION_MIXED),
                   "autotune": {k: v["settings"] for k, v in table.items()} if table else None,
                   "l2": "inputs larger than L2 (the cases' matrices total ~GBs)",
                   "p50_step_ms": float(np.percentile(step_ms, 50)), "p99_step_ms": float(np.percentile(step_ms, 99)),
                   "plain_fp64_sequential_value": plain,
                   "plain_fp64_sample": f"{len(idx)} evenly spaced cases, one step each, alone, FP64 form",
                   "speedup_vs_plain_fp64_sequential": value / plain,
                   "vel_rel_err_vs_fp64_per_step": errs},
        "gpu_launches": launches, "clocks": clk.summary(),
        "e2e": {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": e2e_bytes, "d2h_bytes_per_step": e2e_bytes,
                "steps": e2e_steps, "note": "every case's state uploaded from and read back into pinned host buffers each step"},
    })
    print(json.dumps(line), flush=True)
    return 0


def run_serve(args, line_base):
    """Serving loop: Poisson arrivals (20 cases/s, seed 2) of 2D and 3D cases
    of 1e4..5e5 particles, admitted by device-memory footprint under a 150 GB
    budget, stepped concurrently; steps per case scaled by --serve-step-scale."""
    import threading
    import torch
    from mphimplicit_gb300 import engine, serving
    from mphimplicit_gb300.cabi import PRECISION_FP64, PRECISION_MIXED
    prec = PRECISION_MIXED if args.precision == "mixed" else PRECISION_FP64
    reqs = casegen.serving_requests(args.cases, seed=2, step_scale=args.serve_step_scale)
    srv = serving.Server(int(150e9), workers=args.workers)
    if prec == PRECISION_MIXED:
        srv.set_solver(args.outer_tol, args.inner_tol, 50)
        srv.set_option("extrapolate", args.extrapolate)
        srv.set_option("dense_coarse", args.dense_coarse)
        srv.set_option("device_loop", args.device_loop)
        srv.set_option("mg_depth", args.mg_depth)
    lock = threading.Lock()
    tickets = {}
    t0 = time.perf_counter()

    def submitter():
        for k, r in enumerate(reqs):
            dt = r["t"] - (time.perf_counter() - t0)
            if dt > 0:
                time.sleep(dt)
            t = srv.submit(r["params"], r["parts"], r["dim"], r["steps"], precision=prec, fields=("id",))
            with lock:
                tickets[t] = k

    th = threading.Thread(target=submitter)
    l0 = engine.launch_count()
    with Clocks(0) as clk:
        th.start()
        results = []
        while len(results) < len(reqs):
            results += srv.poll(wait_ms=100)
        th.join()
        torch.cuda.synchronize()
    launches = engine.launch_count() - l0
    stats = srv.stats()
    srv.close()
    bad = [r for r in results if r["status"] not in (0, 7)]
    if bad:
        raise SystemExit(f"served case failed: {bad[0]['error']}")
    first = min(r["submit_s"] for r in results)
    last = min(max(r["done_s"] for r in results), stats["elapsed_s"])
    span = max(r["done_s"] for r in results) - first
    psteps = sum(r["particles"] * r["steps"] for r in results)
    value = psteps / span
    step_ms = np.concatenate([r["step_ms"] for r in results])
    lat = np.array([r["done_s"] - r["submit_s"] for r in results])
    # plain FP64 form, the same requests one after the other (per-step time of
    # each request alone x its steps)
    sample = [(r["params"], r["parts"], r["dim"]) for r in reqs]
    seq_ms = _fp64_sequential_ms(engine, sample, PRECISION_FP64)
    seq_s = sum(ms / 1000.0 * r["steps"] for ms, r in zip(seq_ms, reqs))
    plain = psteps / seq_s
    errs = _vel_error_vs_fp64(engine, sample[:4], PRECISION_MIXED, PRECISION_FP64, args.outer_tol) \
        if prec == PRECISION_MIXED else []
    mid = sorted(range(len(reqs)), key=lambda i: reqs[i]["parts"].count)[len(reqs) // 2]
    roof = case_roofline(engine, reqs[mid]["params"], reqs[mid]["parts"], reqs[mid]["dim"], args) \
        if prec == PRECISION_MIXED else None
    cpu = None if args.no_cpu_baseline else cpu_cases_sample(sample)
    line = dict(line_base)
    line.update({
        "roofline": roof, "cpu_baseline": cpu,
        "value": value, "steps": int(sum(r["steps"] for r in results)), "warmup": 0,
        "ms_per_step": float(np.mean(step_ms)), "dtype": "f64" if prec == PRECISION_FP64 else "f32-inner/f64-outer",
        "config": {"workload": "serve", "description": f"{len(reqs)} requests, Poisson arrivals 20/s (seed 2), 2D and 3D, "
                   "1e4..5e5 particles log-uniform, steps U[50,400] x step scale, 150 GB admission budget (config 4)",
                   "requests": len(reqs), "step_scale": args.serve_step_scale, "precision": args.precision,
                   "outer_tol": args.outer_tol if prec == PRECISION_MIXED else 1e-6,
                   "preconditioner": precond_name(args, prec == PRECISION_MIXED),
                   "workers": args.workers, "parallelism": "single", "particle_steps": psteps, "span_s": span,
                   "l2": "inputs larger than L2",
                   "p50_step_ms": float(np.percentile(step_ms, 50)), "p99_step_ms": float(np.percentile(step_ms, 99)),
                   "p50_completion_s": float(np.percentile(lat, 50)), "p99_completion_s": float(np.percentile(lat, 99)),
                   "plain_fp64_sequential_value": plain,
                   "plain_fp64_sample": "every request alone in the FP64 form: one timed step x its step count",
                   "speedup_vs_plain_fp64_sequential": value / plain,
                   "vel_rel_err_vs_fp64_per_step": errs},
        "gpu_launches": launches, "clocks": clk.summary(),
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": None, "d2h_bytes_per_step": None,
                "note": "requests are submitted from host memory and their fields returned to host buffers"},
    })
    print(json.dumps(line), flush=True)
    return 0


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="gb300", choices=["gb300", "reference"])
    ap.add_argument("--workload", default="cube3d_100")
    ap.add_argument("--precision", default="mixed", choices=["fp64", "mixed"])
    ap.add_argument("--inner-tol", type=float, default=1e-3,
                    help="mixed form: relative residual reduction of each FP32 inner solve")
    ap.add_argument("--e2e-steps", type=int, default=-1, help="end-to-end steps (-1: the same K as the timed region)")
    ap.add_argument("--no-factored", action="store_true",
                    help="mixed form: assemble FP64 blocks instead of the factored FP64 operator")
    ap.add_argument("--extra-sweeps", type=int, default=0, help="mixed form: extra level-0 smoothing sweeps")
    ap.add_argument("--inner-blocks", type=int, default=-1, choices=[-1, 0, 1],
                    help="mixed form: inner operator on FP32 blocks (1) or sliced pair terms (0); -1 keeps the engine default")
    ap.add_argument("--extrapolate", type=int, default=2, choices=[0, 1, 2],
                    help="mixed form: start each CR solve from the linear (1) or quadratic (2) extrapolation of the "
                         "last steps' start velocities instead of v_n (0)")
    ap.add_argument("--dense-coarse", type=int, default=1, choices=[0, 1],
                    help="mixed form: solve the V-cycle's first one-block coarse level (<= 224 rows) exactly")
    ap.add_argument("--cell-sort", type=int, default=0, choices=[0, 1],
                    help="cell sort: 0 the reference's bitonic network (bit-exact order), 1 the counting sort")
    ap.add_argument("--device-loop", type=int, default=0, choices=[0, 1],
                    help="mixed form: the whole solve as one graph with device-side loops (1) or host-driven chunks (0)")
    ap.add_argument("--autotune", type=int, default=1, choices=[0, 1],
                    help="mixed form: choose the launch shapes (operator block widths, graph chunk) with the autotuner")
    ap.add_argument("--mg-pre", type=int, default=1,
                    help="mixed form: V-cycle sweeps before the coarse correction on the levels below 0 (the reference: 2)")
    ap.add_argument("--mg-post", type=int, default=1, help="mixed form: V-cycle sweeps after it (the reference: 3)")
    ap.add_argument("--mg-depth", type=int, default=-1,
                    help="mixed form preconditioner: -1 point Jacobi (no multigrid), 0 the reference's V-cycle over every "
                         "level, k >= 1 its first k levels")
    ap.add_argument("--mg-coarsest", type=int, default=4, help="mixed form: sweeps of a grid-wide coarsest level")
    ap.add_argument("--pair-recompute", type=int, default=0, choices=[0, 1],
                    help="mixed form: pair-term operator evaluates its pair terms per slot from the FP32 positions (1) or "
                         "reads them as FP16 slot records (0)")
    ap.add_argument("--pair-pack", type=int, default=1, choices=[0, 1],
                    help="mixed form: 6-byte slot records of the pair-term operator (packed g + 2-byte index; 0: FP16, 8 bytes)")
    ap.add_argument("--batch-solve", type=int, default=0, choices=[0, 1],
                    help="ensemble: the CR iterations of all cases in one launch per kernel (1) or each case's own (0)")
    ap.add_argument("--split-apply", type=int, default=0, choices=[0, 1],
                    help="mixed form: the operator's transposed apply beside its viscous kernel (1) or before it (0)")
    ap.add_argument("--no-fp64-leg", action="store_true", help="mixed form: skip the plain FP64 comparison run")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--cpu-fluid", type=int, default=100,
                    help="CPU baseline sample: the config-1 geometry at this fluid edge (100: the workload itself)")
    ap.add_argument("--ref-max-steps", type=int, default=8,
                    help="reference arm: time at most this many of the K steps after at most 2 warm-up steps (a CPU "
                         "step of the config-1 workload takes ~15 s; its CR takes the same iterations every step)")
    ap.add_argument("--ref-fluid", type=int, default=0,
                    help="reference arm: time the config-1 geometry scaled to this fluid edge instead of the workload (0)")
    ap.add_argument("--outer-tol", type=float, default=None,
                    help="mixed form: FP64 outer relative residual (default 1e-10 for the single-case workloads, the "
                         "mixed-precision configuration's refinement; 1e-8 for ensemble2d / serve; the reference's own "
                         "tolerance is 1e-6)")
    ap.add_argument("--cases", type=int, default=0, help="ensemble / serve: number of cases (0: 512 / 24)")
    ap.add_argument("--workers", type=int, default=64, help="ensemble / serve: host worker threads")
    ap.add_argument("--sample", type=int, default=16, help="ensemble: cases timed alone in the FP64 form")
    ap.add_argument("--serve-step-scale", type=float, default=1.0,
                    help="serve: factor on each request's step count (1: the configured 50-400 steps)")
    args = ap.parse_args()
    if args.workload in ("ensemble2d", "serve") and args.cases <= 0:
        args.cases = 512 if args.workload == "ensemble2d" else 24
    if args.outer_tol is None:
        # the config-1 mixed configuration refines to 1e-10; the batched
        # workloads (no tolerance stated) to 1e-8, two orders inside the
        # 1e-6 velocity accuracy (reported on every line)
        args.outer_tol = 1e-8 if args.workload in ("ensemble2d", "serve") else 1e-10

    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        return run_reference(args, rank, world)

    import torch
    torch.cuda.set_device(local)
    dist = None
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("nccl", init_method="env://")
    from mphimplicit_gb300 import build, engine
    from mphimplicit_gb300.cabi import PRECISION_FP64, PRECISION_MIXED
    if rank == 0 or world == 1:
        build.build()
    if dist:
        dist.barrier()
    if args.workload in ("ensemble2d", "serve"):
        base = {"metric": METRIC, "unit": UNIT, "n_gpus": world, "higher_is_better": True, "scaling": "weak",
                "vs_baseline": None, "data": "synthetic", "roofline": None, "cpu_baseline": None}
        return run_ensemble(args, base) if args.workload == "ensemble2d" else run_serve(args, base)
    return run_single(args, dist, rank, world, local)


def run_single(args, dist, rank, world, local):
    """One case of the named workload, resident on the GPU (the headline)."""
    import torch
    from mphimplicit_gb300 import engine
    from mphimplicit_gb300.cabi import PRECISION_FP64, PRECISION_MIXED
    dim, params, parts, desc = workload(args.workload)
    stream = torch.cuda.Stream()
    prec = PRECISION_MIXED if args.precision == "mixed" else PRECISION_FP64
    tol = args.outer_tol if prec == PRECISION_MIXED else 1e-6

    def make(prec_, tol_):
        c = engine.Case(params, parts, dim, precision=prec_, stream=stream.cuda_stream)
        c.set_solver(tol_, args.inner_tol, 50)
        if prec_ == PRECISION_MIXED:
            c.set_option("factored", 0 if args.no_factored else 1)
            c.set_option("mixed_extra_sweeps", args.extra_sweeps)
            if args.inner_blocks >= 0:
                c.set_option("inner_blocks", args.inner_blocks)
            c.set_option("extrapolate", args.extrapolate)
            c.set_option("dense_coarse", args.dense_coarse)
            c.set_option("mg_pre", args.mg_pre)
            c.set_option("mg_post", args.mg_post)
            c.set_option("pair_recompute", args.pair_recompute)
            c.set_option("pair_pack", args.pair_pack)
            c.set_option("mg_depth", args.mg_depth)
            c.set_option("mg_coarsest", args.mg_coarsest)
            c.set_option("split_apply", args.split_apply)
        c.set_option("cell_sort", args.cell_sort)
        c.set_option("device_loop", args.device_loop)
        if prec_ == PRECISION_MIXED and getattr(args, "tuned_settings", None):
            for k, v in args.tuned_settings.items():
                c.set_option(k, v)
        return c

    def timed(c, steps, warmup, clocks=None, profile=False):
        """Per-step CUDA-event milliseconds (case stream) and CR iterations
        of `steps` steps after `warmup` untimed ones."""
        for _ in range(warmup):
            c.step(1)
        torch.cuda.synchronize()
        if dist:
            dist.barrier()
        if profile:
            c.profile(True)
        evs = [torch.cuda.Event(enable_timing=True) for _ in range(steps + 1)]
        its, outs = [], []
        l0 = engine.launch_count()
        with (clocks if clocks is not None else _Null()):
            torch.cuda.synchronize()
            evs[0].record(stream)
            for k in range(steps):
                c.step(1)
                evs[k + 1].record(stream)
                ss = c.solve_stats()
                its.append(ss["iter"])
                outs.append(ss["outer"])
            torch.cuda.synchronize()
        launches = engine.launch_count() - l0
        if dist:
            dist.barrier()
        timed.outer = outs
        return [evs[k].elapsed_time(evs[k + 1]) for k in range(steps)], its, launches

    tuned = None
    if prec == PRECISION_MIXED and args.autotune:
        # the project autotuner: launch shapes of this workload's mixed form by
        # coordinate descent over whole steps of fresh copies of the case
        from mphimplicit_gb300 import autotune
        tuned = autotune.tune(lambda: make(prec, tol), steps=3, warmup=2)
        args.tuned_settings = tuned["settings"]
    case = make(prec, tol)
    N, Nf = case.count, case.fluid_count
    clk = Clocks(local)
    # the timed region runs without instrumentation (the mixed solve is then
    # one graph launch with device-side loops); the per-stage and per-kernel
    # times come from a short profiled pass after it (the same kernels, the
    # solve driven from the host so that event pairs can bracket them)
    step_ms, iters, launches = timed(case, args.steps, args.warmup, clk, profile=False)
    outer_main = list(timed.outer)
    total_s = sum(step_ms) / 1000.0
    value, total_s = replica_throughput(N * args.steps, total_s, dist, "cuda")
    psteps = max(1, min(args.steps, 4))
    case.profile(True)
    for _ in range(psteps):
        case.step(1)
    prof = case.profile_read()
    case.profile(False)
    scal = case.scalars()
    st = case.solve_stats()

    # end to end through the public API with host buffers (pinned): a fresh
    # case over the same simulation steps as the timed region (the same W
    # untimed warm-up steps), every timed step uploading the state and reading
    # it back (the wall centres stay on the case: mph_case_set_state keeps
    # them when given none)
    e2e_steps = args.steps if args.e2e_steps < 0 else args.e2e_steps
    if e2e_steps > 0:
        case.close()
        case = make(prec, tol)
        for _ in range(args.warmup):
            case.step(1)

    def pinned(shape, dt):
        return torch.empty(shape, dtype=dt, pin_memory=True).numpy()
    fields = {"id": pinned((N,), torch.int32), "type": pinned((N,), torch.int32), "pos": pinned((N, 3), torch.float64),
              "vel": pinned((N, 3), torch.float64)}
    case.fields(out=fields)
    host = casegen.Particles(case.time(), parts.spacing, parts.domain_min, parts.domain_max, fields["type"], fields["pos"],
                             fields["vel"])
    ids = fields["id"]
    if prec == PRECISION_MIXED:   # the uploaded state continues this case's steps
        case.set_option("keep_history", 1)
    h2d = N * (3 * 8 * 2 + 4 + 4)
    d2h = N * (3 * 8 * 2 + 4 + 4)
    e2e_value = None
    if e2e_steps > 0:
        torch.cuda.synchronize()
        if dist:
            dist.barrier()
        t0 = time.perf_counter()
        for _ in range(e2e_steps):
            case.set_state(host, ids)
            case.step(1)
            case.fields(out=fields)   # read back into the same pinned buffers
            host = casegen.Particles(case.time(), parts.spacing, parts.domain_min, parts.domain_max, fields["type"],
                                     fields["pos"], fields["vel"])
        torch.cuda.synchronize()
        e2e_s = time.perf_counter() - t0
        e2e_value, _ = replica_throughput(N * e2e_steps, e2e_s, dist, "cuda")

    # roofline of the dominant kernel (CUDA events on the case stream) and of
    # the assembly stage
    peak, peak_kind = measured_peaks()
    vb = 4 if prec == PRECISION_MIXED else 8
    pairs = st.get("inner_form") == 2
    rec = "recompute" if args.pair_recompute else ("pack" if args.pair_pack else "fp16")
    pen = pairs and args.mg_depth < 0   # the point-Jacobi form's own operator
    parts64 = prec == PRECISION_FP64 and dim == 3 and not args.no_factored
    kern = {"spmv": ("k_pen_t+k_pen_y", lambda p_, s_, d_: pen_apply_bytes(p_, s_, d_, st)) if pen else
                    ("k_f64_parts+k_f64_rows", f64_parts_bytes) if parts64 else
                    ("k_ct_apply32+k_visc_pen32" if rec != "recompute" else "k_ct_apply32+k_visc_rc32",
                     lambda p_, s_, d_: pair_apply_bytes(p_, s_, d_, st, rec)) if pairs else
                    ("k_spmv32" if vb == 4 else "k_spmv", lambda p_, s_, d_: spmv_bytes(p_, s_, d_, vb)),
            "assemble_a": ("k_assemble_cells", assemble_bytes)}
    dom = max(kern, key=lambda k: prof[f"kern_ms_{k}"])
    nlaunch = max(prof[f"kern_n_{dom}"], 1)
    avg_s = prof[f"kern_ms_{dom}"] / 1000.0 / nlaunch
    bytes_per = kern[dom][1](prof, scal, dim)
    achieved = bytes_per / avg_s / 1e9
    roofline = {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s", "frac": achieved / peak,
                "traffic": ncu_traffic(kern[dom][0], bytes_per) if args.workload == "cube3d_100" else None,
                "kernel": kern[dom][0], "peak_source": peak_kind,
                "algorithmic_bytes_per_launch": bytes_per, "avg_launch_ms": avg_s * 1000.0, "launches": nlaunch}
    asm_ms = prof["stage_ms_assemble"] / psteps
    asm_bytes = (assemble_pen_bytes(prof, scal, dim) if pen else
                 assemble_pair_bytes(prof, scal, dim, case, jacobi=args.mg_depth < 0,
                                     rec_bytes={"pack": 6, "fp16": 8, "recompute": 2}[rec]) if pairs
                 else assemble_bytes(prof, scal, dim))
    roofline_asm = {"bound": "hbm", "achieved": asm_bytes / (asm_ms / 1000.0) / 1e9, "peak": peak, "unit": "GB/s",
                    "frac": asm_bytes / (asm_ms / 1000.0) / 1e9 / peak, "stage": "assemble",
                    "algorithmic_bytes_per_step": asm_bytes, "ms_per_step": asm_ms, "peak_source": peak_kind,
                    "form": "C, b and D^-1 (point-Jacobi mixed)" if pen else
                    "pair terms (mixed)" if pairs else "sliced-ELL blocks"}
    case.close()

    cpu = None
    if rank == 0 and not args.no_cpu_baseline:
        cpu = cpu_sample(os.cpu_count() or 1, 1, args.cpu_fluid, check_gpu=True)

    # the plain FP64 form on the same workload (for the mixed form's
    # speed-up), the mixed form at the reference's 1e-6 (secondary), and one
    # step of each form from the same state against the FP64 form solved to
    # 1e-12 (the accuracy of the metric)
    plain = None
    errs = {}
    secondary = None
    if prec == PRECISION_MIXED and not args.no_fp64_leg:
        f = make(PRECISION_FP64, 1e-6)
        ms, its, _ = timed(f, args.steps, args.warmup)
        plain = N * args.steps / (sum(ms) / 1000.0)
        plain_iters = its
        f.close()
        m6 = make(PRECISION_MIXED, 1e-6)
        ms6, its6, _ = timed(m6, args.steps, args.warmup)
        m6.close()
        secondary = {"outer_tol": 1e-6, "value": N * args.steps / (sum(ms6) / 1000.0), "cr_iterations": its6,
                     "note": "mixed form stopped at the reference's own 1e-6; its velocity differs from the 1e-12 FP64 "
                             "solve by vel_rel_err_vs_fp64_1e-12.mixed_1e-6 (not the headline)"}
        def setup(c):
            c.set_option("factored", 0 if args.no_factored else 1)
            c.set_option("mixed_extra_sweeps", args.extra_sweeps)
            if args.inner_blocks >= 0:
                c.set_option("inner_blocks", args.inner_blocks)
            c.set_option("extrapolate", args.extrapolate)
            c.set_option("dense_coarse", args.dense_coarse)
            c.set_option("mg_pre", args.mg_pre)
            c.set_option("mg_post", args.mg_post)
            c.set_option("pair_recompute", args.pair_recompute)
            c.set_option("pair_pack", args.pair_pack)
            c.set_option("mg_depth", args.mg_depth)
            c.set_option("mg_coarsest", args.mg_coarsest)
            c.set_option("split_apply", args.split_apply)
            for k, v in (getattr(args, "tuned_settings", None) or {}).items():
                c.set_option(k, v)
        errs = _vel_error_vs_fp64(engine, [(params, parts, dim)], PRECISION_MIXED, PRECISION_FP64, args.outer_tol,
                                  extra=True, pre=args.warmup, setup=setup)
    max_err = max(errs["mixed"]) if errs else None

    stage_total = sum(prof[f"stage_ms_{s}"] for s in ("step_begin", "cellsort", "neighbors", "explicit", "assemble", "mg_build", "solve"))
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": 1000.0 * total_s / args.steps, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "f64" if prec == PRECISION_FP64 else "f32-inner/f64-outer" if pen else
                 (f"f32-inner({ {'fp16': 'fp16', 'pack': '11/11/10-bit fixed-point', 'recompute': 'recomputed fp32'}[rec]} "
                  f"pair terms)/f64-outer" if pairs else "f32-inner/f64-outer"),
        "data": "synthetic",
        "config": {"workload": args.workload, "description": desc, "dim": dim, "particles": N, "fluid": Nf,
                   "precision": args.precision, "parallelism": "replicas" if world > 1 else "single",
                   "l2": "inputs larger than L2 (the neighbour lists alone exceed 129 MB by ~5x)",
                   "p50_step_ms": float(np.percentile(step_ms, 50)), "p99_step_ms": float(np.percentile(step_ms, 99)),
                   "outer_tol": tol, "cr_iterations": iters, "outer_refinements": outer_main,
                   "cr_start": {0: "v_n (the reference's)", 1: "linear extrapolation of the last start velocities",
                                2: "quadratic extrapolation of the last start velocities"}[args.extrapolate]
                   if prec == PRECISION_MIXED else "v_n (the reference's)",
                   "preconditioner": precond_name(args, prec == PRECISION_MIXED),
                   "inner_row_blocks": {"staged": st.get("inner_local_blocks"), "gathering": st.get("inner_gather_blocks"),
                                        "ct_blocks_staging_s": st.get("inner_ct_local_blocks"),
                                        "mean_distinct_cols": (st["inner_local_cols"] / st["inner_local_blocks"]
                                                               if st.get("inner_local_blocks") else None)},
                   "profiled_steps": psteps,
                   "stage_ms_per_step": {s: prof[f"stage_ms_{s}"] / psteps for s in
                                         ("step_begin", "cellsort", "neighbors", "explicit", "assemble", "mg_build", "solve")},
                   "stage_sum_ms_per_step": stage_total / psteps,
                   "kernel_avg_ms": {k: (prof[f"kern_ms_{k}"] / prof[f"kern_n_{k}"] if prof[f"kern_n_{k}"] else None)
                                     for k in ("spmv", "precond", "assemble_a", "neighbors")},
                   "kernel_launches": {k: prof[f"kern_n_{k}"] for k in ("spmv", "precond", "assemble_a", "neighbors")},
                   "plain_fp64_value": plain,
                   "plain_fp64_cr_iterations": plain_iters if plain else None,
                   "speedup_vs_plain_fp64": (value / plain) if plain else None,
                   "vel_rel_err_vs_fp64_1e-12": errs or None,
                   "max_vel_rel_err": max_err,
                   "meets_1e-6": (max_err <= 1e-6) if max_err is not None else None,
                   "secondary_mixed_1e-6": secondary,
                   "autotune": tuned},
        "e2e": {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
                "steps": e2e_steps},
        "gpu_launches": launches,
        "roofline": roofline,
        "roofline_assembly": roofline_asm,
        "clocks": clk.summary(),
        "cpu_baseline": cpu,
    }
    if rank == 0:
        print(json.dumps(line), flush=True)
    if dist:
        dist.destroy_process_group()
    return 0


class _Null:
    def __enter__(self):
        return self

    def __exit__(self, *a):
        return False


if __name__ == "__main__":
    sys.exit(main())
