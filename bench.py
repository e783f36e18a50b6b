#!/usr/bin/env python3
"""Throughput of the atmosphere step: cell-steps/s on the precision-form workload.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
                    [--workload precision-512x512x256] [--mode both|plain|mixed]

One step = one environmentGPU::updateGPU of the whole grid (ground, diffusion, PPM advection,
buoyancy, projection, sedimentation, microphysics). Synthetic seeded soundings stand in for the
reference's radiosonde input. Every field is larger than L2 (268 MB per field at 512x256x512),
so timed steps do not reuse L2 contents between steps.

Printed JSON line (rank 0): value = whole-job cell-steps/s of the plain method with the
reference's semantics (the drop-in path, 200 Jacobi-PCG iterations per step) with the state
resident in HBM (CUDA events on the library stream); "mixed" = the same step with the
mixed-precision projection (FP32 multigrid-preconditioned CG inside float-float iterative
refinement to a relative residual of 1e-8) and its speed-up over plain; e2e = the headline
metric through the C ABI from host buffers (init H2D + per-step readback of every prognostic
field, as the reference's per-step GPUSetEnv does, overlapped with the next step); roofline = the dominant kernel's algorithmic
bytes / its event-timed launch duration against the measured HBM copy bandwidth; step_roofline =
algorithmic bytes of the whole step x cell-steps/s against the same peak; cpu_baseline = the
oracle (CPU restatement) on the host cores on a bounded sub-box sample (all threads, and one
thread on a smaller box).

Multi-GPU: the path does not shard (one domain per GPU); N>1 runs N independent replicas, one
per rank, with no collective on the data path ("replicas only").
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

import numpy as np  # noqa: E402

METRIC = "cell-steps/s at 512x512x256, mixed vs plain PCG at 1e-5 rel err; % HBM roofline"

# Algorithmic bytes per cell per launch of each profiled stage (FP32 fields; each array counted
# once per launch; neighbour re-reads excluded).
STAGE_BYTES = {
    # a two-launch PCG iteration with stored coefficients, the model of step_bytes; the library's own
    # iterations are PLAIN_FORMS'
    "pcg_matvec": 40.0,   # z, s_old, aw, ax, ay, az read; p read+write; s_new, As write
    "pcg_update": 20.0,   # r read+write; As, aw read; z write
    "pcg_search": 16.0,   # r, aw read; s read+write
    "diffuse": 8.0,       # per sweep: in read, out write
    "advect": 12.0,       # per pass: q, vel read; out write
    "micro": 64.0,        # 6 Q + th read/write, rho, p read (fused addHeat)
    "precip": 36.0,       # qr, qs, qi read+write; th, qv, p read (one march for the three species)
    "buoyancy": 36.0,
    "eos": 16.0,
    "proj_setup": 48.0,
    "proj_apply": 44.0,
    "mg_matvec": 32.0,    # z, s_old, ax, ay, az, aw read; s_new, As write
    "mg_update": 24.0,    # s, As read; e, r read+write
}


# The plain PCG's three forms: bytes per cell of a launch of each profiled stage, and of an iteration.
# Matrix-free (above about a million cells, nx % 4 == 0): the operator reads z, s_old, the reciprocal density
# and one word and writes s_new and As (24 B); the residual's 20 B and, every fourth iteration, the pressure's
# 24 B (four directions read, p read+write) share a stage of five launches in four iterations. Three launches
# (--pcg-fused 0, or any nx above a million cells): s, ax, ay, az, aw read and As written; s, As, aw read, p
# and r read+write; r, aw read and s read+write. One launch (up to about a million cells): the solver's state
# stays on the chip, and HBM bounds none of it.
PLAIN_FORMS = {
    "matrix-free": ({"pcg_matvec": 24.0, "pcg_update": (4 * 20.0 + 24.0) / 5}, 50.0),
    "three launches": ({"pcg_matvec": 24.0, "pcg_update": 28.0, "pcg_search": 16.0}, 68.0),
    "one launch": ({}, 0.0),
}


def plain_form(stages):
    """Which of PLAIN_FORMS a plain step ran, by the stages that the library profiled."""
    return "one launch" if "pcg_grid" in stages else "three launches" if "pcg_search" in stages else "matrix-free"


# DRAM traffic per cell of one launch: ncu dram__bytes_read.sum + dram__bytes_write.sum of one launch at
# 512x256x256 (33554432 cells). Every array is streamed once per launch, so the traffic grows with the
# cells and is scaled to the launch size here. First of the stored-coefficient model's launches (a check of
# its bytes), then of the matrix-free form's (k_pcg_operator4, and the mean of four k_residual4 and one
# k_pressure4).
MEASURED_TRAFFIC_PER_CELL = {
    "pcg_matvec": (981.662976 + 375.963392) * 1e6 / 33554432,
    "pcg_update": (402.723840 + 224.641536) * 1e6 / 33554432,
}
FREE_TRAFFIC_PER_CELL = {
    "pcg_matvec": (554.915328 + 234.966016) * 1e6 / 33554432,
    "pcg_update": (4 * (402.703104 + 219.609088) + 671.106048 + 112.221696) / 5 * 1e6 / 33554432,
}


def dist_env():
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return rank, world, local


def max_over_ranks(x, pg, device):
    """The largest x over the ranks (the slowest rank's time); x itself with one rank. pg is the
    torch.distributed module once its process group is up (nccl on GPUs, gloo in the CPU tests)."""
    if not pg:
        return float(x)
    import torch
    t = torch.tensor([float(x)], dtype=torch.float64, device=device)
    pg.all_reduce(t, op=pg.ReduceOp.MAX)
    return float(t.item())


def whole_job_rate(units_per_rank, world, seconds):
    """Replicas: every rank processes the same units (weak scaling), so the job's rate is all ranks'
    units over the slowest rank's time."""
    return units_per_rank * world / seconds


class ClockSampler:
    """nvidia-smi clocks/throttle reasons sampled during the timed region."""

    def __init__(self, gpu_index: int):
        self.gpu = gpu_index
        self.proc = None
        self.lines = []

    def __enter__(self):
        q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--query-gpu={q}", "--format=csv,noheader,nounits",
                                          "-i", str(self.gpu), "-lms", "200"], stdout=subprocess.PIPE,
                                         stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except Exception:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self):
        sm, mx, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            f = [x.strip() for x in ln.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx = float(f[2])
            except ValueError:
                continue
            for n, v in zip(names, f[5:9]):
                if v.lower() == "active":
                    reasons.add(n)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": mx, "reasons": sorted(reasons),
                "samples": len(sm)}


def measured_peak():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            d = json.load(f)
        return float(d["hbm_gbs"]), "measured"
    except Exception:
        return 6800.0, "fallback"


def pinned_like(a):
    """A pinned host copy of a numpy array when torch is present (host->device from pinned)."""
    try:
        import torch
        t = torch.from_numpy(np.ascontiguousarray(a)).pin_memory()
        return t.numpy(), t
    except Exception:
        return np.ascontiguousarray(a), None


def cpu_baseline(workload: str, sample_shape, steps: int = 1, threads: int = 0):
    """The oracle (CPU restatement of the reference, OpenMP over the host cores) on a sub-box."""
    import oracle
    from skewtcloudsim_gb300 import sounding
    lib = oracle.lib()
    full = lib.oc_num_threads()
    if threads:
        lib.oc_set_threads(threads)
    try:
        init, dt, speed = sounding.workload(workload, scale=sample_shape)
        st = oracle.OracleState(init, np.float32)
        cfg = oracle.Config()
        t0 = time.perf_counter()
        for _ in range(steps):
            st.step(cfg, dt, speed)
        el = time.perf_counter() - t0
        used = lib.oc_num_threads()
    finally:
        lib.oc_set_threads(full)
    cells = init.nx * init.ny * init.nz
    return {"value": cells * steps / el, "unit": "cell-steps/s", "cores": used, "kind": "port",
            "sample": f"{steps} step(s) of the same workload on a {sample_shape[0]}x{sample_shape[1]}x{sample_shape[2]} "
                      f"(x,y,z; z vertical) sub-box, reference semantics, FP32, {used} thread(s), {el:.1f} s"}


CPU_SAMPLE = (128, 128, 64)  # (x, y, z), z vertical: the bounded sub-box of the CPU legs (1.05M cells)
CPU_STEPS = 10  # steps of the headline CPU leg: about 10 s on 16 Arm cores


def cpu_thread_sweep(workload: str, sample_shape):
    """The same sub-box step at 1, 2, 4, ... threads up to the host's cores (one step each)."""
    import oracle
    full = oracle.lib().oc_num_threads()
    counts, t = [], 1
    while t < full:
        counts.append(t)
        t *= 2
    counts.append(full)
    out = []
    for t in counts:
        r = cpu_baseline(workload, sample_shape, 1, threads=t)
        out.append({"threads": r["cores"], "value": round(r["value"], 1)})
    return out


# Arm CPU part numbers (/proc/cpuinfo "CPU part") of the cores these boxes use
ARM_PARTS = {"0xd4f": "Arm Neoverse V2", "0xd40": "Arm Neoverse V1", "0xd0c": "Arm Neoverse N1", "0xd49": "Arm Neoverse N2"}


def host_cpu():
    try:
        with open("/proc/cpuinfo") as f:
            for ln in f:
                if ln.lower().startswith(("model name", "cpu part", "hardware")):
                    v = ln.split(":", 1)[1].strip()
                    return f"{ARM_PARTS[v]} (CPU part {v})" if v in ARM_PARTS else v
    except Exception:
        pass
    return None


def run_reference(args, rank, world):
    if rank != 0:
        return
    sample = CPU_SAMPLE
    vals = []
    for _ in range(args.warmup):
        cpu_baseline(args.workload, sample, 1)
    t_all = []
    for _ in range(args.steps):
        r = cpu_baseline(args.workload, sample, 1)
        vals.append(r["value"])
        t_all.append(1.0 / r["value"])
    v = float(np.median(vals))
    out = {"metric": METRIC, "value": v, "unit": "cell-steps/s", "n_gpus": world, "steps": args.steps,
           "warmup": args.warmup, "ms_per_step": None, "higher_is_better": True, "scaling": "weak",
           "vs_baseline": None, "dtype": "f32", "data": "synthetic", "impl": "reference",
           "config": {"workload": args.workload, "sample": "128x128x64 sub-box per step", "parallelism": "replicas"},
           "cpu_baseline": {"value": v, "unit": "cell-steps/s", "cores": r["cores"], "kind": "port",
                            "sample": r["sample"]},
           "e2e": {"value": v, "unit": "cell-steps/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    # one whole workload the CPU finishes in seconds: the plain-64x64x32 configuration at its full size
    c1 = cpu_baseline("plain-64x64x32", (64, 64, 32), 1)
    out["full_size_run"] = {"workload": "plain-64x64x32", "value": c1["value"], "unit": "cell-steps/s",
                            "cores": c1["cores"], "same_config": True, "sample": c1["sample"]}
    out["host"] = {"nproc": os.cpu_count(), "cpu": host_cpu()}
    print(json.dumps(out), flush=True)


DIFFUSION_BYTES = 1600.0  # 10 fields x 20 sweeps x (4 B read + 4 B written) at one sweep per pass


def stage_bytes(diffuse_depth=1):
    """The library's stage bytes per cell-step (FP32, one advection substep): the hot-path scope's
    stage total with the three falling species in one march (36 B instead of 3 x 20): 2534 B, of
    which the diffusion is 1600 B at one sweep per pass and half that with two sweeps per pass."""
    return 2534.0 - DIFFUSION_BYTES + DIFFUSION_BYTES / max(diffuse_depth, 1)


def step_bytes(mode, pcg_iters, outer, diffuse_depth=1):
    """Algorithmic bytes per cell-step of the whole step: the stages (stage_bytes) plus the pressure
    solve. Plain: a model with stored coefficients in two launches, 60 B per iteration (the operator with
    the search step and the pressure update 40 B, the residual update with z = r/diag 20 B); what the
    library moves is plain_step_bytes. Mixed, as the library moves them:
    per inner iteration the operator + search (32 B), the update (24 B) and the V-cycle (93 B: four
    finest-level passes of 16-24.5 B with FP16 coefficients plus the coarser levels), per
    refinement step the float-float residual (32 B) and the correction (20 B)."""
    if mode == "plain":
        return stage_bytes(diffuse_depth) + 60.0 * pcg_iters
    return stage_bytes(diffuse_depth) + (32.0 + 24.0 + 93.0) * pcg_iters + 52.0 * max(outer, 1)


def sweeps_per_pass(tuning, nx, ground_height):
    """The diffusion's sweeps per pass: the shapes' depth where the two-sweep kernel runs (flat terrain,
    nx % 4 == 0), else one."""
    return tuning.get("diffuse_depth", 1) if nx % 4 == 0 and not np.any(ground_height) else 1


def plain_step_bytes(form, pcg_iters, diffuse_depth=1):
    """Bytes per cell-step of a plain step as the library moves them, by the PCG's form (PLAIN_FORMS)."""
    return stage_bytes(diffuse_depth) + PLAIN_FORMS[form][1] * pcg_iters


# plain_textbook: the plain Jacobi-PCG on the textbook (symmetric) operator the mixed mode solves,
# run to the reference's own stop test (max |r| <= 1e-5) without the 200-iteration cap
TEXTBOOK_MAX_ITER = 20000


def mode_config(args, mode):
    from skewtcloudsim_gb300 import SolverConfig
    g = args.graph
    if mode == "plain":
        return SolverConfig(semantics=args.semantics, precision=0, mg_half=args.mg_half, pcg_fused=args.pcg_fused, use_graph=g)
    if mode == "plain_textbook":
        return SolverConfig(semantics=1, precision=0, pcg_max_iter=TEXTBOOK_MAX_ITER, pcg_fused=args.pcg_fused, use_graph=g)
    return SolverConfig(semantics=1, precision=1, mg_half=args.mg_half, pcg_fused=args.pcg_fused, use_graph=g)


def scope_step_bytes(mode, pcg_iters, outer):
    """The scope table's algorithmic model of a cell-step: 2558 B of stages plus 52 B per Jacobi-PCG
    iteration (matrix-free: the operator's coefficients formed from the density, 4 B, instead of
    four stored coefficient arrays, 16 B) plus 40 B per refinement step. The library's own matrix-free
    iteration moves 50 B (the pressure four iterations at a time)."""
    assert mode != "mixed"  # the model has no term for the V-cycle
    return 2558.0 + 52.0 * pcg_iters


TUNING_CACHE = os.path.join(ROOT, "skewtcloudsim_gb300", "_build", "tuning.json")


def apply_tuning(args, env):
    """The launch shapes of the run: --tuning's values, else the autotuner's (cached per GPU and
    grid in the build folder, measured on the first run), else the defaults."""
    if args.tuning:
        kv = dict(item.split("=") for item in args.tuning.split(","))
        env.set_tuning(**{k: int(v) for k, v in kv.items()})
        return dict(env.get_tuning(), source="--tuning")
    if args.no_autotune:
        return dict(env.get_tuning(), source="defaults")
    t = env.autotune(TUNING_CACHE)
    return dict(env.get_tuning(), source="autotune cache" if t["from_cache"] else "autotune (measured this run)")


def run_mode(args, mode, init, dt, speed, cells, world, local, pg, torch):
    from skewtcloudsim_gb300 import Environment
    cfg = mode_config(args, mode)
    sem = cfg.semantics
    env = Environment(init.nx, init.ny, init.nz, init.voxel, cfg)
    env.init_from(init)
    tuning = apply_tuning(args, env)
    for _ in range(args.warmup):
        env.update_gpu(dt, speed)
    env.sync()

    def barrier():
        if pg:
            pg.barrier()
        torch.cuda.synchronize()

    # ---- device-resident timed region (CUDA events on the library's stream) ---------------
    barrier()
    l0 = env.stats()["kernel_launches"]
    with ClockSampler(local) as clk:
        env.update_gpu(dt, speed, nsteps=args.steps)
        barrier()
    st = env.stats()
    ms_total = st["gpu_ms"]
    launches = st["kernel_launches"] - l0
    ms_total = max_over_ranks(ms_total, pg, "cuda")
    ms_per_step = ms_total / args.steps
    value = whole_job_rate(cells * args.steps, world, ms_total / 1e3)
    # ---- per-stage profile of one more step (not timed) ----------------------------------
    env.profile(True)
    env.update_gpu(dt, speed)
    prof = env.profile_read()
    env.profile(False)
    sd = env.stats()
    env.close()
    return {"mode": mode, "semantics": "reference" if sem == 0 else "textbook", "value": value, "ms_per_step": ms_per_step,
            "tuning": tuning,
            "launches": int(launches), "clocks": clk.summary(), "prof": prof, "pcg_iters": sd["pcg_iters"],
            "outer": sd.get("outer_iters", 0), "converged": sd["converged"], "residual": sd["pcg_residual"],
            "pcg_max_iter": cfg.pcg_max_iter}


def ensemble_tuning(args, envs):
    """Launch shapes of the members: --tuning's values for all, else the defaults at the members' SM
    shares. (Measured on the 48 members: 100.3 ms per ensemble step with the defaults, 101.6 ms with
    each size's autotuned shapes, which the tuner measures on a member running alone, 103.5 and
    105.5 ms with two-sweep diffusion of 14 and 6 rows.) The shapes never change a member's bits."""
    if args.tuning:
        kv = {k: int(v) for k, v in (item.split("=") for item in args.tuning.split(","))}
        for e in envs:
            e.set_tuning(**kv)
        return dict(kv, source="--tuning")
    return {"source": "defaults at the ensemble SM shares"}


def run_ensemble(args, rank, world, local, pg, torch):
    """The batched ensemble (``--workload ensemble-48``): 48 members of uneven sizes drawn from
    {64x64x32, 96x96x64, 128x128x64, 192x192x96}, each with its own seeded sounding and bubble, all
    advanced together by skt_step_ensemble (a host thread per member, each member on its own
    stream), mixed precision unless ``--mode plain``. Metric: members x cell-steps/s over the whole
    job (host wall clock around the timed steps with a device synchronise on both sides)."""
    from skewtcloudsim_gb300 import Environment, SolverConfig, sounding, step_ensemble
    n = int(args.workload.split("-")[1])
    members = sounding.ensemble_members(n, seed=4000 + 1000 * rank)
    prec = 0 if args.mode == "plain" else 1
    envs = []
    for st, dt, speed in members:
        env = Environment(st.nx, st.ny, st.nz, st.voxel, SolverConfig(semantics=0 if prec == 0 else 1, precision=prec))
        env.init_from(st)
        envs.append(env)
    dts = [m[1] for m in members]
    cells = sum(m[0].n for m in members)
    from skewtcloudsim_gb300 import Ensemble
    ens = Ensemble(envs) if args.ensemble_runner == "graph" else None
    tuning = ensemble_tuning(args, envs)

    def advance(k):
        if ens is not None:
            ens.step(dts, 1.0, nsteps=k)
        else:
            step_ensemble(envs, dts, 1.0, nsteps=k)

    advance(args.warmup)
    if pg:
        pg.barrier()
    torch.cuda.synchronize()
    l0 = sum(e.stats()["kernel_launches"] for e in envs)
    with ClockSampler(local) as clk:
        t0 = time.perf_counter()
        advance(args.steps)
        torch.cuda.synchronize()
        t1 = time.perf_counter()
    launches = sum(e.stats()["kernel_launches"] for e in envs) - l0
    el = t1 - t0
    # the other runner on the same members, for comparison
    other = None
    if ens is not None:
        torch.cuda.synchronize()
        o0 = time.perf_counter()
        step_ensemble(envs, dts, 1.0, nsteps=args.steps)
        torch.cuda.synchronize()
        other = (time.perf_counter() - o0) / args.steps * 1e3
        ens.close()
    el = max_over_ranks(el, pg, "cuda")
    # one sequential pass for comparison: the same members stepped one after another
    torch.cuda.synchronize()
    s0 = time.perf_counter()
    for env, dt in zip(envs, dts):
        env.update_gpu(dt, 1.0, nsteps=1)
    torch.cuda.synchronize()
    seq = time.perf_counter() - s0
    for env in envs:
        env.close()
    if rank == 0:
        value = whole_job_rate(cells * args.steps, world, el)
        print(json.dumps({
            "metric": f"members x cell-steps/s, ensemble of {n} uneven members", "value": value, "unit": "cell-steps/s",
            "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": el / args.steps * 1e3,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": {"workload": args.workload, "members": n, "cells": cells, "pcg": "mixed" if prec else "plain",
                       "sizes": sorted({f"{m[0].nx}x{m[0].nz}x{m[0].ny}" for m in members}),
                       "concurrency": ("one CUDA graph launch per ensemble step, every member's whole step an independent "
                                       "branch (loops as device-side conditional nodes)" if ens is not None
                                       else "one host thread per member, one stream per member"),
                       "host_thread_runner_ms_per_step": other, "tuning": tuning,
                       "sequential_ms_per_step": seq * 1e3, "parallelism": "single" if world == 1 else f"replicas{world}"},
            "gpu_launches": launches, "clocks": clk.summary()}), flush=True)
    return 0


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default="precision-512x512x256")
    ap.add_argument("--mode", default="both", choices=["plain", "mixed", "plain_textbook", "both"],
                    help="both: plain (reference semantics, the headline), mixed and plain_textbook (reported beside it)")
    ap.add_argument("--semantics", type=int, default=0)
    ap.add_argument("--mg-half", type=int, default=1, help="mixed: FP16 finest-level coefficients in the V-cycle")
    ap.add_argument("--pcg-fused", type=int, default=1,
                    help="plain: 1 = the PCG in one launch up to about a million cells, above that (nx %% 4 == 0) matrix-free in "
                         "two launches per iteration; 0 = three launches per iteration from stored coefficients")
    ap.add_argument("--graph", type=int, default=1,
                    help="1 = each step one launch of the captured CUDA graph (device-side loops), 0 = stream-ordered")
    ap.add_argument("--ensemble-runner", default="graph", choices=["graph", "threads"],
                    help="ensemble workloads: one graph launch per step for all members, or a host thread per member")
    ap.add_argument("--tuning", default="",
                    help="launch shapes to set instead of the autotuner's choice, e.g. diffuse_depth=2,diffuse_rows=8")
    ap.add_argument("--no-autotune", action="store_true", help="keep the default launch shapes")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--shape", default=None, help="x,y,z (z vertical) override of the workload size")
    args = ap.parse_args()
    rank, world, local = dist_env()
    if args.impl == "reference":
        return run_reference(args, rank, world)

    import torch
    torch.cuda.set_device(local)
    pg = None
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("nccl")
        pg = dist
    from skewtcloudsim_gb300 import Environment, SolverConfig, sounding, build
    build.build()
    if args.workload.startswith("ensemble-"):
        return run_ensemble(args, rank, world, local, pg, torch)

    shape = tuple(int(v) for v in args.shape.split(",")) if args.shape else None
    init, dt, speed = sounding.workload(args.workload, scale=shape)
    cells = init.nx * init.ny * init.nz
    modes = ["plain", "mixed", "plain_textbook"] if args.mode == "both" else [args.mode]
    res = {m: run_mode(args, m, init, dt, speed, cells, world, local, pg, torch) for m in modes}
    head = res[modes[0]]
    prof = head["prof"]

    # ---- roofline of the dominant kernel (live CUDA-event timing of its launches) --------
    dom = max(prof.items(), key=lambda kv: kv[1]["ms"])
    dname, d = dom
    per_launch_ms = d["ms"] / max(d["kernels"], 1)
    peak, peak_kind = measured_peak()
    form = None if head["mode"] == "mixed" else plain_form(prof)
    bpc = PLAIN_FORMS[form][0].get(dname) if form and dname.startswith("pcg_") else STAGE_BYTES.get(dname)
    roofline = None
    if bpc:
        achieved = bpc * cells / (per_launch_ms / 1e3) / 1e9
        tpc = FREE_TRAFFIC_PER_CELL.get(dname) if form == "matrix-free" else None
        roofline = {"bound": "hbm", "achieved": round(achieved, 1), "peak": peak, "unit": "GB/s",
                    "frac": round(achieved / peak, 4), "traffic": int(tpc * cells) if tpc else None, "kernel": dname,
                    "bytes_per_cell": bpc, "launch_us": round(per_launch_ms * 1e3, 2), "peak_source": peak_kind}
        if tpc:
            roofline["traffic_source"] = ("ncu DRAM bytes read + written by one launch at 512x256x256, scaled to this "
                                          "launch's cells (bytes per launch; pcg_update: the mean of its kernels)")
    step_ms_prof = sum(v["ms"] for v in prof.values())
    depth = sweeps_per_pass(head["tuning"], init.nx, init.ground_height)
    bstep = plain_step_bytes(form, head["pcg_iters"], depth) if form else step_bytes(head["mode"], head["pcg_iters"], head["outer"], depth)
    solver = {None: "149 B per inner MG-PCG iteration + 52 B per refinement step", "one launch": "the plain PCG on the chip"}.get(
        form, f"{PLAIN_FORMS[form][1]:.0f} B per plain PCG iteration ({form})" if form else "")
    step_model = {"bytes_per_cell_step": bstep, "achieved_gbs": round(bstep * head["value"] / 1e9, 1),
                  "frac": round(bstep * head["value"] / 1e9 / peak, 4), "peak_source": peak_kind,
                  "model": (f"the library's own bytes: {stage_bytes(depth):.0f} B of stages (diffusion at {depth} sweep(s) per "
                            "pass) + " + solver)}
    if head["mode"] != "mixed":
        sb = scope_step_bytes(head["mode"], head["pcg_iters"], head["outer"])
        step_model["scope_model"] = {
            "bytes_per_cell_step": sb, "frac": round(sb * head["value"] / 1e9 / peak, 4),
            "model": "2558 B of stages + 52 B per matrix-free Jacobi-PCG iteration (the library's own moves 50 B)"}

    # ---- end to end through the C ABI from host buffers (headline mode) -------------------
    e2e = None
    if not args.no_e2e and rank == 0:
        names = ("th", "qv", "qw", "qc", "qr", "qs", "qi", "u", "v", "w", "p")
        host_in = {k: pinned_like(getattr(init, k)) for k in ("theta", "vel", "qv", "ground_T", "ground_p", "p3d",
                                                               "p_column")}
        outs = {k: pinned_like(np.empty(cells, np.float32)) for k in names}
        cfg = mode_config(args, head["mode"])
        env2 = Environment(init.nx, init.ny, init.nz, init.voxel, cfg)
        K = args.steps
        tuned = {k: v for k, v in head["tuning"].items() if k != "source"}
        env2.set_tuning(**tuned)

        def upload():
            env2.init(host_in["theta"][0], host_in["vel"][0], host_in["qv"][0], host_in["ground_T"][0],
                      host_in["ground_p"][0], host_in["p3d"][0], host_in["p_column"][0], init.ground_height)

        # set-up outside the clock: an environment's first step captures its CUDA graph (once per
        # environment, like the allocations of skt_create); the timed region then starts again from
        # the upload of every input
        upload()
        env2.update_gpu(dt, speed)
        env2.sync()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        upload()
        t_up = time.perf_counter()
        host_outs = {k: outs[k][0] for k in names}
        step_ms = []
        for _ in range(K):
            ts = time.perf_counter()
            env2.update_gpu(dt, speed)
            env2.read_async(host_outs)  # this step's fields copy out while the next step runs
            step_ms.append(round((time.perf_counter() - ts) * 1e3, 1))
        tw = time.perf_counter()
        env2.read_wait()
        el = time.perf_counter() - t0
        h2d = sum(a[0].nbytes for a in host_in.values()) + init.ground_height.nbytes
        d2h = len(names) * cells * 4
        e2e = {"value": cells * K / el, "unit": "cell-steps/s", "h2d_bytes_per_step": int(h2d / K),
               "d2h_bytes_per_step": int(d2h), "steps": K,
               "phases_ms": {"upload": round((t_up - t0) * 1e3, 1), "steps": step_ms,
                             "last_readback": round((time.perf_counter() - tw) * 1e3, 1)},
               "note": "init from pinned host arrays once, then after each step the readback of the 11 "
                       "prognostic fields into pinned host arrays (the reference's per-step GPUSetEnv), "
                       "snapshot on the device and copied into the pinned arrays on a second stream during the "
                       "next step (the copy engine in graph mode, a writer kernel otherwise); host wall clock "
                       "from the start of the upload up to the "
                       "last step's copies; the environment's graph was captured by one untimed step before"}
        env2.close()

    cpu = None
    if not args.no_cpu_baseline and rank == 0:
        cpu = cpu_baseline(args.workload, CPU_SAMPLE, CPU_STEPS)
        cpu["thread_sweep"] = cpu_thread_sweep(args.workload, CPU_SAMPLE)
        cpu["host"] = {"nproc": os.cpu_count(), "cpu": host_cpu()}

    field_mb = cells * 4 / 1e6
    out = {"metric": METRIC, "value": head["value"], "unit": "cell-steps/s", "n_gpus": world, "steps": args.steps,
           "warmup": args.warmup, "ms_per_step": head["ms_per_step"], "higher_is_better": True, "scaling": "weak",
           "vs_baseline": None, "dtype": "f32", "data": "synthetic",
           "config": {"workload": args.workload, "grid_xyz": [init.nx, init.nz, init.ny], "cells": cells,
                      "dt": dt, "pcg": head["mode"], "semantics": head["semantics"],
                      "pcg_iters_per_step": head["pcg_iters"], "graph": bool(args.graph), "tuning": head["tuning"],
                      "l2": (f"inputs larger than L2 ({field_mb:.0f} MB per field, L2 129 MB)" if field_mb > 129
                             else f"fields of {field_mb:.0f} MB fit in L2 (129 MB): timings include L2 reuse"),
                      "parallelism": "replicas" if world > 1 else "single"},
           "roofline": roofline, "step_roofline": step_model, "cpu_baseline": cpu, "e2e": e2e,
           "gpu_launches": head["launches"], "clocks": head["clocks"],
           "profile_ms": {k: round(v["ms"], 3) for k, v in prof.items()}, "profile_step_ms": round(step_ms_prof, 3)}
    if head["mode"] == "plain" and head["semantics"] == "reference":
        out["config"]["pcg_note"] = (f"reference semantics: the PCG stops at its {head['pcg_max_iter']}-iteration cap "
                                     f"without converging (converged={head['converged']}, max residual "
                                     f"{head['residual']:.3g} > 1e-5), as the reference's does")
    if "plain_textbook" in res:
        t = res["plain_textbook"]
        tdepth = sweeps_per_pass(t["tuning"], init.nx, init.ground_height)
        tbytes = plain_step_bytes(plain_form(t["prof"]), t["pcg_iters"], tdepth)
        out["plain_textbook"] = {
            "value": t["value"], "ms_per_step": t["ms_per_step"], "semantics": "textbook",
            "pcg_iters_per_step": t["pcg_iters"], "converged": t["converged"], "max_residual": t["residual"],
            "pcg_max_iter": t["pcg_max_iter"], "gpu_launches": t["launches"], "clocks": t["clocks"],
            "note": "the plain Jacobi-PCG on the textbook (symmetric) operator the mixed mode solves, run without the "
                    "iteration cap to the reference's stop test max |r| <= 1e-5",
            "step_roofline": {"bytes_per_cell_step": tbytes, "frac": round(tbytes * t["value"] / 1e9 / peak, 4),
                              "scope_model_frac": round(scope_step_bytes("plain", t["pcg_iters"], 0) * t["value"] / 1e9 / peak, 4)},
            "profile_ms": {k: round(v["ms"], 3) for k, v in t["prof"].items()}}
    if "mixed" in res and head["mode"] != "mixed":
        m = res["mixed"]
        mbytes = step_bytes("mixed", m["pcg_iters"], m["outer"], sweeps_per_pass(m["tuning"], init.nx, init.ground_height))
        out["mixed"] = {"value": m["value"], "ms_per_step": m["ms_per_step"], "speedup_vs_plain": round(m["value"] / head["value"], 3),
                        "semantics": m["semantics"], "inner_iters_per_step": m["pcg_iters"], "refine_steps": m["outer"],
                        "converged": m["converged"], "rel_residual": m["residual"], "gpu_launches": m["launches"],
                        "step_roofline": {"bytes_per_cell_step": mbytes, "frac": round(mbytes * m["value"] / 1e9 / peak, 4)},
                        "clocks": m["clocks"], "profile_ms": {k: round(v["ms"], 3) for k, v in m["prof"].items()}}
        if "plain_textbook" in res:
            out["mixed"]["speedup_vs_plain_textbook"] = round(m["value"] / res["plain_textbook"]["value"], 3)
        out["mixed"]["note"] = ("speedup_vs_plain: against the capped reference-semantics PCG (the drop-in headline, "
                                "not converged); speedup_vs_plain_textbook: against the plain Jacobi-PCG on the same "
                                "textbook operator run to convergence")
    if rank == 0:
        print(json.dumps(out), flush=True)
    if pg:
        pg.destroy_process_group()


if __name__ == "__main__":
    main()
