#!/usr/bin/env python3
"""Scattering-integral benchmark (one JSON line on stdout, rank 0).

Workload: the large single problem -- 48^3 hexes x 6 tetrahedra = 663,552
cells, 1000 spherical-Fibonacci directions (weights 4 pi / 1000), Thomson
phase function, Illum lognormal(0, 1.5) replicated over the 4 faces, source
B uniform(0.1, 1), albedo lambda = 0.9; a source iteration whose every step
is one scattering integral S = W^T Ibar, the source update
S <- (1 - lambda) B + lambda S, the FP64 residual max|S - S_prev| and the
relaxation Ibar <- 0.5 Ibar + 0.5 S.  Synthetic seeded data of those shapes
and distributions (the reference ships no data set).

* value: cell-direction pairs per second over K timed steps with every input
  resident in HBM (inputs are larger than L2: no flush needed);
* e2e: the same metric through the reference's calling sequence at the
  bench's precision: per direction rts_send_illum_async (CudaSendIllumAsync)
  of the FP64 face-layout Illum from pinned host memory, then the pair of
  rts_scattering_async calls (CalculateIntScatteringAsyncMPIStream on
  scattering streams 1 and 2, each with its D2H of S) and the waits; every
  copy inside the timed region (e2e_host_call: the pipelined host-buffer
  entry point rts_scattering_update);
* roofline: the dominant kernel's algorithmic FLOP/s against the measured
  (or fallback) peak, timed with CUDA events on the library's stream;
* cpu_baseline: the CPU restatement of the reference's CalculateIntCPU on a
  bounded sample of the same workload, all host threads.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

METRIC = "Scatter-integral Gcell·dir/s at ≤1e-6 rel err vs FP64 path; serve p50/p99 ms"
UNIT = "Gcell·dir/s"
WORKLOAD = dict(name="config2: 663,552 cells x 1000 Fibonacci directions, Thomson, I~lognormal(0,1.5), "
                     "B~U(0.1,1), lambda=0.9, source iteration with relaxation I<-0.5I+0.5S",
                N=663_552, M=1000, seed=1, mu=0.0, sigma=1.5, lam=0.9)
FALLBACK_PEAKS = {"hbm_gbs": 6800.0, "bf16_tflops": 1900.0, "bf16_tflops_sustained": 1700.0}
FP64_NOMINAL_TFLOPS = 1.25


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--precision", default="fp16x3", choices=["fp64", "bf16x3", "fp16x3", "tf32x3"])
    ap.add_argument("--cells", type=int, default=WORKLOAD["N"])
    ap.add_argument("--dirs", type=int, default=WORKLOAD["M"])
    ap.add_argument("--check", choices=["full", "first", "none"], default="full",
                    help="accuracy check against the FP64 path after the timed steps")
    ap.add_argument("--cpu-seconds", type=float, default=12.0, help="CPU baseline sample budget")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--e2e-steps", type=int, default=None)
    ap.add_argument("--no-serve", action="store_true", help="skip the short serving stream of the default line")
    ap.add_argument("--no-tune", action="store_true",
                    help="skip the schedule autotuner (rts_autotune_schedule) before the timed steps")
    ap.add_argument("--serve-window", type=float, default=2.0, help="arrival window of that stream, seconds")
    ap.add_argument("--flush", type=int, default=0, choices=[0, 1, 2],
                    help="tensor-core K-slices per FP32 drain (0: the library's automatic choice, which is 2 "
                         "for this workload's smooth Thomson kernel)")
    ap.add_argument("--moments", action="store_true",
                    help="time the FP64 moment kernels on the config 2 Illum instead (one JSON line)")
    ap.add_argument("--sweep", action="store_true",
                    help="the transport sweep producing Illum (mesh n^3 x 6 tetrahedra, --dirs directions)")
    ap.add_argument("--sweep-n", type=int, default=48, help="hexahedra per cube edge of the sweep's mesh")
    ap.add_argument("--config", type=int, default=2, choices=[1, 2, 3, 4, 5],
                    help="2: the headline source iteration (default); 1, 3, 4, 5: the other configurations")
    return ap.parse_args()


def run_other_config(args, rank, world, local):
    """Configurations 1, 3, 4, 5 (bench_configs.py): one JSON line each."""
    import torch

    import bench_configs as bc
    import relativistic_solver_hllc_gb300 as pkg
    from relativistic_solver_hllc_gb300 import _native

    pkg.build_library()
    torch.cuda.set_device(local)
    ctx = pkg.Context(local)
    K, W = args.steps, args.warmup
    prec = args.precision if args.precision != "fp64" else "fp16x3"
    clocks = ClockSampler(local)
    clocks.start()
    if args.config == 1:
        res = bc.config1(pkg, _native, ctx, torch, K, W)
        dtype = "f64"
    elif args.config == 3:
        res = bc.config3(pkg, _native, ctx, torch, K, W, prec)
        # the configuration names the TF32x3 and split-BF16 paths: both beside the headline precision
        for other in ("tf32x3", "bf16x3"):
            res[other] = bc.config3(pkg, _native, ctx, torch, K, W, other) if prec != other else None
        dtype = prec
    elif args.config == 4:
        res = bc.config4(pkg, _native, ctx, torch, K, W, prec)
        dtype = prec
    else:
        res = bc.config5(pkg, _native, ctx, torch, precision=prec)
        dtype = prec
    clk = clocks.stop()
    if args.config == 5:
        row80 = next((r for r in res["loads"] if abs(r["load"] - 0.8) < 1e-9), res["loads"][-1])
        line = {"metric": METRIC, "value": row80["throughput_cell_dir_iter_per_s"] / 1e9, "unit": UNIT,
                "n_gpus": world, "steps": K, "warmup": W, "ms_per_step": None, "higher_is_better": True,
                "scaling": "weak", "vs_baseline": None, "dtype": dtype, "data": "synthetic",
                "config": {"workload": "config5: serving stream, Poisson arrivals 10-120% of saturation, "
                                       "HG, M in {110,302,590,1202}, 5-40 iterations, 120 GB cap"},
                "serve": res, "p50_ms_at_80pct": row80["p50_ms"], "p99_ms_at_80pct": row80["p99_ms"], "clocks": clk}
    else:
        line = {"metric": METRIC, "value": res["value"], "unit": UNIT, "n_gpus": world, "steps": K, "warmup": W,
                "ms_per_step": res["ms_per_step"], "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
                "dtype": dtype, "data": "synthetic",
                "config": {"workload": f"config{args.config}: " + res.pop("workload")}, "result": res,
                "clocks": clk}
    if rank == 0:
        print(json.dumps(line), flush=True)
    ctx.close()


def run_moments(args, rank, world, local):
    """The FP64 moment kernels (energy/flux, and the fused pass with the
    impulse tensor and divergences) on the config 2 Illum: one JSON line."""
    import torch

    import bench_configs as bc
    import relativistic_solver_hllc_gb300 as pkg
    from relativistic_solver_hllc_gb300 import _native

    pkg.build_library()
    torch.cuda.set_device(local)
    ctx = pkg.Context(local)
    clocks = ClockSampler(local)
    clocks.start()
    res = bc.moments_pass(pkg, _native, ctx, torch, args.steps, args.warmup, N=args.cells)
    clk = clocks.stop()
    peaks, src = load_peaks()
    hbm = peak_value(peaks, "hbm_gbs") or FALLBACK_PEAKS["hbm_gbs"]
    fp64_peak = ctx.measure_fp64_peak(2.0)  # this GPU's FP64 FMA rate, after the timed passes
    m = res["illum_params"]
    line = {"metric": "FP64 moment pass Gcell·dir/s", "value": args.cells * 1000 / (m["kernel_ms"] / 1e3) / 1e9,
            "unit": "Gcell·dir/s", "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": m["kernel_ms"], "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "f64", "data": "synthetic",
            "config": {"workload": f"config 2 Illum ({args.cells} cells x 1000 directions, FP64 faces): moments and "
                                   "fused divergence pass"},
            "roofline": {"bound": "fp64", "achieved": m["fp64_tflops"], "peak": fp64_peak,
                         "unit": "TFLOP/s", "frac": m["fp64_tflops"] / fp64_peak, "traffic": None,
                         "hbm_gbs": m["hbm_gbs"], "hbm_frac": m["hbm_gbs"] / hbm,
                         "peak_source": f"measured FP64 FMA rate of this GPU (rts_measure_fp64_peak); HBM {src}",
                         "nominal_fp64_tflops": FP64_NOMINAL_TFLOPS},
            "result": res, "clocks": clk}
    if rank == 0:
        print(json.dumps(line), flush=True)
    ctx.close()


def sweep_medium(N: int, seed: int = 11):
    """Per-cell GetCurIllum coefficients of the sweep workload (scattering
    form): alpha ~ U(0.5, 2), beta ~ U(0, 1), Q ~ U(0, 1), seeded."""
    rng = np.random.default_rng(seed)
    return rng.uniform(0.5, 2.0, N), rng.uniform(0.0, 1.0, N), rng.uniform(0.0, 1.0, N)


def read_sweep_profile():
    """FP64 operations and DRAM bytes per cell-direction of sweep_kernel in the
    form that the timed steps run (663,552 cells x 1000 directions: evaluating)
    from the committed ncu summary."""
    p = ROOT / "profiles" / "sweep_kernel_24576x1000.json"
    try:
        return json.loads(p.read_text())
    except Exception:
        return {}


def run_sweep(args, rank, world, local):
    """The transport sweep that produces Illum (one CTA per direction over
    the dependency steps of the mesh): one JSON line.  Mesh: the unit cube,
    n^3 hexahedra x 6 tetrahedra, turned by the fixed tilt (no face parallel
    to a Fibonacci direction), boundary rule 1 (x = 0 side a source); --dirs
    Fibonacci directions; seeded per-cell coefficients; the source term is the
    FP64 scattering integral of the lognormal(0, 1.5) Illum."""
    import torch

    import relativistic_solver_hllc_gb300 as pkg
    from relativistic_solver_hllc_gb300 import _native

    pkg.build_library()
    torch.cuda.set_device(local)
    n, M, K, W = args.sweep_n, args.dirs, args.steps, args.warmup
    vert, pairs, normals = pkg.mesh_cube(n, 1, True)
    N = vert.shape[0]
    xyz, area, fa = _native.synth_directions(M)
    ctx = pkg.Context(local)
    ctx.init(xyz, area, fa, N)
    t0 = time.perf_counter()
    ctx.sweep_set_mesh(vert, pairs, normals)
    records, steps_max = ctx.sweep_build()
    t_build = time.perf_counter() - t0
    a, b, q = sweep_medium(N)
    ctx.sweep_set_medium(pkg.medium(), a, b, q)
    ctx.synth_illum(WORKLOAD["seed"], WORKLOAD["mu"], WORKLOAD["sigma"])
    ctx.scattering_async(0, M, pkg.STREAM_SCATTERING_1)
    ctx.sync_stream(pkg.STREAM_SCATTERING_1)
    for _ in range(W):
        ctx.sweep(read_norm=False)
    torch.cuda.synchronize()
    clocks = ClockSampler(local)
    clocks.start()
    launches0 = ctx.launch_count()
    ctx.kernel_timing(True)
    t0 = time.perf_counter()
    for _ in range(K):
        ctx.sweep(read_norm=False)
    norm = ctx.sweep()  # one more, read back: the timed region ends synchronised
    elapsed = time.perf_counter() - t0
    kern_ms, kern_n = ctx.kernel_timing(False)
    launches = ctx.launch_count() - launches0
    clk = clocks.stop()
    kern_avg = kern_ms / max(kern_n, 1)
    value = N * M / (kern_avg / 1e3) / 1e9

    # the other two forms of the kernel, timed alone: the sweep that stores
    # the attenuation factors (the first after a change of medium) and sweeps
    # that evaluate them every time (the cache switched off)
    def timed_sweeps(n_sweeps):
        ctx.kernel_timing(True)
        for _ in range(n_sweeps):
            ctx.sweep(read_norm=False)
        ctx.sweep()
        ms, cnt = ctx.kernel_timing(False)
        return ms / max(cnt, 1)

    ctx.sweep_set_medium(pkg.medium(), a, b, q)
    store_ms = timed_sweeps(0)
    ctx.set_tuning(_native.TUNE_SWEEP_CACHE, 0)
    eval_ms = timed_sweeps(2)
    ctx.set_tuning(_native.TUNE_SWEEP_CACHE, 1)
    forms = {"read_ms": kern_avg, "store_ms": store_ms, "evaluate_ms": eval_ms,
             "note": "read: the timed steps (attenuation factors exp(-k s) stored by the first sweep of the medium, "
                     "read since); store: the first sweep after a change of medium; evaluate: "
                     "RTS_TUNE_SWEEP_CACHE 0 (the exponential in every sweep, as the reference). With more than five "
                     "directions per SM and over 2^19 cells nothing is stored and all three evaluate"}

    # parity spot check on two full-size directions against the oracle
    accuracy = None
    if rank == 0 and args.check != "none":
        import oracle

        oracle.build()
        before = np.empty(M * N * 4)
        ctx.read_illum(before)
        S = np.empty(M * N)
        ctx.read_scattering(0, M, pkg.STREAM_SCATTERING_1, S)
        ctx.sync_stream(pkg.STREAM_SCATTERING_1)
        S = S.reshape(M, N)
        ctx.sweep()
        after = np.empty(M * N * 4)
        ctx.read_illum(after)
        worst = 0.0
        for d in (0, M // 2):
            st = oracle.SweepStructures(vert, pairs, normals, xyz[d:d + 1])
            il = before.reshape(M, N, 4)[d:d + 1].copy()
            oracle.sweep(st, S[d:d + 1], a, b, q, il)
            got = after.reshape(M, N, 4)[d:d + 1]
            den = np.maximum(np.abs(il), 1e-300)
            worst = max(worst, float(np.max(np.abs(got - il) / den)))
        accuracy = {"vs": "oracle sweep (restated reference, FP64)", "directions": [0, M // 2],
                    "max_rel_err": worst, "tolerance": 1e-11}

    # end to end: the device source iteration (sweep + FP16x3 scattering per
    # iteration, the norm read back each time) through rts_illum_solve
    Ke = args.e2e_steps if args.e2e_steps is not None else max(3, K // 4)
    ctx.illum_solve("fp16x3", max_iter=1 + 1, accuracy=0.0)  # warm-up of the split operands
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    ctx.sweep_set_medium(pkg.medium(), a, b, q)  # a new medium: the first sweep stores the factors again
    norms = ctx.illum_solve("fp16x3", max_iter=Ke, accuracy=0.0)
    e2e_s = time.perf_counter() - t0
    e2e = {"value": N * M * len(norms) / e2e_s / 1e9, "unit": UNIT, "h2d_bytes_per_step": 0,
           "d2h_bytes_per_step": 8, "steps": len(norms),
           "call": "rts_sweep_set_medium, then rts_illum_solve (sweep + FP16x3 scattering per iteration, "
                   "device-resident Illum and S, the 8-byte norm read back each iteration; the first sweep "
                   "stores the attenuation factors, the others read them)"}

    prof = read_sweep_profile()
    fl = prof.get("fp64_flops_per_cell_dir")
    achieved = fl * value * 1e9 / 1e12 if fl else None
    fp64_peak = ctx.measure_fp64_peak(2.0)  # this GPU's FP64 FMA rate, after the timed sweeps
    roof = {"bound": "fp64", "achieved": achieved, "peak": fp64_peak, "unit": "TFLOP/s",
            "frac": achieved / fp64_peak if achieved else None,
            "traffic": prof.get("dram_bytes_per_cell_dir") and prof["dram_bytes_per_cell_dir"] * N * M,
            "peak_source": "measured FP64 FMA rate of this GPU (rts_measure_fp64_peak)",
            "nominal_fp64_tflops": FP64_NOMINAL_TFLOPS,
            "fp64_pipe_active": prof.get("fp64_pipe_active_frac"),
            "note": "achieved = FP64 operations per cell-direction of the evaluating form counted by ncu "
                    "(dadd + dmul + 2 dfma) x the measured cell-direction rate; the pipe also issues the compares, "
                    "so fp64_pipe_active (ncu, 24,576 x 1000) is the binding figure",
            "hbm": {"algorithmic_bytes_per_cell_dir": prof.get("algorithmic_bytes_per_cell_dir"),
                    "achieved_gbs": prof.get("algorithmic_bytes_per_cell_dir") and
                    prof["algorithmic_bytes_per_cell_dir"] * value, "peak_gbs": peak_value(load_peaks()[0], "hbm_gbs") or FALLBACK_PEAKS["hbm_gbs"]},
            "kernel_ms_avg": kern_avg, "kernel_launches_timed": kern_n}

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        import oracle

        oracle.build()
        nthr = oracle.max_threads()
        Ds = max(1, nthr)
        st = oracle.SweepStructures(vert, pairs, normals, xyz[:Ds])
        S = np.empty(M * N)
        ctx.read_scattering(0, Ds, pkg.STREAM_SCATTERING_1, S)
        ctx.sync_stream(pkg.STREAM_SCATTERING_1)
        S = S[:Ds * N].reshape(Ds, N)
        il = np.random.default_rng(5).uniform(0.1, 1.0, (Ds, N, 4))
        t0 = time.perf_counter()
        oracle.sweep(st, S, a, b, q, il, nthreads=nthr)
        dt = time.perf_counter() - t0
        cpu = {"value": N * Ds / dt / 1e9, "unit": UNIT, "cores": nthr, "kind": "port",
               "sample": f"the oracle sweep (restated Illum_async.cpp:726-784, GetCurIllum, ReCalcIllum; "
                         f"bit-identical to the reference's own code on the golden cases) over directions "
                         f"[0,{Ds}) of the full {N}-cell mesh, one direction per thread"}

    line = {
        "metric": "Transport sweep Gcell·dir/s (FP64, all directions of the mesh)", "value": value, "unit": UNIT,
        "n_gpus": world, "steps": K, "warmup": W, "ms_per_step": kern_avg, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": {"workload": f"transport sweep: unit cube {n}^3 x 6 = {N} tetrahedra (tilted), {M} Fibonacci "
                               f"directions, alpha~U(0.5,2) beta~U(0,1) Q~U(0,1), boundary x=0 source",
                   "cells": N, "dirs": M, "node_records": records, "max_steps": steps_max,
                   "structures_build_s": t_build, "parallelism": "replicas" if world > 1 else "single",
                   "l2": "inputs larger than L2 (no flush)",
                   "step": "one sweep of every direction within a source iteration, medium unchanged since the "
                           "first (sweep_forms)"},
        "roofline": roof, "cpu_baseline": cpu, "e2e": e2e, "gpu_launches": launches, "clocks": clk,
        "accuracy": accuracy, "norm": norm, "wall_ms_per_step": elapsed / (K + 1) * 1e3, "sweep_forms": forms,
    }
    if rank == 0:
        print(json.dumps(line), flush=True)
    ctx.close()


def max_over_ranks(x: float, dist, device: str = "cuda") -> float:
    """The largest value over all ranks (the slowest rank's time); x itself on
    one process."""
    if not dist:
        return x
    import torch

    t = torch.tensor([x], device=device, dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def replicas_value(cells: int, dirs: int, steps: int, world: int, seconds: float) -> float:
    """Whole-job Gcell·dir/s of `world` replicas of the workload, each running
    `steps` steps, over the slowest rank's time."""
    return cells * dirs * steps * world / seconds / 1e9


def dist_env():
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return rank, world, local


def load_peaks():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        try:
            d = json.loads(p.read_text())
            return d, "measured"
        except Exception:
            pass
    return dict(FALLBACK_PEAKS), "fallback"


def peak_value(peaks, *keys):
    for k in keys:
        v = peaks.get(k)
        if isinstance(v, (int, float)):
            return float(v)
        if isinstance(v, dict):
            for kk in ("value", "median", "max"):
                if isinstance(v.get(kk), (int, float)):
                    return float(v[kk])
    return None


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled while the GPU works."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device: int):
        self.device = device
        self.proc = None

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.device}", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-lms", "50"], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except Exception:
            self.proc = None

    def stop(self):
        if not self.proc:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"], "samples": 0}
        time.sleep(0.12)
        self.proc.terminate()
        try:
            out, _ = self.proc.communicate(timeout=5)
        except Exception:
            self.proc.kill()
            out, _ = self.proc.communicate()
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in out.splitlines():
            f = [x.strip() for x in line.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                smax.append(float(f[2]))
            except ValueError:
                continue
            for n, v in zip(names, f[5:9]):
                if v.lower() == "active":
                    reasons.add(n)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(smax) if smax else None,
                "reasons": sorted(reasons), "samples": len(sm)}


def read_traffic():
    """Per-launch DRAM bytes of the dominant kernel from the committed ncu summary."""
    p = ROOT / "profiles" / "traffic.json"
    if not p.exists():
        return {}
    try:
        return json.loads(p.read_text())
    except Exception:
        return {}


# ---------------------------------------------------------------- CPU legs
def cpu_sample(N: int, M: int, seconds: float, seed: int, sigma: float):
    """Time the restated CalculateIntCPU on a bounded sample: cells [0, Ns)
    of the full-size [M][N][4] Illum (real strides), every in-direction,
    out-directions [0, s) with s sized to about `seconds` of work."""
    import oracle

    nthreads = oracle.max_threads()
    Ns = min(N, 4096)
    il = np.empty(M * N * 4)  # untouched pages stay unmapped; only the sample is written
    oracle.illum_cells_into(il, seed, 0.0, sigma, N, M, 0, Ns)
    xyz, area, fa = oracle.fibonacci_directions(M)
    cells = np.arange(Ns, dtype=np.int64)
    s0 = max(1, nthreads)
    t0 = time.perf_counter()
    oracle.calculate_int_cells(N, xyz, area, fa, il, cells, 0, s0, nthreads)
    t_cal = time.perf_counter() - t0
    per = t_cal / (Ns * s0)
    s = int(max(s0, min(M, seconds / max(per * Ns, 1e-12))))
    s = max(nthreads, (s // nthreads) * nthreads) if s >= nthreads else s
    s = min(s, M)
    return dict(il=il, xyz=xyz, area=area, fa=fa, cells=cells, Ns=Ns, s=s, nthreads=nthreads, N=N, M=M)


def cpu_run(sample) -> float:
    import oracle

    t0 = time.perf_counter()
    oracle.calculate_int_cells(sample["N"], sample["xyz"], sample["area"], sample["fa"], sample["il"],
                               sample["cells"], 0, sample["s"], sample["nthreads"])
    dt = time.perf_counter() - t0
    return sample["Ns"] * sample["s"] / dt / 1e9


def run_reference(args, rank):
    """Reference arm: the reference's CPU scattering integral (restated; the
    reference's own source cannot be compiled on the GPU hosts) on the host
    cores, each step a bounded sample of the same workload."""
    if rank != 0:
        return
    import oracle

    oracle.build()
    N, M = args.cells, args.dirs
    sample = cpu_sample(N, M, 2.0, WORKLOAD["seed"], WORKLOAD["sigma"])
    for _ in range(args.warmup):
        cpu_run(sample)
    vals, t0 = [], time.perf_counter()
    for _ in range(args.steps):
        vals.append(cpu_run(sample))
    wall = time.perf_counter() - t0
    value = statistics.mean(vals)
    kind = "port"  # the C restatement is timed; the reference's own source is not built on GPU hosts
    desc = (f"cells [0,{sample['Ns']}) of the {N}-cell Illum (full strides), all {M} in-directions, "
            f"out-directions [0,{sample['s']}) per step")
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "impl": "reference", "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": wall / args.steps * 1e3,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
        "data": "synthetic", "config": {"workload": WORKLOAD["name"], "sample": desc},
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": sample["nthreads"], "kind": kind, "sample": desc},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


# ---------------------------------------------------------------- GPU arm
def run_ours(args, rank, world, local):
    import torch

    import relativistic_solver_hllc_gb300 as pkg
    from relativistic_solver_hllc_gb300 import _native

    pkg.build_library()
    pkg.load_library()
    dist = None
    if world > 1:
        import torch.distributed as dist

        dist.init_process_group("nccl" if torch.cuda.is_available() else "gloo")
    torch.cuda.set_device(local)

    N, M, lam = args.cells, args.dirs, WORKLOAD["lam"]
    prec = args.precision
    K, W = args.steps, args.warmup
    xyz, area, fa = _native.synth_directions(M)
    B = _native.synth_uniform(WORKLOAD["seed"], 2, 0.1, 1.0, N)
    ctx = pkg.Context(local)
    ctx.init(xyz, area, fa, N)
    if args.flush:
        ctx.set_tuning(_native.TUNE_FLUSH, args.flush)
    # the library's schedule autotuner on this workload (not timed): drain
    # period, tile width and order for M directions at this cell count
    schedule = None
    if prec != "fp64" and not args.no_tune:
        best, tried = ctx.autotune_schedule(M, prec, cells=N)
        schedule = {"chosen": {k: best[k] for k in ("flush", "bn", "order", "ms")}, "schedules_timed": len(tried)}
    flush_used = ctx.flush_period(prec) if prec != "fp64" else None

    def fresh(precision):
        ctx.synth_illum(WORKLOAD["seed"], WORKLOAD["mu"], WORKLOAD["sigma"])
        ctx.solve_setup(precision, B, lam)

    # warm-up steps, then restart the iteration so the timed steps are steps 1..K
    fresh(prec)
    for _ in range(W):
        ctx.solve_step_async(True)
    ctx.wait()
    fresh(prec)
    ctx.wait()

    stream = torch.cuda.ExternalStream(ctx.stream_handle(pkg.STREAM_SCATTERING_1))
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    clocks = ClockSampler(local)
    torch.cuda.synchronize()
    if dist:
        dist.barrier()
    clocks.start()
    time.sleep(0.25)  # let the sampler attach before the timed region
    launches0 = ctx.launch_count()
    ctx.kernel_timing(True)
    ev0.record(stream)
    for _ in range(K):
        ctx.solve_step_async(True)
    ev1.record(stream)
    torch.cuda.synchronize()
    kern_ms, kern_n = ctx.kernel_timing(False)
    launches = ctx.launch_count() - launches0
    clk = clocks.stop()
    elapsed = ev0.elapsed_time(ev1) / 1e3
    elapsed = max_over_ranks(elapsed, dist)
    residuals = ctx.solve_residual_history(K).tolist()
    value = replicas_value(N, M, K, world, elapsed)

    # end to end through the call the reference's solver makes: per step, the
    # per-direction CudaSendIllumAsync copies of the FP64 face-layout Illum
    # from pinned host memory, then the pair of
    # CalculateIntScatteringAsyncMPIStream calls of the source iteration
    # (solve_module/illum/Illum_async.cpp:1019-1020: [0, M/3) on scattering
    # stream 1, [0, M) on scattering stream 2) at the bench's precision, each
    # with its D2H of S into the pinned host scattering array, and the wait
    # for both streams.  Measured before any multi-GB pageable host array is
    # allocated (the accuracy check's read-backs): on the GPU hosts the host
    # copies that follow such allocations ran at half speed.
    Ke = args.e2e_steps if args.e2e_steps is not None else K
    illum_host = ctx.host_illum()
    ctx.synth_illum(WORKLOAD["seed"], WORKLOAD["mu"], WORKLOAD["sigma"])
    ctx.read_illum(illum_host)
    S_host = ctx.host_scattering()
    ctx.set_precision(prec)
    size_1 = M // 3

    def reference_sequence():
        for j in range(M):
            ctx.send_illum_async(4 * N, 4 * N * j, 4 * N * j, illum_host)
        ctx.scattering_async(0, size_1, pkg.STREAM_SCATTERING_1, S_host)
        ctx.scattering_async(0, M, pkg.STREAM_SCATTERING_2, S_host)
        ctx.sync_stream(pkg.STREAM_SCATTERING_1)
        ctx.sync_stream(pkg.STREAM_SCATTERING_2)
        ctx._keep.clear()

    reference_sequence()  # warm-up: builds the stream slots' operands
    torch.cuda.synchronize()
    if dist:
        dist.barrier()
    t0 = time.perf_counter()
    per_step = []
    for _ in range(Ke):
        ts = time.perf_counter()
        reference_sequence()
        per_step.append(time.perf_counter() - ts)
    e2e_s = time.perf_counter() - t0
    e2e_s = max_over_ranks(e2e_s, dist)
    ctx.set_precision("fp64")
    e2e = {"value": N * M * Ke * world / e2e_s / 1e9, "unit": UNIT,
           "h2d_bytes_per_step": M * N * 4 * 8, "d2h_bytes_per_step": (size_1 + M) * N * 8,
           "steps": Ke, "ms_per_step": e2e_s / Ke * 1e3,
           "ms_per_step_median": statistics.median(per_step) * 1e3, "ms_per_step_min": min(per_step) * 1e3,
           "call": f"the reference's calling sequence at {prec}: {M} x rts_send_illum_async (CudaSendIllumAsync, "
                   f"pinned host Illum), rts_scattering_async [0,{size_1}) on stream 1 and [0,{M}) on stream 2 "
                   "(CalculateIntScatteringAsyncMPIStream x 2, D2H of S into the pinned host array), "
                   "rts_sync_stream x 2; cell-directions counted once per step"}

    # the same integral through the pipelined host-buffer entry point
    # (rts_scattering_update: H2D of the FP64 Illum and B, integral + update,
    # D2H of the FP64 S, over 16 cell ranges in flight)
    B_pin = _native.PinnedBuffer(N * 8)  # every input of the call from pinned host memory
    B_host = B_pin.array(np.float64, N)
    B_host[:] = B
    ctx.scattering_update(prec, illum_host, B_host, lam, S_host)  # warm-up
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    per_call = []
    for _ in range(Ke):
        ts = time.perf_counter()
        ctx.scattering_update(prec, illum_host, B_host, lam, S_host)
        per_call.append(time.perf_counter() - ts)
    e2e2_s = max_over_ranks(time.perf_counter() - t0, dist)
    h2d, d2h = M * N * 4 * 8 + N * 8, M * N * 8
    e2e_host_call = {"value": N * M * Ke * world / e2e2_s / 1e9, "unit": UNIT, "h2d_bytes_per_step": h2d,
                     "d2h_bytes_per_step": d2h, "steps": Ke, "ms_per_step": e2e2_s / Ke * 1e3,
                     "ms_per_step_median": statistics.median(per_call) * 1e3,
                     "ms_per_step_min": min(per_call) * 1e3,
                     "link_gbs": (h2d + d2h) / (e2e2_s / Ke) / 1e9,
                     "call": "rts_scattering_update (pinned host buffers, 16 cell ranges pipelined)"}

    # accuracy against the FP64 path on identical inputs: the timed steps again
    # (the iteration is bit-reproducible; run after the e2e legs, whose host
    # copies slow down after large pageable host allocations), and the same
    # steps on the FP64 path, timed too (CUDA events on the kernel and around
    # the steps): the plain FP64 GPU kernel's rate on the same workload
    accuracy = None
    fp64_gpu = None
    if prec != "fp64" and args.check != "none":
        n_chk = K if args.check == "full" else 1
        fresh(prec)
        for _ in range(n_chk):
            ctx.solve_step_async(True)
        S_t = ctx.solve_read()
        fresh("fp64")
        ctx.wait()
        ctx.kernel_timing(True)
        ev0.record(stream)
        for _ in range(n_chk):
            ctx.solve_step_async(True)
        ev1.record(stream)
        torch.cuda.synchronize()
        k64_ms, k64_n = ctx.kernel_timing(False)
        step64_s = ev0.elapsed_time(ev1) / 1e3 / n_chk
        fp64_step = N * M / step64_s / 1e9
        fp64_gpu = {"value": fp64_step, "unit": UNIT, "ms_per_step": step64_s * 1e3,
                    "kernel_ms_avg": k64_ms / max(k64_n, 1), "kernel_launches_timed": k64_n,
                    "kernel_ms_per_step": k64_ms / n_chk,
                    "kernel_tflops": 2.0 * N * M * M * n_chk / (k64_ms / 1e3) / 1e12 if k64_n else None,
                    "steps": n_chk, "speedup_of_tensor_path": value / fp64_step,
                    "note": "the FP64 path (sliced_kernel: exact FP16 digit products on the tensor cores, integer "
                            "totals) running the same relaxed source iteration on the same inputs"}
        S_64 = ctx.solve_read()
        r64 = ctx.solve_residual_history(n_chk).tolist()
        rel = np.abs(S_t - S_64) / np.abs(S_64)
        accuracy = {"vs": "FP64 path", "steps_compared": n_chk, "max_rel_err": float(rel.max()),
                    "mean_rel_err": float(rel.mean()), "fp64_residuals": r64}
        del S_t, S_64, rel
        # single-evaluation error on identical inputs
        fresh(prec)
        ctx.solve_step(False)
        S_t = ctx.solve_read()
        fresh("fp64")
        ctx.solve_step(False)
        S_64 = ctx.solve_read()
        rel = np.abs(S_t - S_64) / np.abs(S_64)
        accuracy["eval_max_rel_err"] = float(rel.max())
        accuracy["eval_mean_rel_err"] = float(rel.mean())
        del S_t, S_64, rel

    # the serving loop (configuration 5's request distribution) on a short
    # stream: saturated throughput, the isolated latencies of the 0.8-load
    # stream's requests and that stream's p50 / p99
    serve = None
    if rank == 0 and world == 1 and not args.no_serve:
        import bench_configs as bc

        sres = bc.config5(pkg, _native, ctx, torch, loads=(0.8,), window_s=args.serve_window, precision=prec)
        row = sres["loads"][0]
        serve = {"saturation_cell_dir_iter_per_s": sres["saturation_cell_dir_iter_per_s"],
                 "load": row["offered_load"], "requests": row["requests"], "completed": row["completed"],
                 "p50_ms": row["p50_ms"], "p99_ms": row["p99_ms"],
                 "isolated_p50_ms": row.get("isolated_p50_ms"), "isolated_p99_ms": row.get("isolated_p99_ms"),
                 "p99_over_isolated_p99": row.get("p99_vs_isolated_p99"),
                 "fifo_alone_p99_ms": row.get("fifo_alone_p99_ms"),
                 "fifo_alone_p99_over_isolated_p99": row.get("fifo_alone_p99_vs_isolated_p99"),
                 "ps_alone_p99_over_isolated_p99": row.get("ps_alone_p99_vs_isolated_p99"),
                 "srpt_alone_p99_over_isolated_p99": row.get("srpt_alone_p99_vs_isolated_p99"),
                 "mean_queue_ms": row.get("mean_queue_ms"), "p99_queue_ms": row.get("p99_queue_ms"),
                 "throughput_cell_dir_iter_per_s": row["throughput_cell_dir_iter_per_s"],
                 "policy": sres["policy"], "window_s": args.serve_window,
                 "workload": "configuration 5's requests (cells lognormal median 50,000 clipped to [2k, 500k], "
                             "M in {110, 302, 590, 1202}, HG g~U(0, 0.8), 5-40 iterations, FP32 lognormal(0,1)), "
                             "Poisson arrivals rescaled to 0.8 of the saturated throughput, 120 GB HBM cap; "
                             "latency counts from arrival (queueing included)"}

    # measured ceilings of this machine for the FP64 kernel and the host link
    # (FMA chains on every SM; 1 GiB pinned copies each way and both at once)
    measured = {"fp64_tflops": ctx.measure_fp64_peak(2.0), "link": ctx.measure_link(1 << 30, 5)}
    lk = measured["link"]
    for leg, overlap in ((e2e, False), (e2e_host_call, True)):
        moved = leg["h2d_bytes_per_step"] + leg["d2h_bytes_per_step"]
        leg["link_gbs"] = moved / (leg["ms_per_step"] / 1e3) / 1e9
        t_in = leg["h2d_bytes_per_step"] / (lk["h2d_gbs"] * 1e9)
        t_out = leg["d2h_bytes_per_step"] / (lk["d2h_gbs"] * 1e9)
        if overlap:
            # the pipelined call: H2D of later cell ranges beside D2H of earlier ones
            floor_s = max(t_in, t_out, moved / (lk["bidirectional_gbs"] * 1e9))
            leg["link_floor"] = "H2D and D2H overlapped, at the measured rates"
        else:
            # the reference's sequence: every integral needs the whole Illum,
            # and the D2H of S follows the integrals
            floor_s = t_in + t_out
            leg["link_floor"] = "H2D then D2H, at the measured rates"
        leg["link_floor_ms"] = floor_s * 1e3
        leg["link_frac"] = floor_s / (leg["ms_per_step"] / 1e3)
    if fp64_gpu and fp64_gpu.get("kernel_tflops"):
        fp64_gpu["fp64_peak_tflops"] = measured["fp64_tflops"]
        fp64_gpu["vs_fp64_peak"] = fp64_gpu["kernel_tflops"] / measured["fp64_tflops"]

    # roofline of the dominant kernel
    peaks, src = load_peaks()
    flops = 2.0 * N * M * M
    # FP64 steps run in several launches over cell ranges
    kern_avg = (kern_ms / K if prec == "fp64" else kern_ms / max(kern_n, 1)) / 1e3
    achieved = flops / kern_avg / 1e12 if kern_n else None
    traffic = read_traffic().get(f"{prec}:{N}x{M}")
    if prec == "fp64":
        # sums of six 9-bit digits: 21 tensor products of FP16 digits per FP64 product
        pk = peak_value(peaks, "bf16_tflops") or FALLBACK_PEAKS["bf16_tflops"]
        roof = {"bound": "tensor", "achieved": achieved, "peak": pk / 21, "unit": "TFLOP/s",
                "frac": 21 * achieved / pk if achieved else None, "traffic": traffic,
                "peak_source": f"bf16 dense burst / 21 digit products, {src}",
                "measured_fp64_tflops": measured["fp64_tflops"], "nominal_fp64_tflops": FP64_NOMINAL_TFLOPS}
    else:
        pk = peak_value(peaks, "bf16_tflops") or FALLBACK_PEAKS["bf16_tflops"]
        roof = {"bound": "tensor", "achieved": achieved, "peak": pk, "unit": "TFLOP/s",
                "frac": achieved / pk if achieved else None, "traffic": traffic,
                "peak_source": f"bf16 dense burst, {src}",
                "tensor_pipe_frac": 3 * achieved / pk if achieved else None,
                "note": "achieved counts algorithmic 2*N*M^2 flops; the split runs 3 tensor products"}
    roof["kernel_ms_avg"] = kern_avg * 1e3
    roof["kernel_launches_timed"] = kern_n

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        import oracle

        oracle.build()
        sample = cpu_sample(N, M, args.cpu_seconds, WORKLOAD["seed"], WORKLOAD["sigma"])
        v = cpu_run(sample)
        cpu = {"value": v, "unit": UNIT, "cores": sample["nthreads"],
               "kind": "port",
               "sample": f"cells [0,{sample['Ns']}) of the {N}-cell Illum (full strides), all {M} in-directions, "
                         f"out-directions [0,{sample['s']})"}

    dtype = {"fp64": "f64", "bf16x3": "bf16x3", "fp16x3": "fp16x3", "tf32x3": "tf32x3"}[prec]
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": K, "warmup": W,
        "ms_per_step": elapsed / K * 1e3, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": dtype, "data": "synthetic",
        "config": {"workload": WORKLOAD["name"], "cells": N, "dirs": M, "precision": prec,
                   "flush": flush_used, "schedule": schedule,
                   "truncation_correction": "relaxed steps: each cell's integrals scaled by the previous step's "
                                            "ratio sum_j v_j I_j / sum_k S_k (v = W 1, FP64; conserved), no "
                                            "constant factor; single evaluations uncorrected",
                   "accuracy_gate": "max rel err vs FP64 path <= 1e-6 after the timed steps (see accuracy)",
                   "parallelism": "replicas" if world > 1 else "single",
                   "l2": "inputs larger than L2 (no flush)", "step": "integral + update + residual + relaxation"},
        "roofline": roof, "cpu_baseline": cpu, "e2e": e2e, "e2e_host_call": e2e_host_call,
        "gpu_launches": launches, "clocks": clk, "accuracy": accuracy, "fp64_gpu": fp64_gpu, "serve": serve,
        "measured_peaks": measured, "residuals": residuals,
    }
    if rank == 0:
        print(json.dumps(line), flush=True)
    ctx.close()
    if dist:
        dist.destroy_process_group()


def main():
    args = parse()
    rank, world, local = dist_env()
    if args.impl == "reference":
        run_reference(args, rank)
    elif args.moments:
        run_moments(args, rank, world, local)
    elif args.sweep:
        run_sweep(args, rank, world, local)
    elif args.config != 2:
        run_other_config(args, rank, world, local)
    else:
        run_ours(args, rank, world, local)


if __name__ == "__main__":
    main()
