"""Benchmark of the atmosphere lookup-table build (one GPU per process).

A step is one complete production LUT build (transmittance 255x255, surface
radiance 16x64, ray scatter and Mie strength 32x255x32x8, 5 scattering
iterations, 128 ray steps, sphere steps 32, FP32 with FP64 geometry).  The
build has no input data: its inputs are the physical parameters of the
configuration, so `data` is "synthetic".  `value` is ray-scatter table cells
built per second over the whole job; `e2e` is the same through the public C
ABI with host output buffers (pinned) and the device-to-host copy of all four
tables inside the timed region.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

With N > 1 (torchrun) every rank builds its own LUT: the path has no exchange
step, so this is N replicas ("scaling": "weak").  `--impl reference` times
complete builds of the FP64 CPU restatement of the reference's algorithm
(oracle/) on the host cores, with the workload's steps, iterations and
physics at a 16x15x4x4 ray-scatter table, and reports their cells per
second.
"""
from __future__ import annotations

import argparse
import ctypes
import json
import os
import statistics
import subprocess
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "LUT build s & ray-scatter queries/s: plain vs surrogate at stated rel err"
UNIT = "ray-scatter cells/s (full multi-order LUT build)"
# DRAM bytes read + written per k_point_scatter launch of the production
# build, mean over its five launches in one ncu capture of this workload
# (dram__bytes_read.sum + dram__bytes_write.sum); ncu does not run here, so the
# figure is a recorded capture, not a measurement of this run
PS_DRAM_BYTES_PER_LAUNCH = 38_900_000
# shared-memory wavefronts (128 B each) of the five launches, from the same capture
# (l1tex__data_pipe_lsu_wavefronts_mem_shared.sum)
PS_SMEM_WAVEFRONTS = 546_600_000
TABLES = ("transmittance", "surface_radiance", "ray_scatter", "mie_strength")
SUN_FIT_NODES = 8192 * 8 * 6  # sun rays integrated for the fits: heights x segments x Chebyshev nodes
WORKLOAD = ("production LUT build: T 255x255, E 16x64, S/M 32x255x32x8 RGB, 5 iterations, "
            "128 ray steps, sphere steps 32 (336 directions), R 6378 km, H 100 km")


def parse():
    p = argparse.ArgumentParser()
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=10)
    p.add_argument("--warmup", type=int, default=3)
    p.add_argument("--impl", default="ours", choices=["ours", "reference"])
    p.add_argument("--cpu-sample-s", type=float, default=15.0, help="seconds of CPU baseline sampling")
    p.add_argument("--profile", default=None,
                   help="only run --builds builds of a named configuration (small_fp64, production, "
                        "reference_production, shader_test), for profilers")
    p.add_argument("--builds", type=int, default=2)
    p.add_argument("--profile-surrogate", type=int, default=0, metavar="N",
                   help="only train the surrogate 4 steps on the production tables and run --builds batches of "
                        "N surrogate queries, for profilers")
    p.add_argument("--no-extras", dest="extras", action="store_false",
                   help="skip the parameter-sweep and query/surrogate measurements")
    return p.parse_args()


def dist_env():
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return rank, world, local


# ---------------------------------------------------------------------------
# clocks sampled during the timed region
# ---------------------------------------------------------------------------

class ClockSampler:
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device_index: int):
        self.device = device_index
        self.proc = None
        self.lines = []

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.device}", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-lms", "100"], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.thread = threading.Thread(target=self._read, daemon=True)
            self.thread.start()
        except (OSError, FileNotFoundError):
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self):
        if not self.proc:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        time.sleep(0.25)
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        sm, mx, reasons, power = [], [], set(), []
        names = ("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap")
        for line in self.lines:
            f = [x.strip() for x in line.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx.append(float(f[2]))
                power.append(float(f[3]))
            except ValueError:
                continue
            for n, v in zip(names, f[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(n)
        loaded = [s for s in sm if mx and s > 0.5 * max(mx)] or sm
        return {"sm_mhz": statistics.median(loaded) if loaded else None,
                "sm_max_mhz": max(mx) if mx else None,
                "power_w_max": max(power) if power else None,
                "samples": len(sm), "reasons": sorted(reasons)}


# ---------------------------------------------------------------------------
# our GPU arm
# ---------------------------------------------------------------------------

def flush_l2(buf):
    buf.add_(1.0)


def table_errors(got, ref):
    """Max and mean relative error per table, |g - r| / max(|r|, 1e-6 max|r|)
    (the floor keeps cells that are ~0 from dominating), as the parity tests
    measure it."""
    import numpy as np
    out = {}
    for k in TABLES:
        g = np.asarray(got[k], dtype=np.float64)
        r = np.asarray(ref[k], dtype=np.float64)
        e = np.abs(g - r) / np.maximum(np.abs(r), 1e-6 * max(np.abs(r).max(), 1e-300))
        out[k] = {"max": float(e.max()), "mean": float(e.mean())}
    return out


def run_ours(args):
    import torch
    import torch.distributed as dist

    from sfsim_gb300 import _lib, atmosphere_lut as A, config as C

    rank, world, local = dist_env()
    torch.cuda.set_device(local)
    if world > 1:
        dist.init_process_group("nccl", device_id=torch.device("cuda", local))
    L = _lib.load()
    cfg = C.production()
    n4 = 1
    for v in cfg.ray_scatter_shape:
        n4 *= v
    shapes = A.table_shapes(cfg)
    dev_out = [torch.empty(s, dtype=torch.float32, device="cuda") for s in shapes]
    host_out = [torch.empty(s, dtype=torch.float32, pin_memory=True) for s in shapes]
    flush = torch.empty(64 * 1024 * 1024, dtype=torch.float32, device="cuda")  # 256 MB > L2
    stream = torch.cuda.current_stream()

    def build_device():
        _lib.check(L.sfsim_atmo_build_device(ctypes.byref(cfg), *[t.data_ptr() for t in dev_out],
                                             ctypes.c_void_p(stream.cuda_stream)), "build_device")

    fp = ctypes.POINTER(ctypes.c_float)

    def build_host():
        _lib.check(L.sfsim_atmo_build(ctypes.byref(cfg), *[ctypes.cast(t.data_ptr(), fp) for t in host_out]),
                   "build")

    for _ in range(max(args.warmup, 3)):
        build_device()
    torch.cuda.synchronize()

    # --- device-resident timing: K builds, per-step CUDA events, L2 flushed between steps
    clocks = ClockSampler(local)
    clocks.start()
    starts = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps)]
    ends = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps)]
    if world > 1:
        dist.barrier()
    torch.cuda.synchronize()
    for k in range(args.steps):
        flush_l2(flush)
        starts[k].record(stream)
        build_device()
        ends[k].record(stream)
    torch.cuda.synchronize()
    if world > 1:
        dist.barrier()
    clk = clocks.stop()
    step_ms = [s.elapsed_time(e) for s, e in zip(starts, ends)]
    launches = L.sfsim_atmo_last_launch_count()
    total_ms = sum(step_ms)
    if world > 1:
        t = torch.tensor([total_ms], device="cuda")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        total_ms = float(t.item())
    value = world * n4 * args.steps / (total_ms * 1e-3)

    # --- stage timings and the dominant kernel (first order) with events on the build stream
    read = A.stage_timings(True)
    stage_runs = []
    for _ in range(3):
        flush_l2(flush)
        build_device()
        torch.cuda.synchronize()
        stage_runs.append(read())
    A.stage_timings(False)
    stages = {k: statistics.median(r[k] for r in stage_runs) for k in stage_runs[0]}

    # --- end to end through the public API with host buffers
    for _ in range(2):
        build_host()
    torch.cuda.synchronize()
    if world > 1:
        dist.barrier()
    t0 = time.perf_counter()
    for _ in range(args.steps):
        build_host()
    e2e_s = time.perf_counter() - t0
    if world > 1:
        t = torch.tensor([e2e_s], device="cuda")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        e2e_s = float(t.item())
    e2e = world * n4 * args.steps / e2e_s
    # the bytes the library copied in the last build: parameters and
    # quadrature directions in, the four tables out
    h2d_b, d2h_b = ctypes.c_ulonglong(), ctypes.c_ulonglong()
    _lib.check(L.sfsim_atmo_last_transfer_bytes(ctypes.byref(h2d_b), ctypes.byref(d2h_b)), "transfer bytes")
    params_bytes, d2h = h2d_b.value, d2h_b.value
    assert d2h == sum(t.numel() * 4 for t in host_out)

    # --- per-table error of the production tables against the FP64 path of
    # the same kernels (outside the timed regions)
    fp64_tables = A.build(C.production(precision=C.FP64))
    err_fp64 = table_errors({k: t.numpy() for k, t in zip(TABLES, host_out)}, fp64_tables)
    scan_rays = run_scan_rays(A, C, fp64_tables, stages["setup"]) if args.extras else None
    del fp64_tables

    # --- rooflines: point scatter (the largest stage, shared-memory gathers)
    # and the first order (SFU exponentials)
    counts = (ctypes.c_ulonglong * 10)()
    _lib.check(L.sfsim_atmo_census(ctypes.byref(cfg), counts, 10), "census")
    lit, climb = counts[0], counts[6]
    dir_evals, ground_evals, first_evals = counts[3], counts[7], counts[8]
    # per direction and inner heading: the ring row's RGB value and step to the
    # next texel (24 B); the first iteration's Mie row another 24 B, a ground
    # direction's surface radiance another 24 B.  The first and last heading's
    # sums are formed once per block and read together (24 B a direction).
    n3 = cfg.ray_scatter_shape[3]
    ps_bytes = 24 * (dir_evals + first_evals + ground_evals) * (n3 - 2) // n3 + 24 * dir_evals // n3
    smem_peak = ctypes.c_double()
    _lib.check(L.sfsim_atmo_smem_peak(ctypes.byref(smem_peak)), "smem_peak")
    ps_ms = stages["point_scatter"]
    ps_achieved = 128 * PS_SMEM_WAVEFRONTS / (ps_ms * 1e-3) / 1e9
    ps_gathered = ps_bytes / (ps_ms * 1e-3) / 1e9
    smem_peak_g = smem_peak.value / 1e9
    peak = ctypes.c_double()
    _lib.check(L.sfsim_atmo_sfu_peak(ctypes.byref(peak)), "sfu_peak")
    fo_ms = stages["first_order"]
    # exponentials of the first-order stage: per lit (node, sample) pair 3
    # transmittances and 2 mean densities from the fitted sun rays, and the
    # fits' own integrations (S samples of 2)
    fo_ex2 = 5 * lit + 2 * SUN_FIT_NODES * cfg.ray_steps
    fo_achieved = fo_ex2 / (fo_ms * 1e-3) / 1e9
    peak_g = peak.value / 1e9
    # ray scatter: per view row and ray sample a plane of n2 x n3 cells is
    # written (12 B each) and n2 x (n3 + 2) heading columns gather two of its
    # texels each (24 B), in every iteration
    rs_ms = stages["ray_scatter"]
    rs_samples = n4 // n3 * cfg.ray_steps * cfg.iterations  # (row, sun elevation, sample)
    rs_bytes = (12 * n3 + 24 * (n3 + 2)) * rs_samples
    rs_achieved = rs_bytes / (rs_ms * 1e-3) / 1e9

    sweep = run_sweep(L, A, C) if args.extras else None
    queries = run_queries(C) if args.extras else None
    queries_cond = run_cond_queries(C) if args.extras else None
    small_graph = run_small_graph(A, C) if args.extras else None
    ref_prod = run_reference_production(A, C) if args.extras else None
    noise_builders = run_noise() if args.extras else None

    if world > 1:
        dist.barrier()
    result = None
    if rank == 0:
        cpu, err_oracle = None, None
        if world == 1:
            # the CPU leg evaluates its sampled nodes from the GPU build's own
            # previous-order tables and reports their agreement
            inter = A.build(cfg, intermediates=True)
            cpu = cpu_baseline(cfg, args.cpu_sample_s, inter)
            err_oracle = cpu.pop("err_vs_gpu")
            del inter
        result = {
            "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": max(args.warmup, 3), "ms_per_step": total_ms / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": {"workload": WORKLOAD, "cells_per_build": n4, "parallelism": f"replicas{world}",
                       "l2": "L2 flushed (256 MB write) between timed steps; working set ~450 MB > L2"},
            "build_s": total_ms / args.steps * 1e-3,
            "e2e": {"value": e2e, "unit": UNIT, "h2d_bytes_per_step": params_bytes, "d2h_bytes_per_step": d2h,
                    "build_s": e2e_s / args.steps},
            "gpu_launches": launches * args.steps,
            "stage_ms": {k: round(v, 4) for k, v in stages.items()},
            "roofline": {"bound": "smem", "kernel": "k_point_scatter", "achieved": ps_achieved,
                         "peak": smem_peak_g, "unit": "GB/s", "frac": ps_achieved / smem_peak_g if smem_peak_g else None,
                         "traffic": PS_DRAM_BYTES_PER_LAUNCH,
                         "traffic_source": "ncu capture of this workload (recorded figure, not measured in this run)",
                         "gather_achieved": ps_gathered,
                         "note": ("achieved = 128 B per shared-memory wavefront of the point-scatter stage (a recorded "
                                  "ncu count of this workload) / its event time; gather_achieved = the gathers' bytes "
                                  "by lane (24 B per direction and inner heading for the ring's row, 24 B more in the "
                                  "first iteration and on the ground, 24 B per direction for the two outer headings; "
                                  "census counts), of which lanes that share a record are served together; issue and "
                                  "the FMA pipe are as busy; peak = "
                                  "conflict-free shared-memory read bandwidth measured live on this GPU by "
                                  "sfsim_atmo_smem_peak (no such figure in MEASURED_PEAKS.json); DRAM is not "
                                  "the bound (the tables live in L2); traffic = DRAM bytes read + written per "
                                  "point-scatter launch, mean of the build's five launches in one ncu capture of "
                                  "this workload"),
                         "direction_evaluations": dir_evals, "kernel_ms": ps_ms},
            "roofline_first_order": {"bound": "issue", "kernel": "k_first_order_fit", "achieved": fo_achieved,
                                     "peak": peak_g, "unit": "Gex2/s", "frac": fo_achieved / peak_g if peak_g else None,
                                     "note": ("exponentials of the stage: 3 transmittances and 2 fitted mean densities "
                                              "per lit sample, 2 per sample of the fits' own sun rays (8192 heights x 8 "
                                              "segments x 6 nodes); the stage is bound by instruction issue and "
                                              "latency, not the SFU; peak = ex2.approx throughput measured live"),
                                     "lit_pairs": lit, "climbing_pairs": climb, "kernel_ms": fo_ms},
            "roofline_ray_scatter": {"bound": "smem", "kernel": "k_ray_scatter", "achieved": rs_achieved,
                                     "peak": smem_peak_g, "unit": "GB/s",
                                     "frac": rs_achieved / smem_peak_g if smem_peak_g else None,
                                     "note": ("achieved = shared-memory bytes of the stage (planes written, 12 B a "
                                              "cell, and two RGB texels, 24 B, gathered per heading column) / its "
                                              "event time; the L1 data pipe also carries the builders' constants and "
                                              "the J loads; peak = the live conflict-free shared-memory read "
                                              "bandwidth"),
                                     "node_samples": n4 * cfg.ray_steps * cfg.iterations, "kernel_ms": rs_ms},
            "clocks": clk,
            "err_vs_fp64": {"tables": err_fp64, "against": ("the FP64 production build of the same kernels "
                                                            "(every cell)")},
            "err_vs_oracle": err_oracle,
            "scan_rays": scan_rays,
            "cpu_baseline": cpu,
            "sweep": sweep,
            "queries": queries,
            "queries_conditioned": queries_cond,
            "small_build_graph": small_graph,
            "reference_production_build": ref_prod,
            "noise": noise_builders,
        }
        print(json.dumps(result), flush=True)
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()
    return result


# ---------------------------------------------------------------------------
# secondary measurements: parameter sweep, queries and the surrogate
# ---------------------------------------------------------------------------

def run_sweep(L, A, C):
    """64 atmospheres drawn from the sweep distribution, shapes 16x128x16x8, 4
    iterations, built in one batched pass; device time from the stage events."""
    import time as _t
    import numpy as np
    cfgs = C.parameter_sweep(64)
    read = A.stage_timings(True)
    A.build_batch(cfgs[:2])  # warm-up
    t0 = _t.perf_counter()
    A.build_batch(cfgs)
    wall = _t.perf_counter() - t0
    dev_ms = sum(read().values())
    A.stage_timings(False)
    n4 = 1
    for v in cfgs[0].ray_scatter_shape:
        n4 *= v
    # per-table error of the FP32 tables against the FP64 path of the same
    # kernels on the same 64 atmospheres (outside the timed region)
    got = A.build_batch(cfgs)
    ref = A.build_batch(C.parameter_sweep(64, precision=C.FP64))
    err = {}
    for k in ("transmittance", "surface_radiance", "ray_scatter", "mie_strength"):
        g = got[k].reshape(len(cfgs), -1).astype(np.float64)
        r = ref[k].reshape(len(cfgs), -1).astype(np.float64)
        floor = 1e-6 * np.maximum(np.abs(r).max(axis=1, keepdims=True), 1e-300)
        e = np.abs(g - r) / np.maximum(np.abs(r), floor)
        err[k] = {"max": float(e.max()), "mean": float(e.mean())}
    return {"atmospheres": len(cfgs), "shape": list(cfgs[0].ray_scatter_shape), "iterations": cfgs[0].iterations,
            "device_s": dev_ms * 1e-3, "e2e_s": wall, "cells_per_s": len(cfgs) * n4 / (dev_ms * 1e-3),
            "err_vs_fp64": err}


def run_scan_rays(A, C, fp64_tables, nested_setup_ms, reps=10):
    """The production build with the SCAN_RAYS flag (view-ray transmittances
    by one prefix scan per ray instead of the nested quadrature, a different
    discretisation): device time per build (CUDA events, L2 flushed between
    builds), its set-up stage beside the nested build's, and its per-table
    deviation from the FP64 nested production tables."""
    import torch
    cfg = C.production()
    cfg.flags = C.SCAN_RAYS
    dev = [torch.empty(s, dtype=torch.float32, device="cuda") for s in A.table_shapes(cfg)]
    flush = torch.empty(64 * 1024 * 1024, dtype=torch.float32, device="cuda")
    for _ in range(3):
        A.build_device(cfg, dev)
    torch.cuda.synchronize()
    ms = []
    for _ in range(reps):
        flush.add_(1.0)
        s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s.record()
        A.build_device(cfg, dev)
        e.record()
        torch.cuda.synchronize()
        ms.append(s.elapsed_time(e))
    read = A.stage_timings(True)
    flush.add_(1.0)
    A.build_device(cfg, dev)
    torch.cuda.synchronize()
    setup_ms = read()["setup"]
    A.stage_timings(False)
    err = table_errors(A.build(cfg), fp64_tables)
    return {"ms_per_build": statistics.median(ms), "setup_ms": setup_ms, "nested_setup_ms": nested_setup_ms,
            "err_vs_nested_fp64": err,
            "note": ("not the reference's algorithm: T(x, p_s) from the midpoint rule on the whole cells before "
                     "p_s plus the half cell up to it, one warp-shuffle scan per view ray; the transmittance "
                     "table does not depend on it")}


def run_reference_production(A, C, reps=10):
    """The build sfsim's own `clj -T:build atmosphere-lut` runs (the
    reference's settings: 35 km atmosphere, T 64x255, E 16x63, S/M
    32x127x32x8, 100 ray steps, sphere steps 15, 5 iterations) in FP32:
    device time per build (CUDA events, L2 flushed between builds) and end to
    end through sfsim_atmo_build with pinned host buffers."""
    import torch
    cfg = C.reference_production()
    dev = [torch.empty(s, dtype=torch.float32, device="cuda") for s in A.table_shapes(cfg)]
    host = [torch.empty(s, dtype=torch.float32, pin_memory=True) for s in A.table_shapes(cfg)]
    flush = torch.empty(64 * 1024 * 1024, dtype=torch.float32, device="cuda")
    for _ in range(3):
        A.build_device(cfg, dev)
    torch.cuda.synchronize()
    ms = []
    for _ in range(reps):
        flush.add_(1.0)
        s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s.record()
        A.build_device(cfg, dev)
        e.record()
        torch.cuda.synchronize()
        ms.append(s.elapsed_time(e))
    L = A._lib.load()
    fp = ctypes.POINTER(ctypes.c_float)
    A._lib.check(L.sfsim_atmo_build(ctypes.byref(cfg), *[ctypes.cast(t.data_ptr(), fp) for t in host]), "build")
    t0 = time.perf_counter()
    for _ in range(reps):
        A._lib.check(L.sfsim_atmo_build(ctypes.byref(cfg), *[ctypes.cast(t.data_ptr(), fp) for t in host]), "build")
    e2e = (time.perf_counter() - t0) / reps
    n4 = 1
    for v in cfg.ray_scatter_shape:
        n4 *= v
    return {"config": cfg.describe(), "cells": n4, "device_ms": statistics.median(ms), "e2e_ms": e2e * 1e3}


def run_small_graph(A, C, reps=200):
    """The small FP64 and FP32 builds (8x16x8x4, 64 ray steps, 2 iterations),
    where launch overhead matters: device time per build through
    build_device, and through a plan's build captured once into a CUDA graph
    and replayed (CUDA events around `reps` back-to-back builds)."""
    import torch
    out = {}
    for name, prec in (("fp64", C.FP64), ("fp32", C.FP32)):
        cfg = C.small_fp64(precision=prec)
        tensors = [torch.empty(s, dtype=torch.float32, device="cuda") for s in A.table_shapes(cfg)]
        plan = A.Plan(cfg)
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(3):
                plan.build(tensors, stream=side)
                A.build_device(cfg, tensors, stream=side)
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            plan.build(tensors, stream=torch.cuda.current_stream())
        torch.cuda.synchronize()

        def timed(fn):
            s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            fn()
            torch.cuda.synchronize()
            s.record()
            for _ in range(reps):
                fn()
            e.record()
            torch.cuda.synchronize()
            return s.elapsed_time(e) / reps
        out[name] = {"build_device_ms": timed(lambda: A.build_device(cfg, tensors)),
                     "graph_replay_ms": timed(g.replay), "reps": reps}
        del g
        plan.close()
    return out


def _random_queries(n, R, H, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    h = torch.rand(n, device="cuda", dtype=torch.float64, generator=g) * H

    def unit():
        v = torch.randn(n, 3, device="cuda", dtype=torch.float64, generator=g)
        return v / v.norm(dim=1, keepdim=True)
    return unit() * (R + h)[:, None], unit(), unit()


def _timed(fn, reps=3):
    import torch
    fn()
    torch.cuda.synchronize()
    s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    best = None
    for _ in range(reps):
        s.record()
        r = fn()
        e.record()
        torch.cuda.synchronize()
        ms = s.elapsed_time(e)
        best = ms if best is None else min(best, ms)
    return best, r


def query_error_stats(a, ref):
    """Per-query relative error (max over RGB, floor 1e-6 of the largest
    reference value) summarised."""
    import torch
    floor = 1e-6 * ref.abs().max()
    e = ((a - ref).abs() / torch.maximum(ref.abs(), floor)).max(dim=1).values
    sample = e[:: max(1, e.numel() >> 20)].double()  # quantile takes at most 2^24 values
    q = torch.quantile(sample, torch.tensor([0.5, 0.9, 0.99], device=e.device, dtype=torch.float64))
    return {"median": float(q[0]), "p90": float(q[1]), "p99": float(q[2]), "max": float(e.max()),
            "frac_le_1e-3": float((e <= 1e-3).double().mean()), "frac_le_1e-2": float((e <= 1e-2).double().mean())}


def run_noise():
    """The cloud-noise build steps through the C ABI (host arrays in and out,
    allocation and copies included) against the oracle's single-threaded C
    restatement on the same random inputs, at the reference's default sizes
    and at larger ones."""
    import time as _t

    import numpy as np

    from oracle import oracle as O
    from sfsim_gb300 import noise

    def timed(fn, reps=3):
        fn()
        best = None
        for _ in range(reps):
            t0 = _t.perf_counter()
            r = fn()
            dt = _t.perf_counter() - t0
            best = dt if best is None else min(best, dt)
        return best * 1e3, r

    out = {}
    rng = np.random.default_rng(7)
    for d, size in ((4, 16), (8, 128)):
        grid = noise.random_point_grid(d, size, rng)
        g_ms, g = timed(lambda: noise.worley_noise(d, size, grid=grid))
        c_ms, c = timed(lambda: O.worley(d, size, grid), reps=1)
        out[f"worley_{size}^3_div{d}"] = {"gpu_ms": g_ms, "cpu_oracle_ms": c_ms, "max_abs_diff": float(np.abs(g - c).max())}
        grad = noise.random_gradient_grid(d, rng)
        g_ms, g = timed(lambda: noise.perlin_noise(d, size, gradients=grad))
        c_ms, c = timed(lambda: O.perlin(d, size, grad), reps=1)
        out[f"perlin_{size}^3_div{d}"] = {"gpu_ms": g_ms, "cpu_oracle_ms": c_ms, "max_abs_diff": float(np.abs(g - c).max())}
    for m in (64, 128):
        pixels = rng.permutation(m * m)[: (m * m) // 10]
        g_ms, g = timed(lambda: noise.blue_noise(m, sigma=1.5, seed_pixels=pixels), reps=2)
        c_ms, c = timed(lambda: O.blue(m, pixels, 1.5), reps=1)
        out[f"bluenoise_{m}x{m}"] = {"gpu_ms": g_ms, "cpu_oracle_ms": c_ms, "ranks_equal": bool(np.array_equal(g, c))}
    out["note"] = ("GPU times through sfsim_noise_* with host buffers; CPU = the FP64 C oracle, one thread, "
                   "same random inputs")
    return out


MLP_FLOPS_PER_QUERY = 2 * (192 * 256 + 3 * 256 * 256 + 256 * 4)


def surrogate_roofline(n, ms):
    """Tensor roofline of a surrogate call: the network's algorithmic flops
    over the whole call (lookup and packing included) against the measured
    BF16 peak (burst, the call is timed alone)."""
    peak = None
    try:
        with open(os.path.join(os.path.dirname(os.path.abspath(__file__)), "MEASURED_PEAKS.json")) as f:
            peak = json.load(f).get("bf16_tflops")
    except (OSError, ValueError):
        pass
    src = "MEASURED_PEAKS.json bf16_tflops (burst)"
    if not peak:
        peak, src = 1900.0, "fallback 1.9 PFLOP/s"
    achieved = n * MLP_FLOPS_PER_QUERY / (ms * 1e-3) / 1e12
    return {"bound": "tensor", "kernel": "k_surrogate_infer", "achieved": achieved, "peak": peak,
            "unit": "TFLOP/s", "frac": achieved / peak, "peak_source": src,
            "flops_per_query": MLP_FLOPS_PER_QUERY}


def run_queries(C, steps=20000, batch=65536, direct_samples=1 << 25, lr=3e-3, huber_delta=0.02,
                thresholds=(3e-2, 1e-2, 3e-3, 1e-3)):
    """2^24 random in-scatter queries (height uniform 0-100 km, view and sun
    uniform on the sphere) on the production tables: table lookup, direct
    quadrature, the trained surrogate (the lookup with the network's
    correction) and the surrogate with fallback to direct quadrature where its
    predicted error exceeds a threshold; errors relative to direct quadrature."""
    import time as _t

    import torch

    from sfsim_gb300.query import Context
    cfg = C.production()
    ctx = Context(cfg)
    t0 = _t.perf_counter()
    hist = ctx.train_surrogate(steps=steps, batch=batch, direct_samples=direct_samples, node_fraction=0.0, lr=lr,
                               seed=1, huber_delta=huber_delta)
    torch.cuda.synchronize()
    train_s = _t.perf_counter() - t0
    n = 1 << 24
    x, v, l = _random_queries(n, cfg.radius, cfg.height, 2)
    x32, v32, l32 = x.float(), v.float(), l.float()
    out = torch.empty((n, 3), dtype=torch.float32, device="cuda")
    t_table, table = _timed(lambda: ctx.table(4, x32, v32, l32, out=out).clone())
    t_direct, direct = _timed(lambda: ctx.direct(x, v, l, out=out).clone(), reps=1)
    t_sur, (sur, _) = _timed(lambda: ctx.surrogate(x, v, l, out=out))
    sur = sur.clone()
    qps = lambda ms: n / (ms * 1e-3)  # noqa: E731
    r = {"n": n, "train_steps": steps, "train_batch": batch, "direct_samples": direct_samples, "lr": lr,
         "huber_delta": huber_delta, "train_s": train_s,
         "train_loss_first": float(hist[:10].mean()), "train_loss_last": float(hist[-100:].mean()),
         "table": {"qps": qps(t_table), "err": query_error_stats(table, direct)},
         "direct": {"qps": qps(t_direct)},
         "surrogate": {"qps": qps(t_sur), "err": query_error_stats(sur, direct), "vs_direct": t_direct / t_sur,
                       "roofline": surrogate_roofline(n, t_sur)}}
    del table, sur
    for thr in thresholds:
        t_fb, (fb, nf) = _timed(lambda: ctx.surrogate(x, v, l, threshold=thr, out=out), reps=1)
        r[f"surrogate_fallback_{thr:g}"] = {"qps": qps(t_fb), "fallback_fraction": nf / n,
                                            "err": query_error_stats(fb, direct), "vs_direct": t_direct / t_fb}
    r["first_recipe_baseline"] = first_recipe_baseline(ctx, cfg, x[: 1 << 21], v[: 1 << 21], l[: 1 << 21],
                                                 direct[: 1 << 21], steps=steps, batch=batch)
    ctx.close()
    return r


def first_recipe_baseline(ctx, cfg, x, v, l, direct, steps, batch, n_direct=1 << 23, seed=1):
    """The surrogate recipe as first specified, the baseline the product's
    correction network replaced: the four table coordinates -> 16 sin/cos
    Fourier frequencies each (128 features) -> 4 x 256 SiLU -> 3 log-RGB
    values, predicted outright; Adam, learning rate 1e-3 with cosine decay,
    batches of 65536 drawing 75% table nodes (the node's S + M phase) and 25%
    uniform points integrated by the direct quadrature.  Fitted with torch
    (TF32 matmuls, FP32 weights) as a baseline only; errors on the given
    queries against the direct quadrature."""
    import torch
    eps = 1e-7
    g = torch.Generator(device="cuda").manual_seed(seed)
    T, E, S2, M2 = ctx.tables()
    n0, n1, n2, n3 = cfg.ray_scatter_shape
    S = S2.view(n0, n2, n1, n3, 3).permute(0, 2, 1, 3, 4).reshape(-1, 3)
    M = M2.view(n0, n2, n1, n3, 3).permute(0, 2, 1, 3, 4).reshape(-1, 3)
    idx = torch.stack(torch.meshgrid(*[torch.arange(m, device="cuda") for m in (n0, n1, n2, n3)], indexing="ij"),
                      -1).reshape(-1, 4).float()
    node_u = idx / torch.tensor([n0 - 1, n1 - 1, n2 - 1, n3 - 1], device="cuda", dtype=torch.float32)
    mu = 2.0 * node_u[:, 3] - 1.0
    gm = 0.76
    phase = 3 * (1 - gm * gm) * (1 + mu * mu) / (8 * torch.pi * (2 + gm * gm) * (1 + gm * gm - 2 * gm * mu) ** 1.5)
    node_t = torch.log((S + M * phase[:, None]).clamp(min=0) + eps)
    dx, dv, dl = _random_queries(n_direct, cfg.radius, cfg.height, 11)
    dir_u = ctx.coords(dx, dv, dl)[:, :4].contiguous()
    dir_t = torch.log(ctx.direct(dx, dv, dl).clamp(min=0) + eps)
    del dx, dv, dl
    k = torch.arange(16, device="cuda")
    freq = torch.where(k % 2 == 1, torch.tensor(2 ** 0.5, device="cuda"), torch.tensor(1.0, device="cuda")) * 2.0 ** (k // 2)

    def features(u):
        a = torch.pi * u[:, :, None] * freq[None, None, :]
        return torch.stack([torch.sin(a), torch.cos(a)], -1).reshape(u.shape[0], 128)

    torch.manual_seed(seed)
    layers = [torch.nn.Linear(128, 256), torch.nn.SiLU()]
    for _ in range(3):
        layers += [torch.nn.Linear(256, 256), torch.nn.SiLU()]
    net = torch.nn.Sequential(*layers, torch.nn.Linear(256, 3)).cuda()
    opt = torch.optim.Adam(net.parameters(), lr=1e-3)
    sched = torch.optim.lr_scheduler.CosineAnnealingLR(opt, steps)
    tf32 = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = True
    nn_ = batch * 3 // 4
    for _ in range(steps):
        a = torch.randint(0, node_u.shape[0], (nn_,), device="cuda", generator=g)
        b = torch.randint(0, dir_u.shape[0], (batch - nn_,), device="cuda", generator=g)
        u = torch.cat([node_u[a], dir_u[b]])
        t = torch.cat([node_t[a], dir_t[b]])
        loss = torch.nn.functional.mse_loss(net(features(u)), t)
        opt.zero_grad(set_to_none=True)
        loss.backward()
        opt.step()
        sched.step()
    with torch.no_grad():
        u = ctx.coords(x, v, l)[:, :4].contiguous()
        pred = torch.cat([torch.exp(net(features(u[i:i + (1 << 18)]))) - eps for i in range(0, u.shape[0], 1 << 18)])
    torch.backends.cuda.matmul.allow_tf32 = tf32
    return {"err": query_error_stats(pred.clamp(min=0), direct), "n": int(u.shape[0]), "steps": steps,
            "note": ("the first surrogate recipe (4 coordinates, 128 Fourier features, 4 x 256 SiLU, 3 log-RGB "
                     "outright, 75% table nodes, lr 1e-3 cosine), fitted in torch as the baseline the "
                     "correction network replaced; not the product")}


def run_cond_queries(C, n_train=32, n_held_out=8, steps=10000, batch=65536, direct_samples=1 << 20, lr=3e-3,
                     huber_delta=0.02, thresholds=(3e-2, 1e-3)):
    """The conditioned surrogate: trained on 32 atmospheres of the parameter
    sweep (tables 16x128x16x8, 4 iterations; 2^20 direct samples each, 2^25 in
    all), queried on 8 held-out atmospheres drawn from the same distribution
    with another seed, 2^21 queries each (height uniform 0-100 km, view and sun
    uniform); errors relative to each atmosphere's direct quadrature."""
    import time as _t

    import torch

    from sfsim_gb300.query import ConditionedSurrogate, Context
    train_cfgs = C.parameter_sweep(n_train)
    held_cfgs = C.parameter_sweep(n_held_out, seed=C.SWEEP_SEED + 1)
    t0 = _t.perf_counter()
    train_ctx = [Context(c) for c in train_cfgs]
    torch.cuda.synchronize()
    build_s = _t.perf_counter() - t0
    cs = ConditionedSurrogate(seed=1)
    t0 = _t.perf_counter()
    hist = cs.train(train_ctx, steps=steps, batch=batch, direct_samples=direct_samples, node_fraction=0.0, lr=lr,
                    seed=1, huber_delta=huber_delta)
    torch.cuda.synchronize()
    train_s = _t.perf_counter() - t0
    for c in train_ctx:
        c.close()
    n = 1 << 21
    ms = {"table": 0.0, "direct": 0.0, "surrogate": 0.0}
    parts = {"table": [], "direct": [], "surrogate": []}
    for thr in thresholds:
        ms[thr] = 0.0
        parts[thr] = []
    flagged = {thr: 0 for thr in thresholds}
    for k, cfg in enumerate(held_cfgs):
        ctx = Context(cfg)
        x, v, l = _random_queries(n, cfg.radius, cfg.height, 100 + k)
        x32, v32, l32 = x.float(), v.float(), l.float()
        out = torch.empty((n, 3), dtype=torch.float32, device="cuda")
        t, r = _timed(lambda: ctx.table(4, x32, v32, l32, out=out).clone())
        ms["table"] += t
        parts["table"].append(r)
        t, r = _timed(lambda: ctx.direct(x, v, l, out=out).clone(), reps=1)
        ms["direct"] += t
        parts["direct"].append(r)
        t, (r, _) = _timed(lambda: cs.query(ctx, x, v, l, out=out))
        ms["surrogate"] += t
        parts["surrogate"].append(r.clone())
        for thr in thresholds:
            t, (r, nf) = _timed(lambda: cs.query(ctx, x, v, l, threshold=thr, out=out), reps=1)
            ms[thr] += t
            parts[thr].append(r.clone())
            flagged[thr] += nf
        ctx.close()
    cat = {k: torch.cat(v) for k, v in parts.items()}
    total = n * len(held_cfgs)
    qps = lambda t: total / (t * 1e-3)  # noqa: E731
    cs.close()
    r = {"train_atmospheres": n_train, "held_out_atmospheres": n_held_out, "shape": list(train_cfgs[0].ray_scatter_shape),
            "n": total, "train_steps": steps, "train_batch": batch, "direct_samples": direct_samples * n_train,
            "lr": lr, "huber_delta": huber_delta, "context_builds_s": build_s, "train_s": train_s,
            "train_loss_first": float(hist[:10].mean()), "train_loss_last": float(hist[-100:].mean()),
            "table": {"qps": qps(ms["table"]), "err": query_error_stats(cat["table"], cat["direct"])},
            "direct": {"qps": qps(ms["direct"])},
            "surrogate": {"qps": qps(ms["surrogate"]), "err": query_error_stats(cat["surrogate"], cat["direct"]),
                          "vs_direct": ms["direct"] / ms["surrogate"]}}
    for thr in thresholds:
        r[f"surrogate_fallback_{thr:g}"] = {"qps": qps(ms[thr]), "fallback_fraction": flagged[thr] / total,
                                            "err": query_error_stats(cat[thr], cat["direct"]),
                                            "vs_direct": ms["direct"] / ms[thr]}
    return r


# ---------------------------------------------------------------------------
# CPU baseline: the FP64 restatement of the reference (oracle/), all host threads
# ---------------------------------------------------------------------------

def cpu_sample(cfg, seconds: float, threads: int, seed: int = 0, inter=None, min_nodes: int = 256):
    """Times sampled nodes of each build stage with `threads` host threads and
    extrapolates the whole build by node counts.  Returns (build_s, detail,
    errors).

    Without `inter` the nodes read synthetic previous-order tables (the work
    per node does not depend on the values).  With `inter`, the GPU build's
    intermediate tables of the same configuration, every node of every
    iteration is evaluated from the GPU's own previous-order tables, as the
    parity tests do, at least `min_nodes` seeded nodes per stage and
    iteration, and `errors` holds the relative error of the GPU's value at
    those nodes (max over RGB, floor 1e-6 of the GPU table's largest value)."""
    import concurrent.futures

    import numpy as np

    from oracle import oracle as O

    t_shape, e_shape, s = cfg.shapes()
    n4 = int(np.prod(s))
    rng = np.random.default_rng(seed)
    it = cfg.iterations

    def nodes(shape, n):
        return [tuple(int(rng.integers(0, m)) for m in shape) for _ in range(n)]

    if inter is None:
        tab4 = rng.uniform(0.0, 1e-2, size=tuple(s) + (3,))
        tab2 = rng.uniform(0.0, 1e-1, size=tuple(e_shape) + (3,))
        tasks = [("first_order", None, lambda nd: O.first_order_node(cfg, *nd), None, s),
                 ("point_scatter", None, lambda nd: O.point_scatter_node(cfg, tab4, tab2, *nd), None, s),
                 ("ray_scatter", None, lambda nd: O.ray_scatter_node(cfg, tab4, *nd), None, s)]
    else:
        f64 = lambda a: np.ascontiguousarray(a, dtype=np.float64)  # noqa: E731
        S1R, M = f64(inter["rayleigh_first"]), f64(inter["mie_first"])
        tasks = [("first_order", None, lambda nd: np.concatenate(O.first_order_node(cfg, *nd)),
                  lambda nd: np.concatenate([S1R[nd], M[nd]]), s)]
        for k in range(it):
            dS_prev = S1R if k == 0 else f64(inter["ray_scatter_delta"][k - 1])
            dE_prev = f64(inter["surface_base"] if k == 0 else inter["surface_delta"][k - 1])
            mf = M if k == 0 else None
            J, dS, dE = f64(inter["point_scatter"][k]), inter["ray_scatter_delta"][k], inter["surface_delta"][k]
            tasks.append(("point_scatter", k,
                          lambda nd, a=dS_prev, b=dE_prev, c=mf: O.point_scatter_node(cfg, a, b, *nd, mie_first=c),
                          lambda nd, J=J: J[nd], s))
            tasks.append(("ray_scatter", k, lambda nd, J=J: O.ray_scatter_node(cfg, J, *nd),
                          lambda nd, dS=dS: dS[nd], s))
            tasks.append(("surface_radiance", k,
                          lambda nd, a=dS_prev, c=mf: O.surface_radiance_node(cfg, a, *nd, mie_first=c),
                          lambda nd, dE=dE: dE[nd], e_shape))
    timed = ("first_order", "point_scatter", "ray_scatter")
    per_stage = {name: sum(1 for t in tasks if t[0] == name) for name in timed}
    spent, done = {n: 0.0 for n in timed}, {n: 0 for n in timed}
    errors = {}
    with concurrent.futures.ThreadPoolExecutor(max_workers=threads) as ex:
        for name, order, fn, gpu_value, shape in tasks:
            budget = seconds / len(timed) / per_stage.get(name, 1)
            count, errs, t0 = 0, [], time.perf_counter()
            while count < (min_nodes if gpu_value is not None else 1) or \
                    (name in timed and time.perf_counter() - t0 < budget):
                batch = nodes(shape, threads * 2)
                vals = list(ex.map(fn, batch))
                count += len(batch)
                if gpu_value is not None:
                    for nd, v in zip(batch, vals):
                        errs.append((np.asarray(gpu_value(nd), dtype=np.float64), np.asarray(v, dtype=np.float64)))
            if name in timed:
                spent[name] += time.perf_counter() - t0
                done[name] += count
            if gpu_value is not None:
                g = np.array([a for a, _ in errs])
                r = np.array([b for _, b in errs])
                if name == "first_order":  # Rayleigh and Mie, each against its own table's largest value
                    scale = np.repeat([np.abs(inter["rayleigh_first"]).max(), np.abs(inter["mie_first"]).max()], 3)
                else:
                    scale = np.abs({"point_scatter": inter["point_scatter"], "ray_scatter": inter["ray_scatter_delta"],
                                    "surface_radiance": inter["surface_delta"]}[name][order]).max()
                e = (np.abs(g - r) / np.maximum(np.abs(r), 1e-6 * np.maximum(scale, 1e-300))).max(axis=1)
                key = name if order is None else f"{name}[{order}]"
                errors[key] = {"max": float(e.max()), "mean": float(e.mean()), "nodes": int(len(e))}
    per_node = {n: spent[n] / max(done[n], 1) for n in timed}  # wall seconds per node at `threads`
    build_s = n4 * (per_node["first_order"] + it * (per_node["point_scatter"] + per_node["ray_scatter"]))
    return build_s, per_node, errors


CHECK_SHAPE = (16, 15, 4, 4)  # ray-scatter shape of the CPU baseline's complete build


def small_config(cfg):
    """cfg with its tables reduced to a 16x15x4x4 ray-scatter table (T 16x15, E
    16x16) and everything else (steps, iterations, physics) kept."""
    small = cfg.copy()
    for i, v in enumerate(CHECK_SHAPE):
        small.ray_scatter_shape[i] = v
    small.transmittance_shape[0], small.transmittance_shape[1] = 16, 15
    small.surface_radiance_shape[0], small.surface_radiance_shape[1] = 16, 16
    return small


def cpu_full_build(cfg, threads):
    """Wall seconds of one complete oracle build of small_config(cfg) on
    `threads` host threads (threaded over its 16 heights, as the reference's
    pmap is over dimension 0), and its ray-scatter cell count."""
    from oracle import oracle as O
    small = small_config(cfg)
    t0 = time.perf_counter()
    O.build(small, nthreads=threads)
    n4 = 1
    for v in CHECK_SHAPE:
        n4 *= v
    return time.perf_counter() - t0, n4


def cpu_baseline(cfg, seconds: float, inter=None):
    """The CPU baseline: complete FP64 oracle builds of the workload's steps,
    iterations and physics at a 16x15x4x4 ray-scatter table on all host
    threads, scaled to the workload's table by cell count (the work per cell
    does not depend on the table's shape).  The per-node sampler is reported
    beside it as a cross-check and, with `inter`, yields the GPU's errors at
    the sampled nodes."""
    threads = os.cpu_count() or 1
    n4 = 1
    for v in cfg.ray_scatter_shape:
        n4 *= v
    t_small, n_small = min((cpu_full_build(cfg, threads) for _ in range(2)), key=lambda r: r[0])
    build_s = t_small * n4 / n_small
    sampled_s, per_node, errors = cpu_sample(cfg, seconds, threads, inter=inter)
    out = {"value": n4 / build_s, "unit": UNIT, "cores": threads, "kind": "port",
           "build_s_extrapolated": build_s,
           "sample": (f"FP64 C restatement of the reference (oracle/atmo_oracle.c), {threads} threads: complete "
                      f"builds with the workload's steps, iterations and physics at a 16x15x4x4 ray-scatter "
                      f"table ({t_small:.2f} s, best of 2), scaled by cell count to {n4} cells"),
           "full_build_s_small": t_small,
           "per_node_sampler": {"build_s_extrapolated": sampled_s, "seconds_per_node": per_node,
                                "note": ("seeded random nodes of the first-order, point-scatter and ray-scatter "
                                         "stages timed one node at a time; overestimates the complete build "
                                         "(per-call set-up, Python threads)")}}
    if inter is not None:
        worst = max(v["max"] for v in errors.values())
        out["err_vs_gpu"] = {"stages": errors, "max": worst,
                             "against": ("the oracle at seeded nodes of every stage and iteration, each evaluated "
                                         "from the GPU build's own previous-order tables")}
    return out


def run_reference(args):
    """The reference arm: each step is one complete FP64 oracle build at a
    16x15x4x4 ray-scatter table with the workload's steps, iterations and
    physics on all host threads; value = its ray-scatter cells per second,
    the rate the workload's table is built at (the work per cell does not
    depend on the table's shape)."""
    rank, world, local = dist_env()
    if rank != 0:
        return None
    from sfsim_gb300 import config as C
    cfg = C.production()
    threads = os.cpu_count() or 1
    n4 = 1
    for v in cfg.ray_scatter_shape:
        n4 *= v
    for _ in range(max(args.warmup, 3)):
        cpu_full_build(C.shader_test(), threads)
    vals, times = [], []
    t0 = time.perf_counter()
    for _ in range(args.steps):
        t, n_small = cpu_full_build(cfg, threads)
        times.append(t)
        vals.append(n_small / t)
    wall = time.perf_counter() - t0
    value = statistics.median(vals)
    result = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
        "warmup": max(args.warmup, 3), "ms_per_step": wall / args.steps * 1e3, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic", "impl": "reference",
        "config": {"workload": WORKLOAD, "cells_per_build": n4, "parallelism": "host threads"},
        "build_s": n4 / value,
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": threads, "kind": "port",
                         "sample": (f"each step: one complete build of the FP64 C restatement "
                                    f"(oracle/atmo_oracle.c; the Clojure reference needs a JVM that is not "
                                    f"installed) with the workload's steps, iterations and physics at a "
                                    f"16x15x4x4 ray-scatter table ({statistics.median(times):.2f} s), whose cells "
                                    f"per second are the rate of the {n4}-cell table")},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(result), flush=True)
    return result


def run_profile(args):
    """Plain builds of one configuration with nothing else on the GPU (for ncu)."""
    import torch

    from sfsim_gb300 import atmosphere_lut as A, config as C
    cfg = getattr(C, args.profile)()
    torch.cuda.set_device(0)
    for _ in range(args.builds):
        A.build_device(cfg)
    torch.cuda.synchronize()
    print(json.dumps({"profile": args.profile, "builds": args.builds, "config": cfg.describe()}))


def run_profile_surrogate(args):
    """Four training steps (batch 65536) and --builds batches of N fused
    surrogate queries on the production tables (for ncu)."""
    import torch

    from sfsim_gb300 import config as C
    from sfsim_gb300.query import Context
    torch.cuda.set_device(0)
    cfg = C.production()
    with Context(cfg) as ctx:
        ctx.train_surrogate(steps=4, batch=65536, direct_samples=1 << 16, lr=1e-3, seed=1)
        n = args.profile_surrogate
        x, v, l = _random_queries(n, cfg.radius, cfg.height, 2)
        out = torch.empty((n, 3), dtype=torch.float32, device="cuda")
        for _ in range(args.builds):
            ctx.surrogate(x, v, l, out=out)
        torch.cuda.synchronize()
    print(json.dumps({"profile_surrogate": n, "builds": args.builds}))


def main():
    args = parse()
    if args.profile_surrogate:
        run_profile_surrogate(args)
    elif args.profile:
        run_profile(args)
    elif args.impl == "reference":
        run_reference(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
