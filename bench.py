#!/usr/bin/env python
"""Benchmark of the polesitter FMM tick on B200.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl b200|reference]
                    [--workload closure|plain]

A step is one tick exactly as the reference's callers run it
(tests/benchmark.c:175-184, README.md:74-88): ps_prepare_particles +
ps_calc_forces, every step from the same unsorted particle order (the tick
sorts the caller's arrays in place) and with L2 flushed, both outside the
timed step.

--workload closure (default; the headline metric): N = 1,048,576 particles of
the learned closure's snapshot family (an equal-mass Plummer sphere plus 32
sub-clumps holding 30% of the mass, seeded), theta = 6.25, leaf capacity 16,
closure mode 2: the order-1 local expansion, the shipped MLP correction and
the per-tick FP64 judge on 1024 sampled particles.  Beside it, the metric
itself: each method's ticks/s at the closure's error bound (median relative
force error <= 1e-3 against the FP64 direct sum) on the same snapshot -- the
plain GPU FMM (the reference's far field, mode 0) on the reference's tree and
on larger leaves, and the order-1 expansion without the network (mode 1) --
each at the first theta of its ladder that meets the bound.
--workload plain: the reference's plain tick on an N = 1,048,576 Plummer
sphere at theta = 2 (the configuration the parity tests pin).

Reported (one JSON line on rank 0):
  value      ticks/s of the whole job, device-resident arrays (all ranks)
  e2e        ticks/s through the same C ABI with pinned HOST arrays, the
             host<->device copies inside each step
  accuracy   median relative force error against FP64 direct sums
  roofline   the dominant phase (the leaf pass: MAC + M2L + L2L + P2P + L2P,
             or the full-leaf P2P + L2P), FP32-bound, from its CUDA-event time
             and algorithmic flop count
  cpu_baseline  the reference's own threaded CPU tick (oracle/_ref) on the
             same workload, timed on this host's cores
  plain_c2, tick_loop, ensemble  (closure workload, unless --minimal) the
             plain Plummer theta=2 tick; 100 device-resident Euler ticks of
             two colliding 4M-particle Plummer spheres; 256 independent
             systems in replayed CUDA graphs with the autotuner
With --gpus N > 1 every rank runs an independent replica (the path has no
exchange step on one system): weak scaling, value = N x ticks / max time.

--impl reference times the reference's CPU implementation of the same tick
(the unmodified header compiled by oracle/build_ref.sh) with all host threads.
"""

from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "ticks/s at N=1M, learned-closure vs plain GPU FMM at equal 1e-3 force error"
UNIT = "ticks/s"
N_DEFAULT = 1 << 20
ERROR_TARGET = 1e-3
CLOSURE_THETA = 6.25       # operating point: every tick's judge <= 8.7e-4 with the shipped
                           # weights (trained at theta 6.5); 6.0 sits at 9.8e-4
CLOSURE_LEAF_CAP = 16      # leaf capacity of the closure's tree (PS_B200_OPT_LEAF_CAP)
CLOSURE_SEED = 424242      # snapshot seed (the weights were trained on other seeds)
# theta ladders of the methods the closure is compared with at equal error:
# the plain GPU FMM on the reference's tree (leaf capacity 1) and on larger
# leaves, and the order-1 expansion without the network
PLAIN_LADDERS = ((1, (12.0, 16.0)),
                 (16, (24.0, 32.0, 40.0, 48.0)),
                 (32, (24.0, 28.0, 32.0, 40.0)),
                 (64, (24.0, 28.0, 32.0, 40.0)))
MODE1_LADDERS = ((16, (8.0, 9.0, 10.0, 11.0, 12.0)),
                 (32, (8.0, 9.0, 10.0, 11.0, 12.0)))
C2_THETA, C2_SEED = 2.0, 42
WORKLOADS = {
    "closure": ("learned-closure FMM tick (ps_prepare_particles + ps_calc_forces, closure mode 2: "
                "order-1 local expansion + BF16 MLP correction + FP64 judge on 1024 particles), "
                "N=1,048,576 clumpy Plummer (a=1, r<=10a, plus 32 sub-clumps with 30% of the mass, "
                "equal mass 1/N), theta=6.25, leaf capacity 16, float32 SoA"),
    "plain": ("plain FMM tick (ps_prepare_particles + ps_calc_forces), Plummer sphere "
              "N=1,048,576, a=1, r<=10a, equal mass 1/N, theta=2, float32 SoA"),
}
# kernels of this library launched per 1M tick: 2 prepare + 5 sort + gather +
# write-back + 4 tree + 4 upward + the internal levels + 2 leaf-pass variants +
# full leaves; the closure runs one leaf-pass variant, the internal levels in
# two launches with the split shallow groups between, and adds the judge
# (sample, FP64 direct sum over source splits, their fixed-order sum,
# decision), the MLP and the apply kernel
KERNELS_PER_TICK = {"plain": 21, "closure": 28}
# DRAM bytes (read + write) of one launch of the dominant kernel, from the
# ncu captures summarised under profiles/ (None: not captured for this
# configuration)
DOMINANT_DRAM_BYTES = {"plain": 271.9e6, "closure": 0.39e9}
TRAFFIC_NOTE = {
    "plain": "dram read+write bytes per launch, ncu capture of this workload",
    "closure": "dram read+write bytes per launch of k_dense_p2p, ncu capture of the same kernel "
               "at N=131072 (46.6 MB) scaled by the full-leaf pair count (x 8.41) to N=1M"}
FLOP_M2L = 35         # per M2L pair: polesitter.h:1065-1092
FLOP_M2L_ORDER1 = 59  # ... plus the monopole field gradient (closure order 1)
FLOP_P2P = 20         # per particle pair: polesitter.h:1424-1444


def parse_args():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=200)
    ap.add_argument("--warmup", type=int, default=10)
    ap.add_argument("--impl", choices=("b200", "reference"), default="b200")
    ap.add_argument("--workload", choices=("closure", "plain"), default="closure")
    ap.add_argument("--n", type=int, default=N_DEFAULT)
    ap.add_argument("--theta", type=float, default=None)
    ap.add_argument("--leaf-cap", type=int, default=None)
    ap.add_argument("--e2e-steps", type=int, default=10)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-plain-curve", action="store_true")
    ap.add_argument("--minimal", action="store_true",
                    help="only the timed ticks (for profiling runs): no plain curve, no plain "
                         "C2 line, one e2e step, no CPU baseline")
    return ap.parse_args()


def dist_info():
    return (int(os.environ.get("RANK", 0)), int(os.environ.get("LOCAL_RANK", 0)),
            int(os.environ.get("WORLD_SIZE", 1)))


def measured_peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(path):
        with open(path) as f:
            return json.load(f), "measured"
    return {"hbm_gbs": 6650.0, "bf16_tflops": 1590.0, "sm_max_mhz": 1965.0}, "fallback"


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled every 200 ms."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index):
        self.gpu = gpu_index
        self.proc = None
        self.tmp = tempfile.NamedTemporaryFile(mode="w+", suffix=".csv", delete=False)

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.gpu), f"--query-gpu={self.FIELDS}",
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=self.tmp, stderr=subprocess.DEVNULL)
        except FileNotFoundError:
            self.proc = None
        return self

    def __exit__(self, *exc):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        self.tmp.flush()
        rows = []
        with open(self.tmp.name) as f:
            for line in f:
                parts = [x.strip() for x in line.split(",")]
                if len(parts) >= 9:
                    rows.append(parts)
        os.unlink(self.tmp.name)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        sm = [float(r[1]) for r in rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in rows if r[2].replace(".", "").isdigit()]
        names = ("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap")
        reasons = sorted({n for r in rows for n, v in zip(names, r[5:9]) if v == "Active"})
        return {"sm_mhz": statistics.median(sm) if sm else None,
                "sm_max_mhz": max(mx) if mx else None, "reasons": reasons,
                "samples": len(rows)}


def particles(workload, n):
    from polesitter_b200 import workloads as W
    if workload == "closure":
        return W.clumpy_plummer(n, CLOSURE_SEED)
    return W.plummer(n, C2_SEED)


def theta_of(args):
    if args.theta is not None:
        return args.theta
    return CLOSURE_THETA if args.workload == "closure" else C2_THETA


def leaf_cap_of(args):
    if args.leaf_cap is not None:
        return args.leaf_cap
    return CLOSURE_LEAF_CAP if args.workload == "closure" else 1


def cpu_reference_ticks(p0, ticks, warmup, theta):
    """Time the reference's own tick (oracle/_ref, all host threads);
    fall back to the oracle port, single-threaded, if that build is absent."""
    cores = os.cpu_count() or 1
    from oracle import refbind
    if refbind.available(""):
        ref = refbind.RefLib("")
        run = lambda p: ref.tick(p, theta=theta, thrd_cnt=cores)  # noqa: E731
        kind, used = "reference", cores
    else:
        from oracle.oracle import Oracle
        o = Oracle()
        run = lambda p: o.tick(p, theta=theta, want_tree=False)  # noqa: E731
        kind, used = "port", 1
    for _ in range(warmup):
        run(p0.copy())
    times = []
    for _ in range(ticks):
        p = p0.copy()
        t0 = time.perf_counter()
        run(p)
        times.append(time.perf_counter() - t0)
    return {"value": len(times) / sum(times), "unit": UNIT, "cores": used, "kind": kind,
            "sample": f"{len(times)} full tick(s) of the workload (N={p0.n}, theta={theta}, the "
                      f"reference's own far field) after {warmup} warm-up, thrd_cnt={used}; "
                      f"median {statistics.median(times):.3f} s/tick"}


def run_reference(args):
    rank, _, world = dist_info()
    if rank != 0:
        return 0
    theta = theta_of(args)
    p0 = particles(args.workload, args.n)
    # a reference tick of the closure workload takes tens of seconds on the
    # host: a bounded sample of ticks
    ticks = min(args.steps, 2 if args.workload == "closure" else args.steps)
    warm = min(args.warmup, 1 if args.workload == "closure" else args.warmup)
    base = cpu_reference_ticks(p0, ticks, warm, theta)
    line = {"metric": METRIC, "value": base["value"], "unit": UNIT, "impl": "reference",
            "n_gpus": world, "steps": ticks, "warmup": warm,
            "ms_per_step": 1000.0 / base["value"], "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32",
            "data": "synthetic (seeded clumpy Plummer)" if args.workload == "closure"
            else "synthetic (seeded Plummer sphere)",
            "config": {"workload": WORKLOADS[args.workload], "n": args.n, "theta": theta,
                       "leaf_cap": 1,
                       "note": "the reference has only the plain far field on its own tree "
                               "(leaf capacity 1); at this theta its error is ~10x the "
                               "closure's, so it does less work than the 1e-3 bound needs"}
            if args.workload == "closure"
            else {"workload": WORKLOADS[args.workload], "n": args.n, "theta": theta},
            "cpu_baseline": base,
            "e2e": {"value": base["value"], "unit": UNIT, "h2d_bytes_per_step": 0,
                    "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)
    return 0


class Arrays:
    pass


def median_rel_error(ctx, arrs_dev, n, seed):
    """Median relative force error of the last tick against an FP64 direct
    sum on the GPU for 4096 sampled particles (arrays already sorted)."""
    rng = np.random.default_rng(seed)
    sample = np.sort(rng.choice(n, size=min(4096, n), replace=False)).astype(np.uint32)
    host = Arrays()
    for k in ("x", "y", "z", "mass", "fx", "fy", "fz"):
        setattr(host, k, getattr(arrs_dev, k).cpu().numpy())
    host.id = arrs_dev.id.cpu().numpy().view(np.uint32)
    f64 = ctx.direct_f64(host, sample)
    f32 = np.stack([host.fx[sample], host.fy[sample], host.fz[sample]], axis=1).astype(np.float64)
    rel = np.linalg.norm(f32 - f64, axis=1) / np.linalg.norm(f64, axis=1)
    return {"median_rel": float(np.median(rel)),
            "rms_rel": float(np.sqrt(((f32 - f64) ** 2).sum() / (f64 ** 2).sum())),
            "max_rel": float(rel.max())}


def run_b200(args):
    import torch
    import polesitter_b200 as P
    from polesitter_b200 import closure as CL
    from polesitter_b200.replicas import job_time

    rank, local_rank, world = dist_info()
    torch.cuda.set_device(local_rank)
    if world > 1:
        import torch.distributed as dist
        from datetime import timedelta
        dist.init_process_group("nccl", timeout=timedelta(seconds=120),
                                device_id=torch.device("cuda", local_rank))
    n = args.n
    theta = theta_of(args)
    closure = args.workload == "closure"
    p0 = particles(args.workload, n)
    dev = torch.device("cuda", local_rank)

    def device_arrays(p):
        a = Arrays()
        for k in ("x", "y", "z", "mass", "fx", "fy", "fz"):
            setattr(a, k, torch.from_numpy(getattr(p, k).copy()).to(dev))
        a.id = torch.from_numpy(p.id.view(np.int32).copy()).to(dev)
        return a

    d = device_arrays(p0)
    pristine = device_arrays(p0)
    codes = torch.zeros(n, dtype=torch.int32, device=dev)
    flush = torch.empty(256 << 20, dtype=torch.uint8, device=dev)  # > 126 MB L2

    def reset(dst=d, src=pristine):
        for k in ("x", "y", "z", "mass", "id"):
            getattr(dst, k).copy_(getattr(src, k))
        flush.fill_(1)
        torch.cuda.synchronize()

    ctx = P.Context(n, theta=theta)
    leaf_cap = leaf_cap_of(args)
    ctx.set_option(P.OPT_LEAF_CAP, leaf_cap)
    if closure:
        params, meta = CL.load(CL.default_weights_path())
        ctx.closure_set_weights(params)
        ctx.set_closure(2)
    # one untimed tick with per-node interaction counters on: the algorithmic
    # work of this workload (identical in every timed step)
    ctx.set_option(P.OPT_DEBUG, 1)
    reset()
    ctx.tick(d, codes)
    st = ctx.stats()
    tree = ctx.tree()
    leaf = tree["nchild"] == 0
    m2l_leaf = int(tree["m2l_cnt"][leaf].sum())
    m2l_all = int(st["m2l_pairs"])
    p2p_inter = int(st["p2p_interactions"])
    p2p_full = int(st["full_leaf_interactions"])
    ctx.set_option(P.OPT_DEBUG, 0)
    ctx.set_option(P.OPT_TIMING, 1)

    for _ in range(args.warmup):
        reset()
        ctx.tick(d, codes)

    step_s, phases, judge = [], [], []
    gpu_index = int(os.environ.get("CUDA_VISIBLE_DEVICES", str(local_rank)).split(",")[0]) \
        if os.environ.get("CUDA_VISIBLE_DEVICES", "").split(",")[0].isdigit() else local_rank
    if world > 1:
        torch.distributed.barrier()
    torch.cuda.synchronize()
    with ClockSampler(gpu_index) as clocks:
        time.sleep(0.5)  # let nvidia-smi start sampling before the timed steps
        for _ in range(args.steps):
            reset()
            t0 = time.perf_counter()
            ctx.tick(d, codes)  # synchronous: returns after the forces are written
            step_s.append(time.perf_counter() - t0)
            phases.append(ctx.timing())
            if closure:
                judge.append(ctx.closure_last())
        torch.cuda.synchronize()
    if world > 1:
        torch.distributed.barrier()
    total = job_time(sum(step_s), dev)
    value = world * args.steps / total
    ph = {k: statistics.mean(t[k] for t in phases) for k in phases[0]}

    accuracy = {"vs": "FP64 direct sum on the GPU, 4096 sampled particles (last timed tick)"}
    accuracy.update(median_rel_error(ctx, d, n, 7))
    if closure:
        med = [j["median_mlp"] if j["used"] else j["median_base"] for j in judge]
        accuracy["judge"] = {
            "per_tick": "the tick's own FP64 judge (1024 particles, a new sample every tick)",
            "median_of_tick_medians": float(statistics.median(med)),
            "max_of_tick_medians": float(max(med)),
            "median_without_correction": float(statistics.median(j["median_base"] for j in judge)),
            "correction_applied": f"{sum(j['used'] for j in judge)}/{len(judge)} ticks",
            "meets_target": bool(max(med) <= ERROR_TARGET)}

    # e2e: the same tick through the public API with pinned host buffers
    e2e_steps = max(1, min(args.e2e_steps, args.steps))
    pin = {k: torch.empty(n, dtype=torch.float32 if k != "id" else torch.int32,
                          pin_memory=True).numpy() for k in
           ("x", "y", "z", "mass", "fx", "fy", "fz", "id")}
    pin_codes = torch.empty(n, dtype=torch.int32, pin_memory=True).numpy().view(np.uint32)
    hp = Arrays()
    for k, v in pin.items():
        setattr(hp, k, v.view(np.uint32) if k == "id" else v)

    def reset_host():
        for k in ("x", "y", "z", "mass"):
            getattr(hp, k)[:] = getattr(p0, k)
        hp.id[:] = p0.id
        flush.fill_(1)
        torch.cuda.synchronize()

    reset_host()
    ctx.tick(hp, pin_codes)  # allocates the host-path mirrors
    e2e_s = []
    for _ in range(e2e_steps):
        reset_host()
        t0 = time.perf_counter()
        ctx.tick(hp, pin_codes)
        e2e_s.append(time.perf_counter() - t0)
    e2e_total = job_time(sum(e2e_s), dev)
    e2e = {"value": world * e2e_steps / e2e_total, "unit": UNIT,
           # prepare: x,y,z in / codes out; calc: x,y,z,mass,id,codes in /
           # x,y,z,mass,id,codes,fx,fy,fz out -- 4 bytes per particle each
           "h2d_bytes_per_step": 4 * n * (3 + 6), "d2h_bytes_per_step": 4 * n * (1 + 9),
           "steps": e2e_steps, "ms_per_step": 1000.0 * e2e_total / e2e_steps}

    peaks, peak_src = measured_peaks()
    props = torch.cuda.get_device_properties(dev)
    fp32_peak = props.multi_processor_count * 128 * 2 * float(peaks.get("sm_max_mhz", 1965.0)) * 1e6
    # the dominant phase: the leaf pass (k_trav leaf and split groups: M2L of
    # the leaf targets, P2P outside full leaves) or the full-leaf P2P
    # (k_dense_p2p: P2P + L2P of the records)
    m2l_flop = FLOP_M2L_ORDER1 if closure else FLOP_M2L
    flops_leaf = m2l_flop * m2l_leaf + FLOP_P2P * (p2p_inter - p2p_full)
    flops_full = FLOP_P2P * p2p_full
    if ph["full_leaves"] > ph["leaves"]:
        kern, launch_ms, flops = ("full-leaf P2P: k_dense_p2p (P2P + L2P of the leaf records)",
                                  ph["full_leaves"], flops_full)
        counts = {"p2p_particle_pairs": p2p_full, "flop_per_p2p": FLOP_P2P}
    else:
        kern, launch_ms, flops = ("leaf pass: k_trav<MODE_LEAF> "
                                  "(MAC+M2L+L2L+P2P+L2P)", ph["leaves"], flops_leaf)
        counts = {"m2l_pairs_leaf_targets": m2l_leaf,
                  "p2p_particle_pairs": p2p_inter - p2p_full,
                  "flop_per_m2l": m2l_flop, "flop_per_p2p": FLOP_P2P}
    achieved = flops / (launch_ms / 1e3) / 1e12
    roofline = {"kernel": kern,
                "bound": "fp32", "achieved": achieved, "peak": fp32_peak / 1e12,
                "unit": "TFLOP/s", "frac": achieved * 1e12 / fp32_peak,
                "peak_source": f"computed: {props.multi_processor_count} SMs x 128 FP32 lanes x 2 x "
                               f"{peaks.get('sm_max_mhz', 1965.0)} MHz (sm_max_mhz, {peak_src}); "
                               "no measured FP32 peak exists",
                "traffic": DOMINANT_DRAM_BYTES[args.workload],
                "traffic_note": TRAFFIC_NOTE[args.workload],
                "algorithmic_flop": flops, "counts": counts, "launch_ms": launch_ms,
                "other_phase": {"leaf_pass_ms": ph["leaves"], "leaf_pass_flop": flops_leaf,
                                "full_leaf_ms": ph["full_leaves"], "full_leaf_flop": flops_full}}

    line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": 1000.0 * total / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32",
            "data": "synthetic (seeded clumpy Plummer)" if closure
            else "synthetic (seeded Plummer sphere)",
            "config": {"workload": WORKLOADS[args.workload], "n": n, "theta": theta,
                       "leaf_cap": leaf_cap,
                       "per_gpu": "independent replica of the workload",
                       "l2": "flushed (256 MB write) and inputs reset before every step, untimed",
                       "timing": "wall clock around the synchronous API call, max over ranks"},
            "device_ms": ph,
            "interactions": {"m2l_pairs": m2l_all, "p2p_particle_pairs": p2p_inter},
            "accuracy": accuracy, "e2e": e2e, "roofline": roofline,
            "clocks": clocks.summary(),
            "gpu_launches": KERNELS_PER_TICK[args.workload] * args.steps}

    # the extra lines run on single-GPU runs only (a multi-GPU run is the
    # replica scaling measurement)
    extras = world == 1 and not args.minimal
    if closure and extras and not args.no_plain_curve:
        line["equal_error"] = equal_error(ctx, P, d, pristine, codes, flush, n, value,
                                          accuracy["judge"]["max_of_tick_medians"])
    ctx.destroy()
    if closure and extras:
        line["ensemble"] = ensemble_run(P, torch, dev)
        line["plain_c2"] = plain_c2(P, torch, dev, flush)
        line["tick_loop"] = tick_loop(P, torch, dev)
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        line["cpu_baseline"] = cpu_reference_ticks(p0, ticks=1 if closure else 3, warmup=1,
                                                   theta=theta)
    if world > 1:
        torch.distributed.barrier()
        torch.distributed.destroy_process_group()
    if rank == 0:
        print(json.dumps(line), flush=True)
    return 0


def method_curve(ctx, P, d, pristine, codes, flush, n, mode, cap, thetas):
    """One method on the closure's snapshot (mode 0: the plain GPU FMM, the
    reference's far field; mode 1: the order-1 local expansion without the
    network) at leaf capacity cap, theta up the ladder until its median
    error against the FP64 direct sum meets the target.  Its tick only gets
    slower as theta grows, so the first theta that meets the target is the
    method's fastest setting at that error."""
    import torch
    ctx.set_closure(mode)
    ctx.set_option(P.OPT_LEAF_CAP, cap)
    rows = []

    def one_tick():
        for k in ("x", "y", "z", "mass", "id"):
            getattr(d, k).copy_(getattr(pristine, k))
        flush.fill_(1)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        ctx.tick(d, codes)
        return time.perf_counter() - t0

    for th in thetas:
        ctx.set_option(P.OPT_THETA, th)
        first = one_tick()  # grows the stores (or settles the near-list depth) once
        err = median_rel_error(ctx, d, n, 11)
        met = err["median_rel"] <= ERROR_TARGET
        # the setting that meets the target is timed over more ticks
        ts = [one_tick() for _ in range(3 if met else 1)]
        st = ctx.stats()
        rows.append({"theta": th, "leaf_cap": cap, "ticks_per_s": 1.0 / min(ts),
                     "first_tick_s": first, "median_rel_error": err["median_rel"],
                     "rms_rel_error": err["rms_rel"], "max_rel_error": err["max_rel"],
                     "near_levels": st["near_levels"], "p2p_streamed": bool(st["streamed"])})
        if met:
            break
    at = rows[-1] if rows and rows[-1]["median_rel_error"] <= ERROR_TARGET else None
    return rows, at


def equal_error(ctx, P, d, pristine, codes, flush, n, closure_value, closure_error):
    """The metric itself: ticks/s of each method at the closure's error
    bound (median relative force error <= 1e-3 against the FP64 direct sum),
    on the same 1M snapshot.  The plain GPU FMM is tried on the reference's
    tree and on larger leaves; the order-1 expansion without the network
    (closure mode 1) shows what the network itself buys."""
    ctx.set_option(P.OPT_TIMING, 1)
    out = {"target_median_rel_error": ERROR_TARGET,
           "closure": {"theta": CLOSURE_THETA, "leaf_cap": CLOSURE_LEAF_CAP,
                       "ticks_per_s": closure_value,
                       "max_tick_median_rel_error": closure_error}}
    plain_rows, plain_at = [], []
    for cap, thetas in PLAIN_LADDERS:
        rows, at = method_curve(ctx, P, d, pristine, codes, flush, n, 0, cap, thetas)
        plain_rows += rows
        if at:
            plain_at.append(at)
    m1_rows, m1_at_all = [], []
    for cap, thetas in MODE1_LADDERS:
        rows, at = method_curve(ctx, P, d, pristine, codes, flush, n, 1, cap, thetas)
        m1_rows += rows
        if at:
            m1_at_all.append(at)
    m1_at = max(m1_at_all, key=lambda r: r["ticks_per_s"]) if m1_at_all else None
    best_plain = max(plain_at, key=lambda r: r["ticks_per_s"]) if plain_at else None
    out["plain_gpu_fmm"] = plain_rows
    out["plain_reaches_target"] = bool(plain_at)
    out["plain_at_target"] = best_plain
    out["order1_without_network"] = m1_rows
    out["order1_at_target"] = m1_at
    out["closure_vs_plain"] = (closure_value / best_plain["ticks_per_s"]) if best_plain else None
    out["closure_vs_order1"] = (closure_value / m1_at["ticks_per_s"]) if m1_at else None
    out["note"] = ("each method's ticks/s at the first theta of its ladder whose median error "
                   "meets the target (its tick only gets slower as theta grows); "
                   "closure_vs_plain is the metric, closure_vs_order1 what the trained network "
                   "itself buys")
    return out


def plain_c2(P, torch, dev, flush):
    """The plain tick on the parity configuration (Plummer N=1M, theta=2)."""
    from polesitter_b200 import workloads as W
    p = W.plummer(1 << 20, C2_SEED)
    a = Arrays()
    for k in ("x", "y", "z", "mass", "fx", "fy", "fz"):
        setattr(a, k, torch.from_numpy(getattr(p, k).copy()).to(dev))
    a.id = torch.from_numpy(p.id.view(np.int32).copy()).to(dev)
    codes = torch.zeros(p.n, dtype=torch.int32, device=dev)
    src = {k: getattr(a, k).clone() for k in ("x", "y", "z", "mass", "id")}
    ts = []
    with P.Context(p.n, theta=C2_THETA) as ctx:
        for i in range(23):
            for k, v in src.items():
                getattr(a, k).copy_(v)
            flush.fill_(1)
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            ctx.tick(a, codes)
            if i >= 3:
                ts.append(time.perf_counter() - t0)
        err = median_rel_error(ctx, a, p.n, 13)
    return {"workload": WORKLOADS["plain"], "ticks_per_s": len(ts) / sum(ts), "steps": len(ts),
            "warmup": 3, "accuracy": dict(vs="FP64 direct sum on the GPU, 4096 sampled "
                                             "particles (last tick)", **err)}


def tick_loop(P, torch, dev):
    """The device-resident tick loop on two colliding Plummer spheres
    (N=4,194,304, mass ratio 3:1, 20a apart, 0.3 relative velocity, theta=2):
    100 ticks of semi-implicit Euler, dt=1e-3 (ps_b200_run_ticks)."""
    from polesitter_b200 import workloads as W
    n, ticks = 1 << 22, 100
    p, vx, vy, vz = W.two_plummer(n, 1)
    a = Arrays()
    for k in ("x", "y", "z", "mass", "fx", "fy", "fz"):
        setattr(a, k, torch.from_numpy(getattr(p, k).copy()).to(dev))
    a.id = torch.from_numpy(p.id.view(np.int32).copy()).to(dev)
    v = [torch.from_numpy(x.astype(np.float32)).to(dev) for x in (vx, vy, vz)]
    codes = torch.zeros(n, dtype=torch.int32, device=dev)
    with P.Context(n, theta=2.0) as ctx:
        ctx.run_ticks(a, codes, *v, 1e-3, 2)  # warm-up: grows the stores
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        ctx.run_ticks(a, codes, *v, 1e-3, ticks)
        torch.cuda.synchronize()
        dt = time.perf_counter() - t0
        # the forces of the last tick, on the positions it saw: the arrays
        # hold the positions after its Euler step, so recompute that tick's
        # forces with one more prepare + calc of the same positions
        ctx.tick(a, codes)
        err = median_rel_error(ctx, a, n, 17)
    return {"workload": "two colliding Plummer spheres, N=4,194,304 (3:1), theta=2, "
                        "100 ticks of semi-implicit Euler dt=1e-3 on the device "
                        "(ps_b200_run_ticks)",
            "ticks_per_s": ticks / dt, "particle_ticks_per_s": n * ticks / dt,
            "accuracy": dict(vs="FP64 direct sum on the GPU, 4096 sampled particles, forces "
                                "of one more tick on the final state", **err)}


def ensemble_run(P, torch, dev):
    """The batched ensemble: 256 independent systems, N log-uniform in
    [1024, 262144], half uniform cubes and half Plummer spheres (a in
    [0.5, 2]); theta and leaf capacity (from {1, 16, 32, 64}) per size class,
    the expansion order (0 or 1) and the traversal grid scale from the
    autotuner (target median force error 3e-2); 50 ticks of semi-implicit
    Euler, dt=1e-3, each tick two replayed CUDA graphs of one launch per phase
    over all systems.  Beside it, the same systems advanced one after the
    other through ps_b200_run_ticks."""
    from polesitter_b200 import workloads as W
    # the workload names no accuracy; 3e-2 is half the median error of the
    # reference's own setting (theta 2, leaf capacity 1: 6.2e-2 on the 1M
    # Plummer sphere), so every tuned system is at least that accurate
    nsys, ticks, target = 256, 50, 3e-2
    counts, p, vx, vy, vz = W.ensemble(nsys, 2026)

    def arrays():
        a = Arrays()
        for k in ("x", "y", "z", "mass", "fx", "fy", "fz"):
            setattr(a, k, torch.from_numpy(getattr(p, k).copy()).to(dev))
        a.id = torch.from_numpy(p.id.view(np.int32).copy()).to(dev)
        return a, [torch.from_numpy(x.copy()).to(dev) for x in (vx, vy, vz)]

    a, v = arrays()
    codes = torch.zeros(p.n, dtype=torch.int32, device=dev)
    with P.Ensemble(counts) as ens:
        theta, scale = ens.autotune(a, codes, target)
        caps = ens.leaf_caps()
        order = ens.order()
        ens.run(a, codes, *v, 1e-3, 2)  # warm-up: captures the graphs, grows stores
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        ens.run(a, codes, *v, 1e-3, ticks)
        torch.cuda.synchronize()
        dt = time.perf_counter() - t0
    offs = np.concatenate([[0], np.cumsum(counts)])
    # FP64 errors of the last tick's forces: the first system of each size
    # class (floor(log2 N)); the ensemble's arrays hold the positions after
    # that tick's Euler step, so those systems are ticked once more as they are
    cls = np.floor(np.log2(np.asarray(counts, np.float64) + 1)).astype(int)
    per_class = {}
    for c in sorted(set(cls.tolist())):
        k = int(np.argmax(cls == c))
        lo, hi = int(offs[k]), int(offs[k + 1])
        s = Arrays()
        for key in ("x", "y", "z", "mass", "fx", "fy", "fz", "id"):
            setattr(s, key, getattr(a, key)[lo:hi].clone())
        with P.Context(hi - lo, theta=float(theta[k])) as ectx:
            ectx.set_option(P.OPT_LEAF_CAP, int(caps[k]))
            if order:
                ectx.set_closure(order)
            s.id.copy_(torch.arange(hi - lo, dtype=torch.int32, device=dev))
            ectx.tick(s, codes[lo:hi])
            e = median_rel_error(ectx, s, hi - lo, 19 + c)
        per_class[str(c)] = dict(system=k, n=hi - lo, theta=float(theta[k]),
                                 leaf_cap=int(caps[k]), **e)
    # the same systems one after the other, without graphs
    b, w = arrays()
    ctxs = [P.Context(int(counts[k]), theta=float(theta[k])) for k in range(nsys)]
    for k in range(nsys):
        ctxs[k].set_option(P.OPT_LEAF_CAP, int(caps[k]))
        if order:
            ctxs[k].set_closure(order)

    def one_pass():
        for k in range(nsys):
            lo, hi = int(offs[k]), int(offs[k + 1])
            s = Arrays()
            for key in ("x", "y", "z", "mass", "fx", "fy", "fz", "id"):
                setattr(s, key, getattr(b, key)[lo:hi])
            ctxs[k].run_ticks(s, codes[lo:hi], *(x[lo:hi] for x in w), 1e-3, 1)

    one_pass()
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for _ in range(3):
        one_pass()
    torch.cuda.synchronize()
    seq = 3 / (time.perf_counter() - t0)
    for c in ctxs:
        c.destroy()
    vals, cnts = np.unique(theta, return_counts=True)
    cvals, ccnts = np.unique(caps, return_counts=True)
    return {"workload": "256 independent systems, N log-uniform in [1024, 262144] "
                        f"({int(p.n)} particles), half uniform cubes, half Plummer a in "
                        "[0.5, 2]; 50 ticks of Euler dt=1e-3",
            "ensemble_ticks_per_s": ticks / dt, "particle_ticks_per_s": p.n * ticks / dt,
            "autotuner": {"target_median_rel_error": target,
                          "theta_per_class": {str(float(t)): int(c) for t, c in zip(vals, cnts)},
                          "leaf_cap_per_class": {str(int(t)): int(c)
                                                 for t, c in zip(cvals, ccnts)},
                          "grid_scale": scale,
                          "expansion_order": order},
            "accuracy_per_size_class": per_class,
            "one_system_at_a_time_ticks_per_s": seq,
            "speedup_over_one_at_a_time": (ticks / dt) / seq}


def main():
    args = parse_args()
    if args.minimal:
        args.no_plain_curve = args.no_cpu_baseline = True
        args.e2e_steps = 1
    if args.impl == "reference":
        return run_reference(args)
    return run_b200(args)


if __name__ == "__main__":
    sys.exit(main())
