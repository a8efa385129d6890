#!/usr/bin/env python
"""Induced-velocity (Biot-Savart) benchmark on the large helical wake.

Workload (one step = one full evaluation): 3 blades x 41 cosine-spaced nodes x
720 wake steps at 1 deg (two revolutions), every shed and trailing filament
(175,080) onto every wake node and lifting-line point (88,803), Vatistas n=2
core, FP32-compensated arithmetic with FP64 near-singular terms. Synthetic,
seeded inputs (no dataset). Metric: Gint/s (1e9 target-filament interactions
per second), whole job over all ranks.

``python bench.py [--gpus N --steps K --warmup W]`` -- this engine.
``python bench.py --impl reference``                 -- the reference's CPU
  formula (the C restatement of core/BiotSavart.m, all host threads) on a
  bounded sample of the same workload.
For N > 1 (torchrun) each rank evaluates its own wake (seed + rank): weak
scaling, no data-path collective; the time is the max over ranks. Beside that
line, at N > 1: the 64-case batch split by case (``wake_batch_sharded``) and
one wake's evaluation split by target with an NCCL all-gather of the
velocities (``target_sharded``, strong scaling).
"""
from __future__ import annotations

import argparse
import ctypes as C
import importlib
import json
import os
import statistics
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)
# FLOP per target-filament interaction of the Vatistas n=2 kernel, FMA = 2:
# r1, r2 (6), |r1|^2, |r2|^2 (10), r1.r2 (5), r1 x r2 (9), |r1||r2| and the
# denominator (3), numerator (2), L.r1 and h^2 (8), the Vatistas factor (3),
# scale (1), accumulate (6); rsqrt/rcp are counted apart (3 per interaction)
FLOP_PER_INTERACTION = 52
# the cut-off core's count: the d |L|^2 denominator term in place of h^2 and
# the Vatistas factor
FLOP_PER_INTERACTION_CUTOFF = 44
METRIC = "biot_savart_gint_per_s"
UNIT = "Gint/s"


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=40)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--no-fp64", action="store_true", help="skip the plain FP64 comparison")
    ap.add_argument("--workload", default="large", choices=["large", "medium"],
                    help="large: 3x41x720 (the metric's case); medium: 3x41x180 for profiling")
    ap.add_argument("--tiling", default=None,
                    help="force the FP32 tiling 'T,KF,waves' instead of the autotuner's choice")
    ap.add_argument("--layout", default=None, choices=["input", "chained"],
                    help="with --tiling: the filament stream layout (default: input order)")
    ap.add_argument("--core", default="vatistas", choices=["vatistas", "cutoff"],
                    help="profiling aid: the timed loop's core (cutoff: d = 1e-4); the metric's "
                         "case is vatistas")
    ap.add_argument("--wake-steps", type=int, default=10,
                    help="timed pcc steps of the 64-case batched wake (0: skip)")
    ap.add_argument("--quick", action="store_true",
                    help="timed loop only (no FP64 comparison, e2e, CPU baseline or studies)")
    ap.add_argument("--no-studies", action="store_true",
                    help="skip the start-value study and the end-to-end run")
    ap.add_argument("--e2e-steps", type=int, default=20,
                    help="pcc steps of the 16-case end-to-end run (each path)")
    ap.add_argument("--wake-only", action="store_true",
                    help="profiling aid: only the 64-case batched wake (fast path, default "
                         "tiling, no FP64 comparison); prints its sub-object")
    return ap.parse_args()


# ------------------------------------------------------------------ clocks
class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled every 200 ms."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index):
        self.idx = str(gpu_index)
        self.rows = []
        self.proc = None
        self.mark = 0

    def start(self, wait_s=5.0):
        """Starts sampling and waits until the first sample arrives."""
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits", "-lms", "100"],
                stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        except OSError:
            self.proc = None
            return
        self.th = threading.Thread(target=self._read, daemon=True)
        self.th.start()
        t0 = time.time()
        while not self.rows and time.time() - t0 < wait_s and self.proc.poll() is None:
            time.sleep(0.02)

    def begin(self):
        """Marks the start of the timed region (samples before it are dropped)."""
        self.mark = len(self.rows)

    def _read(self):
        self.errors = []
        for line in self.proc.stdout:
            parts = [p.strip() for p in line.split(",")]
            if len(parts) >= 9 and parts[0] == self.idx:
                self.rows.append(parts)
            elif len(self.errors) < 3:
                self.errors.append(line.strip())

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        rows = self.rows[self.mark:] or self.rows[-1:]
        sm = [float(r[1]) for r in rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in rows if r[2].replace(".", "").isdigit()]
        reasons = sorted({names[k] for r in rows for k in range(4) if r[5 + k].lower() == "active"})
        out = {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
               "reasons": reasons, "samples": len(self.rows) - self.mark}
        if not self.rows and getattr(self, "errors", None):
            out["error"] = " | ".join(self.errors)
        return out


# ------------------------------------------------------------------ workload
def workload(seed, kind="large"):
    synth = importlib.import_module("winds-master_b200.synth")
    case = synth.large_case(seed=seed)
    if kind == "medium":
        case.nsteps = 180
    w = synth.make_wake(case)
    fams = [synth.shed_filaments(w["dom"]) + (w["gamma_shed"], w["rc_shed"]),
            synth.trail_filaments(w["dom"]) + (w["gamma_trail"], w["rc_trail"])]
    pts = np.concatenate([synth.flat_points(w["dom"]), synth.flat_points(w["ll"])])
    P = np.asfortranarray(pts.reshape(-1, 3, 1, 1))
    nf = sum(f[0].shape[0] * f[0].shape[2] * f[0].shape[3] for f in fams)
    return w, fams, P, nf, P.shape[0]


def bench_config(kind, nt, nf, world):
    """The workload description both arms print (the same dict on both)."""
    return {"workload": f"helical wake 3x41x{720 if kind == 'large' else 180} (1 deg), Vatistas n=2, "
            "all shed+trailing filaments onto all wake nodes + lifting-line points",
            "targets": nt, "filaments": nf, "interactions_per_step": nt * nf,
            "l2": "256 MB buffer written between timed steps (GPU arm)",
            "parallelism": f"replicated wakes x{world}" if world > 1 else "single GPU"}


def profiled_traffic(interactions, chained=False):
    """DRAM bytes per launch of bs_f32c from the committed ncu summary of its
    stream layout (dram__bytes_read.sum + dram__bytes_write.sum of one
    captured launch), scaled to this launch by interactions; None without a
    summary."""
    path = os.path.join(ROOT, "profiles",
                        "bs_f32c_large_chained.md" if chained else "bs_f32c_large.md")
    if not os.path.exists(path):
        return None
    for line in open(path):
        if line.startswith("traffic_bytes_per_launch:"):
            b, n = line.split(":", 1)[1].split()[:2]
            return float(b) * interactions / float(n)
    return None


def cpu_rate(fams, P, n_targets, seed=0):
    """C oracle (FP64 restatement of BiotSavart.m, OpenMP on all host threads)
    over n_targets sampled targets x all filaments; returns (Gint/s, seconds)."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as orc
    rng = np.random.default_rng(seed)
    idx = rng.choice(P.shape[0], n_targets, replace=False)
    Ps = np.asfortranarray(P[idx])
    nf = sum(f[0].shape[0] * f[0].shape[2] * f[0].shape[3] for f in fams)
    t0 = time.perf_counter()
    for F1, F2, g, rc in fams:
        orc.c_eval(F1, F2, Ps, g, rc, "visc2", 1000.0, nthreads=os.cpu_count())
    dt = time.perf_counter() - t0
    return n_targets * nf / dt / 1e9, dt


def other_cpu_baselines(fams, P, seed=3):
    """The two other host paths, each on a small seeded target sample x all
    filaments: the NumPy restatement of core/BiotSavart.m (vectorised over
    filaments per target block, one process) and, when it was built, the
    reference MEX's own serial host loop (cuda/source/BiotSavartMex.cu:268-282;
    cut-off core only, so it runs the cut-off form d = 1e-4 on the same
    geometry). Gint/s each; a reported baseline, not a target."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import biot_savart_ref as bsr
    import oracle as orc
    rng = np.random.default_rng(seed)
    nf = sum(f[0].shape[0] * f[0].shape[2] * f[0].shape[3] for f in fams)
    out = {}
    idx = rng.choice(P.shape[0], 48, replace=False)
    pts = np.ascontiguousarray(P[idx, :, 0, 0])
    flat = []
    for F1, F2, g, rc in fams:
        m = lambda a: np.moveaxis(a, 1, -1).reshape(-1, a.shape[1], order="F")
        flat.append((m(F1), m(F2), g.ravel(order="F"), rc.ravel(order="F")))
    t0 = time.perf_counter()
    for x1, x2, g, rc in flat:
        bsr.biot_savart_flat(x1, x2, g, rc, pts, "visc2", 1000.0)
    dt = time.perf_counter() - t0
    out["numpy_port"] = {"value": len(idx) * nf / dt / 1e9, "unit": UNIT, "cores": 1,
                         "sample": f"{len(idx)} sampled targets x {nf} filaments ({dt:.1f} s), NumPy "
                                   "restatement of core/BiotSavart.m, Vatistas n=2"}
    if orc.ref_available():
        idx = rng.choice(P.shape[0], 256, replace=False)
        Ps = np.asfortranarray(P[idx])
        t0 = time.perf_counter()
        for F1, F2, g, rc in fams:
            orc.ref_host_eval(F1, F2, Ps, g, rc, 1e-4, 1000.0)
        dt = time.perf_counter() - t0
        out["reference_mex_host"] = {
            "value": len(idx) * nf / dt / 1e9, "unit": UNIT, "cores": 1,
            "sample": f"{len(idx)} sampled targets x {nf} filaments ({dt:.1f} s), the reference "
                      "MEX host loop compiled from its source, cut-off core d=1e-4"}
    return out


def reference_arm(args):
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    _, fams, P, nf, nt = workload(1, args.workload)
    cores = os.cpu_count()
    # size one step to about 3 s of CPU work
    rate, _ = cpu_rate(fams, P, 16)
    n = int(max(16, min(nt, 3.0 * rate * 1e9 / nf)))
    for i in range(args.warmup):
        cpu_rate(fams, P, max(16, n // 8), seed=100 + i)
    total_t, total_int = 0.0, 0
    for i in range(args.steps):
        r, dt = cpu_rate(fams, P, n, seed=i)
        total_t += dt
        total_int += n * nf
    value = total_int / total_t / 1e9
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * total_t / args.steps,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
        "data": "synthetic",
        "config": bench_config(args.workload, nt, nf, int(os.environ.get("WORLD_SIZE", "1"))),
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": cores, "kind": "port",
                         "sample": f"{n} sampled targets x {nf} filaments per step"},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "note": "oracle/_ref (the reference MEX host loop) implements only the cut-off core, so "
                "the Vatistas workload runs on the FP64 C restatement of core/BiotSavart.m",
    }
    print(json.dumps(line), flush=True)


# ------------------------------------------------------------------ batched wake
def timed_steps(b, n, graph):
    """Steps ``b`` n times; mean device ms per step (CUDA events per call)."""
    ms = []
    for _ in range(n):
        b.step(1, graph=graph)
        ms.append(b.stats()[0])
    return statistics.mean(ms)


def wake_bench(args, seed=2, ncases=64, plain=True, mlp=None):
    """64 uneven rotor cases (wake steps 60-720, span nodes 17-41, U 5-25 m/s,
    TSR 4-10, yaw 0-30 deg, shear 0-0.3), pcc predictor-corrector step. Three
    paths: the FP32-compensated batch replaying one CUDA graph per step (the
    product), the same batch in FP64 (batching and graphs without the FP32
    direct sum), and the plain FP64 path (each case on its own, eager, FP64).
    plain / batched FP64 is the batching-and-graph gain, batched FP64 / fast
    the FP32c gain."""
    synth = importlib.import_module("winds-master_b200.synth")
    wake = importlib.import_module("winds-master_b200.wake")
    rcases = synth.batch_cases(ncases, seed=seed)
    warm, n_fast, n_b64 = 1, args.wake_steps, 3
    cases = [synth.make_wake_case(rc, nsteps=warm + max(n_fast, n_b64) + 3, jitter=0.05)
             for rc in rcases]
    b = wake.WakeBatch(cases, integrator="pcc", precision="f32c")
    b.step(warm, graph=True)
    ms = timed_steps(b, n_fast, True)
    _, inter, launches = b.stats()
    b.close()
    nodes = int(sum(c["nst"] * c["na"] * c["nb"] for c in cases))
    if not plain:
        return {"cases": ncases, "integrator": "pcc", "graph": True, "steps_per_s": 1000.0 / ms,
                "ms_per_step": ms, "launches_per_step": launches, "nodes": nodes}
    b64 = wake.WakeBatch(cases, integrator="pcc", precision="f64")
    b64.step(warm, graph=True)
    ms64 = timed_steps(b64, n_b64, True)
    b64.close()
    plain_ms = 0.0
    for c in cases:
        p = wake.WakeBatch([c], integrator="pcc", precision="f64")
        p.step(1)
        p.step(1)
        plain_ms += p.stats()[0]
        p.close()
    return {"cases": ncases, "integrator": "pcc", "graph": True, "timed_steps": n_fast,
            "steps_per_s": 1000.0 / ms, "ms_per_step": ms,
            "interactions_per_step": inter, "gint_per_s": inter / (ms * 1e-3) / 1e9,
            "launches_per_step": launches,
            "batched_fp64_steps_per_s": 1000.0 / ms64, "batched_fp64_timed_steps": n_b64,
            "plain_fp64_steps_per_s": 1000.0 / plain_ms,
            "speedup_vs_plain_fp64": plain_ms / ms,
            "gain_batching_and_graphs": plain_ms / ms64, "gain_fp32c_over_fp64": ms64 / ms,
            "nodes": nodes,
            "lifting_line": wake_kj_bench(rcases, cases, mlp=mlp)}


def sharded_wake_bench(args, rank, world, seed=2, ncases=64):
    """The 64-case batch split over the ranks by case (sharding.ShardedRun):
    each rank steps the batch of its own cases with graph replay, with no
    collective on the data path; per-case values are gathered on the host
    after every step. The batch's step time is the slowest rank's (CUDA
    events around each rank's steps, max over ranks)."""
    import torch
    import torch.distributed as dist
    synth = importlib.import_module("winds-master_b200.synth")
    sh = importlib.import_module("winds-master_b200.sharding")
    rcases = synth.batch_cases(ncases, seed=seed)
    cases = [synth.make_wake_case(rc, nsteps=1 + args.wake_steps + 3, jitter=0.05) for rc in rcases]
    run = sh.ShardedRun(cases, rank=rank, world=world, integrator="pcc", precision="f32c")
    run.step(1)  # capture
    ms = 0.0
    for _ in range(args.wake_steps):
        run.step(1)
        ms += run.local.step_ms() if run.local is not None else 0.0
    parts = run.parts
    run.close()
    t = torch.tensor([ms], device="cuda", dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    costs = [sh.case_cost(c) for c in cases]
    return {"cases": ncases, "ranks": world, "parallelism": "case-sharded", "integrator": "pcc",
            "graph": True, "timed_steps": args.wake_steps,
            "steps_per_s": 1000.0 * args.wake_steps / float(t.item()),
            "cases_per_rank": [len(p) for p in parts], "imbalance": sh.imbalance(costs, parts),
            "timing": "CUDA events around each rank's steps, max over ranks"}


def target_sharded_bench(args, rank, world, stream, flush):
    """The headline evaluation of ONE wake (seed 1 on every rank) split over
    the ranks by target (sharding.TargetShardedEval): each rank evaluates its
    run of targets against all filaments, and one NCCL all-gather of the
    velocities (24 bytes per target) gives every rank the whole field. Strong
    scaling: one evaluation per step whatever the number of ranks. CUDA events
    around each step on the stream the ranks launch on, max over ranks; rank
    0 checks the gathered field against its own evaluation of all targets."""
    import torch
    import torch.distributed as dist
    wb = importlib.import_module("winds-master_b200")
    sh = importlib.import_module("winds-master_b200.sharding")
    _, fams, P, nf, nt = workload(1, args.workload)

    def dev(a):
        return torch.from_numpy(np.asarray(a).ravel(order="F").copy()).cuda()

    dfams = [(dev(F1), dev(F2), dev(g), dev(rc), F1.shape) for F1, F2, g, rc in fams]
    dP = dev(P)
    sp = stream.cuda_stream
    core = wb.bs.CORE_VATISTAS
    ev = sh.device_evaluator(dfams, core, 2.0, 1000.0, "f32c", stream=sp)
    te = sh.TargetShardedEval(P.shape, rank=rank, world=world)
    out = torch.zeros(P.size, dtype=torch.float64, device="cuda")
    for _ in range(3):  # warm-up (the first call tunes the run's size bucket)
        te(dP, out, ev)
    torch.cuda.synchronize()
    dist.barrier()
    ms = 0.0
    for _ in range(args.steps):
        flush.zero_()
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        te(dP, out, ev)
        e1.record(stream)
        torch.cuda.synchronize()
        ms += e0.elapsed_time(e1)
    t = torch.tensor([ms], device="cuda", dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    ms = float(t.item())
    err = None
    if rank == 0:
        full = torch.zeros_like(out)
        wb.eval_device(dfams, (dP, P.shape), core, 2.0, 1000.0, full, "f32c", stream=sp)
        wb.sync(sp)
        a = out.cpu().numpy().reshape(P.shape, order="F")
        b = full.cpu().numpy().reshape(P.shape, order="F")
        a = np.stack([a[:, c].ravel(order="F") for c in range(3)], 1)
        b = np.stack([b[:, c].ravel(order="F") for c in range(3)], 1)
        err = float(np.max(np.linalg.norm(a - b, axis=1) / np.linalg.norm(b, axis=1)))
    return {"parallelism": "target-sharded", "ranks": world, "scaling": "strong",
            "targets": nt, "filaments": nf, "timed_steps": args.steps,
            "targets_per_rank": [t1 - t0 for t0, t1 in te.slices],
            "gint_per_s": nf * nt * args.steps / (ms * 1e-3) / 1e9,
            "ms_per_step": ms / args.steps,
            "exchange_bytes_per_rank": 3 * 8 * te.n_max * world,
            "rel_diff_max_vs_one_rank": err,
            "timing": "CUDA events around each step (own run + all-gather), max over ranks"}


def batch_start_value(seed=12, n_train=48, n_val=8, steps=10, relax=0.3, tol=1e-6, maxiter=200):
    """A start-value network for the 64-case mix: pairs from the plain solver
    on other draws of the same case distribution (batch_cases, no root
    cylinders); of a network on the previous-step base and one on the
    extrapolated base, each with its output scale chosen on validation draws,
    the one that saves more iterations there."""
    synth = importlib.import_module("winds-master_b200.synth")
    gi = importlib.import_module("winds-master_b200.gamma_init")
    kw = dict(relax=relax, tol=tol, maxiter=maxiter, root_cut=0.0)
    pts = [gi.OperatingPoint(rc, 0.0) for rc in synth.batch_cases(n_train + n_val, seed=seed)]
    tr = gi.run(pts[:n_train], steps, record=True, **kw)
    keep = (tr["step_case"][:, 0] >= 4) & tr["lift"]
    return gi.fit_start_value(tr["X"][keep], tr["dG"][keep], pts[n_train:], steps, **kw)


def wake_kj_bench(rcases, cases, tol=1e-6, relax=0.3, maxiter=200, warm=3, timed=3, mlp=None):
    """The 64-case batch with the lifting line and rotor loads: every pcc step
    runs the Kutta-Joukowski fixed point to the same tolerance on every path.
    Fast: FP32c, one CUDA graph per step (the iteration one of its launches),
    started from the previous step's circulation (the reference), from its
    extrapolation alone, and from the extrapolation plus the network (when
    given). Host loop: the same FP32c batch launched kernel by kernel, the
    lifting line's flags read before the commit. Plain: each case alone, FP64, eager.
    ``warm`` untimed steps, then ``timed`` steps; iterations are summed over
    the timed steps and split by case subset: converged on both the fast and
    the plain path at every timed step, and the rest (stations past the
    synthetic polar's stall, whose relaxed iteration does not settle)."""
    synth = importlib.import_module("winds-master_b200.synth")
    wake = importlib.import_module("winds-master_b200.wake")
    gi = importlib.import_module("winds-master_b200.gamma_init")
    kjs = [synth.make_kj_case(rc, nsteps=c["nsteps"], t0=c["t0"]) for rc, c in zip(rcases, cases)]
    n = len(cases)

    def run(prec, graph, net=None, one=None, ll_fp64=False):
        sel = range(n) if one is None else [one]
        b = wake.WakeBatch([cases[k] for k in sel], integrator="pcc", precision=prec)
        b.set_kj([kjs[k] for k in sel], relax=relax, tol=tol, maxiter=maxiter, ll_fp64=ll_fp64)
        if net is not None:
            b.set_mlp(net)
        for _ in range(warm):
            b.step(1, graph=graph)
        its, ms, evals = 0, 0.0, 0
        capped = np.zeros(len(sel), dtype=bool)
        for _ in range(timed):
            b.step(1, graph=graph)
            ms += b.stats()[0]
            it, _, ev = b.kj_stats()
            its = its + it.astype(np.int64)
            capped |= it >= maxiter
            evals += ev
        out = dict(ms=ms / timed, iters=its, evals=evals, capped=capped, T=b.loads()[0].copy(),
                   G=[b.bound(k) for k in range(len(sel))])
        b.close()
        return out

    fast = run("f32c", True)
    host = run("f32c", False)
    fast_ll64 = run("f32c", True, ll_fp64=True)
    plain = dict(ms=0.0, iters=[], T=[], G=[], capped=[])
    for k in range(n):
        r = run("f64", False, one=k)
        plain["ms"] += r["ms"]
        plain["iters"].append(int(r["iters"][0]))
        plain["T"].append(float(r["T"][0]))
        plain["G"].append(r["G"][0])
        plain["capped"].append(bool(r["capped"][0]))
    it_f, it_p = fast["iters"], np.array(plain["iters"])
    # cases whose every timed step converged on both paths
    conv = ~fast["capped"] & ~np.array(plain["capped"])
    dT = np.abs(fast["T"] - np.array(plain["T"])) / np.abs(np.array(plain["T"]))
    dG = np.array([float(np.abs(gf - gp).max() / np.abs(gp).max()) for gf, gp in zip(fast["G"], plain["G"])])
    out = {"tol": tol, "relax": relax, "maxiter": maxiter, "warm_steps": warm, "timed_steps": timed,
           "steps_per_s": 1000.0 / fast["ms"], "ms_per_step": fast["ms"],
           "host_loop_steps_per_s": 1000.0 / host["ms"],
           "plain_fp64_steps_per_s": 1000.0 / plain["ms"], "speedup_vs_plain_fp64": plain["ms"] / fast["ms"],
           "kj_iterations_fast": int(it_f.sum()), "kj_iterations_plain": int(it_p.sum()),
           "converged_cases": int(conv.sum()), "stalled_cases": int((~conv).sum()),
           "converged_subset": {
               "kj_iterations_fast": int(it_f[conv].sum()), "kj_iterations_plain": int(it_p[conv].sum()),
               "iterations_ratio_fast_over_plain": float(it_f[conv].sum() / max(it_p[conv].sum(), 1)),
               "cases_iterations_equal": int((it_f[conv] == it_p[conv]).sum()),
               "thrust_rel_diff_max": float(dT[conv].max()) if conv.any() else None,
               "bound_rel_diff_max": float(dG[conv].max()) if conv.any() else None},
           "stalled_subset": {"kj_iterations_fast": int(it_f[~conv].sum()),
                              "kj_iterations_plain": int(it_p[~conv].sum())},
           # the same FP32c batch with the lifting-line evaluations in FP64
           "fast_lifting_line_fp64": {
               "steps_per_s": 1000.0 / fast_ll64["ms"],
               "kj_iterations_converged_subset": int(fast_ll64["iters"][conv].sum()),
               "iterations_ratio_over_plain": float(fast_ll64["iters"][conv].sum()
                                                    / max(it_p[conv].sum(), 1)),
               "cases_iterations_equal_plain": int((fast_ll64["iters"][conv] == it_p[conv]).sum())}}
    # start-value arms on the fast path
    arms = {"previous": fast}
    xo = gi.extrapolation_only()
    arms["extrapolated"] = run("f32c", True, net=xo)
    xo.close()
    if mlp is not None:
        arms["network"] = run("f32c", True, net=mlp)
    ref = arms["previous"]
    out["start_value_arms"] = {}
    for name, r in arms.items():
        ok = conv & ~r["capped"]
        dTa = np.abs(r["T"] - ref["T"]) / np.abs(ref["T"])
        out["start_value_arms"][name] = {
            "kj_iterations_converged_subset": int(r["iters"][conv].sum()),
            "lifting_line_evaluations": int(r["evals"]), "steps_per_s": 1000.0 / r["ms"],
            "thrust_rel_diff_vs_previous_max": float(dTa[ok].max()) if ok.any() else None}
    if mlp is not None:
        out["start_value_arms"]["network"].update(
            {"base": mlp.base, "output_shrink": mlp.shrink,
             "bases_tried": getattr(mlp, "bases_tried", None)})
    return out


# ------------------------------------------------------------------ start value
def kj_mlp_bench():
    """Learned Kutta-Joukowski start value: pairs from the plain solver on the
    attached-flow points among 800 seeded operating points (U 5-25 m/s, pitch
    0-15 deg, yaw 0-30 deg, TSR 5-9, 10 deg steps), trained on the GPU, then
    the iteration from the previous step's circulation, from its
    extrapolation alone and from the network on held-out points at tol 1e-6,
    and the converged results of the starts at tol 1e-6 and 1e-10."""
    gi = importlib.import_module("winds-master_b200.gamma_init")
    r = gi.study(n_train=800, n_test=120, epochs=60)
    r.pop("model").close()

    def rnd(v):
        if isinstance(v, float):
            return float(f"{v:.6g}")
        if isinstance(v, dict):
            return {k: rnd(x) for k, x in v.items()}
        return v
    return rnd(r)


# ------------------------------------------------------------------ end to end
def e2e_run_bench(steps, ncases=16, ages=1440, seed=5, plain_cases=2):
    """16 rotor cases, 3 blades x 41 nodes, wake truncated at 1440 steps of
    1 deg, U = 11.4 m/s, shear 0.2, yaw 0-30 deg, pcc with the lifting-line
    iteration (tol 1e-6) and rotor loads every step, ``steps`` steps per path.
    Fast: the FP32-compensated batch with graph replay, started from the
    network (previous-step base, trained here on plain-solver pairs of the
    same conditions with 120-step wakes, its output scale chosen on
    validation runs that must keep the reference start's fixed point; the
    start applies only at stations inside their polar's stall bounds), from
    the previous step's circulation, and from its extrapolation alone.
    Plain FP64 (FP64 direct sum, previous-step start, each case alone, no
    graphs) runs ``plain_cases`` of the 16 cases (every 16/plain_cases-th:
    the same size as every other case, so its time per case scales to the
    batch) for the same steps; thrust and power histories are compared step
    by step on those cases."""
    synth = importlib.import_module("winds-master_b200.synth")
    wake = importlib.import_module("winds-master_b200.wake")
    gi = importlib.import_module("winds-master_b200.gamma_init")
    rng = np.random.Generator(np.random.PCG64(seed))
    yaws = rng.uniform(0.0, 30.0, ncases)

    def points(n_ages, yaw_list, s0):
        return [gi.OperatingPoint(synth.RotorCase(nst=41, nsteps=n_ages, dpsi_deg=1.0, U=11.4,
                                                  omega_rpm=12.1, yaw_deg=float(y), shear=0.2,
                                                  seed=s0 + k, jitter=0.0), 0.0)
                for k, y in enumerate(yaw_list)]

    t0 = time.perf_counter()
    tr = gi.run(points(120, rng.uniform(0.0, 30.0, 64), 900), 48, record=True, maxiter=200)
    keep = (tr["step_case"][:, 0] >= 4) & tr["lift"]
    # the previous-step base: these cases have stations past stall, where a
    # start on the extrapolated base passed the validation guards on 120-age
    # wakes yet moved stalled stations of the 1440-age run to another fixed
    # point (thrust 3% off the plain path); output scale from solver runs on
    # validation points of the same conditions
    m = gi.fit_start_value(tr["X"][keep], tr["dG"][keep], points(120, rng.uniform(0.0, 30.0, 8), 950),
                           16, bases=("previous",), maxiter=200)
    mlp_base, mlp_shrink, mlp_val, mlp_tried = m.base, m.shrink, m.validation, m.bases_tried
    train_s = time.perf_counter() - t0
    pts = points(ages, yaws, 100)
    cases, kjs = gi.build(pts, steps + 1)
    sub = list(range(0, ncases, ncases // plain_cases))
    xo = gi.extrapolation_only()
    out = {}
    for name, prec, mlp, graph, sel in (("fast", "f32c", m, True, None),
                                        ("fast_previous_start", "f32c", None, True, None),
                                        ("fast_extrapolated_start", "f32c", xo, True, None),
                                        ("plain_fp64", "f64", None, False, sub)):
        idx = list(range(ncases)) if sel is None else sel
        T, P, its, ms = [], [], [], []
        if sel is None:
            batches = [wake.WakeBatch([cases[k] for k in idx], integrator="pcc", precision=prec)]
            batches[0].set_kj([kjs[k] for k in idx], relax=0.3, tol=1e-6, maxiter=200)
            if mlp is not None:
                batches[0].set_mlp(mlp)
        else:  # each case alone
            batches = []
            for k in idx:
                b = wake.WakeBatch([cases[k]], integrator="pcc", precision=prec)
                b.set_kj([kjs[k]], relax=0.3, tol=1e-6, maxiter=200)
                batches.append(b)
        for s in range(steps):
            t_row, p_row, it_row, ms_s = [], [], [], 0.0
            for b in batches:
                b.step(1, graph=graph)
                t_, _, p_ = b.loads()
                t_row += list(t_)
                p_row += list(p_)
                it_row += list(b.kj_stats()[0])
                ms_s += b.stats()[0]
            T.append(t_row)
            P.append(p_row)
            its.append(int(np.sum(it_row)))
            ms.append(ms_s)
        inter = sum(b.stats()[1] for b in batches)
        for b in batches:
            b.close()
        out[name] = dict(T=np.array(T), P=np.array(P), iters=its, ms=ms, inter=inter, idx=idx)
    m.close()
    xo.close()
    f, p = out["fast"], out["plain_fp64"]

    def rel(x, y, idx):
        a, b_ = x["T"][:, idx], y["T"]
        c, d = x["P"][:, idx], y["P"]
        return (float((np.abs(a - b_) / np.abs(b_)).max()),
                float((np.abs(c - d) / np.maximum(np.abs(d), 1e-9 * np.abs(b_))).max()))
    relT, relP = rel(f, p, p["idx"])
    fast_ms = statistics.mean(f["ms"])
    plain_ms = statistics.mean(p["ms"]) * ncases / len(p["idx"])
    arms = {}
    for name in ("fast", "fast_previous_start", "fast_extrapolated_start"):
        a = out[name]
        tT, tP = rel(a, p, p["idx"])
        dT = np.abs(a["T"] - out["fast_previous_start"]["T"]) / np.abs(out["fast_previous_start"]["T"])
        arms[name] = {"steps_per_s": 1000.0 / statistics.mean(a["ms"]), "kj_iterations": a["iters"],
                      "kj_iterations_total": int(sum(a["iters"])),
                      "thrust_rel_diff_vs_plain_max": tT, "power_rel_diff_vs_plain_max": tP,
                      "thrust_rel_diff_vs_previous_start_max": float(dT.max())}
    return {"cases": ncases, "nodes_per_case": 41 * (ages + 1) * 3,
            "filaments_per_case": (40 * (ages + 1) + 41 * ages) * 3, "steps": steps,
            "steps_per_s": 1000.0 / fast_ms, "plain_fp64_steps_per_s": 1000.0 / plain_ms,
            "plain_fp64_cases_run": len(p["idx"]),
            "speedup_vs_plain_fp64": plain_ms / fast_ms,
            "interactions_per_step": f["inter"],
            "kj_iterations_fast": f["iters"], "kj_iterations_plain_on_subset": p["iters"],
            "thrust_rel_diff_max": relT, "power_rel_diff_max": relP,
            "start_value_arms": arms,
            "thrust_history_N": f["T"].sum(1).round(1).tolist(),
            "power_history_W": f["P"].sum(1).round(1).tolist(),
            "mlp_training_s": round(train_s, 2), "mlp_base": mlp_base, "mlp_output_shrink": mlp_shrink,
            "mlp_validation": mlp_val, "mlp_bases_tried": mlp_tried,
            "timing": "CUDA events around each step (fast paths: the lifting-line iteration is one "
            "launch of the step's graph; plain path: launched kernel by kernel, its "
            f"time per step measured on {len(p['idx'])} of the {ncases} equal-size cases and scaled "
            "to all of them)"}


# ------------------------------------------------------------------ our arm
def ours(args):
    import torch
    import torch.distributed as dist
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    if world > 1:
        import datetime
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))
    wb = importlib.import_module("winds-master_b200")
    lib = wb.lib()
    w, fams, P, nf, nt = workload(1 + rank, args.workload)
    interactions = nf * nt

    def dev(a):
        return torch.from_numpy(np.asarray(a).ravel(order="F").copy()).cuda()

    dfams = [(dev(F1), dev(F2), dev(g), dev(rc), F1.shape) for F1, F2, g, rc in fams]
    dP = (dev(P), P.shape)
    out = torch.zeros(P.size, dtype=torch.float64, device="cuda")
    flush = torch.empty(256 * 1024 * 1024 // 4, dtype=torch.float32, device="cuda")
    core, dval = ((wb.bs.CORE_CUTOFF, 1e-4) if args.core == "cutoff"
                  else (wb.bs.CORE_VATISTAS, 2.0))

    torch.cuda.synchronize()
    if args.tiling:
        T, KF, waves = args.tiling.split(",")
        wb.set_tuning(core, nt, nf, int(T), int(KF), float(waves))
        if args.layout:
            wb.set_layout(core, nt, nf, args.layout == "chained")
    # warm-up on the library's own stream (the first call autotunes the tiling)
    for _ in range(max(1, args.warmup)):
        wb.eval_device(dfams, dP, core, dval, 1000.0, out, "f32c")
    wb.sync()
    # timed work runs on a dedicated (non-default) stream shared with the events
    stream = torch.cuda.Stream()
    torch.cuda.set_stream(stream)
    sp = stream.cuda_stream
    for _ in range(2):
        wb.eval_device(dfams, dP, core, dval, 1000.0, out, "f32c", stream=sp)
    peak = C.c_double()
    lib.winds_bs_fp32_peak(C.byref(peak))

    clocks = ClockSampler(torch.cuda.current_device() if "CUDA_VISIBLE_DEVICES" not in os.environ
                          else int(os.environ["CUDA_VISIBLE_DEVICES"].split(",")[local]))
    clocks.start()
    if world > 1:
        dist.barrier()
    torch.cuda.synchronize()
    clocks.begin()
    step_ms, main_ms = [], []
    launches = 0
    near_pairs = 0
    for _ in range(args.steps):
        flush.zero_()  # L2 flush between timed steps (outside the events)
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        wb.eval_device(dfams, dP, core, dval, 1000.0, out, "f32c", stream=sp)
        e1.record(stream)
        torch.cuda.synchronize()
        step_ms.append(e0.elapsed_time(e1))
        m, n, near = wb.last_stats()
        main_ms.append(m)
        launches += n
        near_pairs = near
        free_pairs = wb.last_core_free()
        chained = wb.last_chained()
    torch.cuda.synchronize()
    clk = clocks.stop()
    wb.sync(sp)
    total_ms = sum(step_ms)
    if world > 1:
        t = torch.tensor([total_ms], device="cuda", dtype=torch.float64)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        total_ms = float(t.item())
    value = world * interactions * args.steps / (total_ms * 1e-3) / 1e9
    u32 = out.cpu().numpy()

    # plain FP64 GPU direct sum (the comparison path) and the accuracy of FP32c against it
    fp64 = None
    rel_err = None
    if not (args.no_fp64 or args.quick):
        out64 = torch.zeros_like(out)
        wb.eval_device(dfams, dP, core, dval, 1000.0, out64, "f64", stream=sp)
        torch.cuda.synchronize()
        t64 = []
        for _ in range(2):
            flush.zero_()
            e0 = torch.cuda.Event(enable_timing=True)
            e1 = torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            wb.eval_device(dfams, dP, core, dval, 1000.0, out64, "f64", stream=sp)
            e1.record(stream)
            torch.cuda.synchronize()
            t64.append(e0.elapsed_time(e1))
        fp64 = interactions / (statistics.median(t64) * 1e-3) / 1e9
        a = np.stack([u32.reshape(P.shape, order="F")[:, c].ravel(order="F") for c in range(3)], 1)
        b64 = out64.cpu().numpy().reshape(P.shape, order="F")
        b = np.stack([b64[:, c].ravel(order="F") for c in range(3)], 1)
        rel_err = float(np.max(np.linalg.norm(a - b, axis=1) / np.linalg.norm(b, axis=1)))

    # the same workload with the reference's default core (cut-off, d = 1e-4)
    cutoff_line = None
    if not args.quick:
        core_c = wb.bs.CORE_CUTOFF
        outc = torch.zeros_like(out)
        # the first call, on the library's own stream, tunes this core's bucket
        wb.eval_device(dfams, dP, core_c, 1e-4, 1000.0, outc, "f32c")
        wb.sync()
        for _ in range(2):
            wb.eval_device(dfams, dP, core_c, 1e-4, 1000.0, outc, "f32c", stream=sp)
        tc = []
        for _ in range(5):
            flush.zero_()
            e0 = torch.cuda.Event(enable_timing=True)
            e1 = torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            wb.eval_device(dfams, dP, core_c, 1e-4, 1000.0, outc, "f32c", stream=sp)
            e1.record(stream)
            torch.cuda.synchronize()
            tc.append(e0.elapsed_time(e1))
        free_c = wb.last_core_free()
        chained_c = wb.last_chained()
        out64c = torch.zeros_like(out)
        wb.eval_device(dfams, dP, core_c, 1e-4, 1000.0, out64c, "f64", stream=sp)
        torch.cuda.synchronize()
        a = outc.cpu().numpy().reshape(P.shape, order="F")
        b = out64c.cpu().numpy().reshape(P.shape, order="F")
        a = np.stack([a[:, c].ravel(order="F") for c in range(3)], 1)
        b = np.stack([b[:, c].ravel(order="F") for c in range(3)], 1)
        cutoff_line = {"core": "cut-off, d = 1e-4", "timed_steps": 5,
                       "gint_per_s": interactions / (statistics.median(tc) * 1e-3) / 1e9,
                       "core_free_fraction": free_c / interactions,
                       "rel_err_max_vs_fp64": float(np.max(np.linalg.norm(a - b, axis=1) /
                                                           np.linalg.norm(b, axis=1))),
                       "tiling": dict(zip(("targets_per_thread", "filaments_per_tile", "waves"),
                                          wb.get_tuning(core_c, nt, nf)),
                                      chained_stream=chained_c)}

    # end to end through the public host API: pinned host inputs, H2D + eval + D2H per step
    e2e_line = None
    if not args.quick:
        def pin(a):
            # a Fortran-order view of page-locked memory holding a copy of a
            a = np.asfortranarray(a, dtype=np.float64)
            f = torch.empty(a.size, dtype=torch.float64, pin_memory=True).numpy()
            f = f.reshape(a.shape, order="F")
            f[...] = a
            return f
        hfams = [tuple(pin(x) for x in f) for f in fams]
        hP = pin(P)
        hout = pin(np.zeros(P.shape, order="F"))
        h2d = sum(sum(x.nbytes for x in f) for f in hfams) + hP.nbytes
        d2h = hout.nbytes
        wb.eval_host(hfams, hP, core, dval, 1000.0, "f32c", out=hout)
        e2e_t = []
        for _ in range(max(1, min(args.steps, 5))):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            wb.eval_host(hfams, hP, core, dval, 1000.0, "f32c", out=hout)
            e2e_t.append(time.perf_counter() - t0)
        e2e = world * interactions / statistics.median(e2e_t) / 1e9
        e2e_line = {"value": e2e, "unit": UNIT, "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
                    "timing": "wall clock around the synchronous host-API call"}

    mean_main = statistics.mean(main_ms)
    flop = FLOP_PER_INTERACTION if args.core == "vatistas" else FLOP_PER_INTERACTION_CUTOFF
    achieved = flop * interactions / (mean_main * 1e-3) / 1e12
    traffic = profiled_traffic(interactions, chained)

    cpu = None
    if rank == 0 and world == 1 and not args.quick:
        rate, _ = cpu_rate(fams, P, 16)
        n = int(max(16, min(nt, 10.0 * rate * 1e9 / nf)))
        rate, dt = cpu_rate(fams, P, n, seed=1)
        cpu = {"value": rate, "unit": UNIT, "cores": os.cpu_count(), "kind": "port",
               "sample": f"{n} sampled targets x {nf} filaments ({dt:.1f} s), FP64 C restatement "
                         "of core/BiotSavart.m, OpenMP",
               "others": other_cpu_baselines(fams, P)}
    # the sub-benchmarks run on one GPU only: under torchrun the other ranks
    # would wait at the final barrier for minutes, past the group's timeout
    wake_line = None
    if rank == 0 and world == 1 and args.wake_steps > 0 and not args.quick:
        net = batch_start_value() if not args.no_studies else None
        wake_line = wake_bench(args, mlp=net)
        if net is not None:
            net.close()
    sharded_line = target_line = None
    if world > 1 and args.wake_steps > 0 and not args.quick:
        sharded_line = sharded_wake_bench(args, rank, world)
    if world > 1 and not args.quick:
        target_line = target_sharded_bench(args, rank, world, stream, flush)
    mlp_line = e2e_line_run = None
    if rank == 0 and world == 1 and not (args.quick or args.no_studies):
        mlp_line = kj_mlp_bench()
        if args.e2e_steps > 0:
            e2e_line_run = e2e_run_bench(args.e2e_steps)
    if rank == 0:
        line = {
            "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": total_ms / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32+f64",
            "data": "synthetic",
            "config": bench_config(args.workload, nt, nf, world),
            "roofline": {"bound": "fp32", "achieved": achieved, "peak": peak.value, "unit": "TFLOP/s",
                         "frac": achieved / peak.value if peak.value else None, "traffic": traffic,
                         "peak_source": "FFMA probe measured in this run (winds_bs_fp32_peak)",
                         "kernel": "bs_f32c", "flop_per_interaction": flop,
                         "kernel_ms": mean_main},
            "cpu_baseline": cpu,
            "e2e": e2e_line,
            "gpu_launches": launches,
            "clocks": clk,
            "plain_fp64_gint_per_s": fp64,
            "speedup_vs_plain_fp64": (value / world / fp64) if fp64 else None,
            "rel_err_max_vs_fp64": rel_err,
            "near_pairs_per_step": near_pairs,
            "core_free_pairs_per_step": free_pairs,
            "core_free_fraction": free_pairs / interactions,
            "tiling": dict(zip(("targets_per_thread", "filaments_per_tile", "waves"),
                               wb.get_tuning(core, nt, nf)), chained_stream=chained),
            "cutoff_core": cutoff_line,
            "wake_batch": wake_line,
            "wake_batch_sharded": sharded_line,
            "target_sharded": target_line,
            "kj_start_value": mlp_line,
            "e2e_run": e2e_line_run,
        }
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()


if __name__ == "__main__":
    a = parse()
    if a.impl == "reference":
        reference_arm(a)
    elif a.wake_only:
        wbm = importlib.import_module("winds-master_b200")
        wbm.set_autotune(False)
        print(json.dumps({"wake_batch": wake_bench(a, plain=False)}), flush=True)
    else:
        ours(a)
