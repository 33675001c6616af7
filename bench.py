#!/usr/bin/env python
"""Benchmark: DMRG solves/s of the Schwinger-model chain (spin formulation,
N=100 sites, x=100, m/g=0.125 -> mu=2.5, MPO bond 5, D=128), one solve =
ground state (seed-1 initial MPS) + first excited state by the projector
penalty (seed-11 initial MPS), convergence 1e-10, complex FP64.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl mpsgpu|reference]

One step is a batch of B (default 32) independent solves with different
seeds, swept in lockstep as four groups of 8 (each group on its own library
context and host thread; within a group the chains' local eigenproblems share
the grouped launches of every Lanczos round), in the split-precision form
(BF16-limb tcgen05 products until the energy settles, FP64 to convergence).
One process per GPU; the path does not shard (independent solves), so N GPUs
run N replicas of the workload ("replicas only", weak scaling) and `value`
is the total solves of all ranks divided by the max-over-ranks device time.
The line also carries the plain form (one solve alone) and the p50/p99
latency of the solves inside the batches.

Prints one JSON line (rank 0).  `value` is timed with CUDA events on the
library's stream with the initial states already in HBM; `e2e` is the same
metric through the C ABI with host buffers (initial MPS and MPO uploaded and
both result states downloaded inside the timed region).  L2 (126 MB) is
flushed between timed steps by writing a 256 MB buffer.
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

WORKLOAD = dict(workload="schwinger_N100_D128_gs+gap", N=100, x=100.0, mg=0.125, D=128,
                seed_gs=1, seed_exc=11, convtol=1e-10, d=2, mpo_bond=5)
MU = 2 * WORKLOAD["mg"] * np.sqrt(WORKLOAD["x"])
PRECISION = {"schedule": 2, "mixed": 1, "fp64": 0}  # options.precision of each form
PRECISION_TEXT = {
    "schedule": "FP64 products; eigensolver residual 1e-6 until the half-sweep energy change first falls below "
                "1e-6, then 1e-9 to convergence (the first such half-sweep cannot end the solve)",
    "mixed": "split-precision (BF16-limb tcgen05) products and residual 1e-6 until the half-sweep energy change "
             "first falls below 1e-6, then FP64 products at residual 1e-9 to convergence",
    "fp64": "FP64 products, eigensolver residual 1e-12 throughout (the reference's tolerance)"}
METRIC = "DMRG solves/s (Schwinger N=100 D=128, E0 + first gap, |dE/E|<=1e-10)"
UNIT = "solves/s"


def parse():
    p = argparse.ArgumentParser()
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=3)
    p.add_argument("--warmup", type=int, default=3)
    p.add_argument("--impl", default="mpsgpu", choices=["mpsgpu", "reference"])
    p.add_argument("--no-cpu-baseline", action="store_true")
    p.add_argument("--ref-iter-cap", type=int, default=0,
                   help="tests only: stop the sampled eigensolves after this many products instead of the "
                        "calibrated 60 (the line is then not a measurement)")
    p.add_argument("--batch", type=int, default=32, help="concurrent solves per step")
    p.add_argument("--batch-form", default="lockstep", choices=["lockstep", "streams"],
                   help="lockstep: one context sweeps the batch together (grouped launches); "
                        "streams: one context, stream and host thread per solve")
    p.add_argument("--groups", type=int, default=4,
                   help="lockstep: the batch as this many lockstep groups, each on its own context and host "
                        "thread, so that one group's host work and site steps overlap another's rounds")
    p.add_argument("--plain", type=int, default=1, help="also time one solve alone (the plain form)")
    p.add_argument("--arm-steps", type=int, default=1,
                   help="steps of each comparison arm (FP64 batch, FP64 batch with the mixed schedule)")
    p.add_argument("--precision", default="mixed", choices=["schedule", "mixed", "fp64"],
                   help="schedule: FP64 products with the mixed schedule of eigensolver tolerances; mixed: the "
                        "same schedule with split-precision (tcgen05) products until the energy settles; fp64: "
                        "FP64 with the reference's tolerance throughout")
    p.add_argument("--workload", default="schwinger",
                   choices=["schwinger", "grouped", "serving", "quench", "sample", "split_gemm"],
                   help="schwinger: the headline line; grouped/serving/quench: the secondary workloads; "
                        "sample/split_gemm: bounded cases for profilers")
    p.add_argument("--sites", type=int, default=40, help="sample: chain length of the bounded sweep sample")
    p.add_argument("--rounds", type=int, default=1, help="sample: half-sweeps of the bounded sweep sample")
    p.add_argument("--sample-batch", type=int, default=1,
                   help="sample: chains swept in lockstep (seeds 1, 1001, ...), one batch of grouped launches")
    p.add_argument("--mnk", default="4096,4096,2048", help="split_gemm: m,n,k")
    p.add_argument("--instances", type=int, default=512, help="grouped: matvec instances")
    p.add_argument("--requests", type=int, default=48, help="serving: requests in the stream")
    p.add_argument("--rate", type=float, default=50.0, help="serving: Poisson arrival rate, req/s")
    p.add_argument("--quenches", type=int, default=8, help="quench: concurrent chains")
    p.add_argument("--qsteps", type=int, default=20, help="quench: time steps per chain")
    p.add_argument("--qD", type=int, default=256, help="quench: maximum bond dimension")
    return p.parse_args()


# ---------------------------------------------------------------------------
# clocks sampled during the timed region
# ---------------------------------------------------------------------------

class ClockSampler:
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index: int):
        self.index = index
        self.samples = []
        self.proc = None

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.index), f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-lms", "200"], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.thread = threading.Thread(target=self._read, daemon=True)
            self.thread.start()
        except FileNotFoundError:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            parts = [s.strip() for s in line.split(",")]
            if len(parts) >= 9:
                self.samples.append(parts)

    def stop(self) -> dict:
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        sm = [float(s[1]) for s in self.samples if s[1].replace(".", "").isdigit()]
        mx = [float(s[2]) for s in self.samples if s[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for s in self.samples for i in range(4) if s[5 + i] == "Active"})
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(self.samples)}


# ---------------------------------------------------------------------------
# CPU baseline: the reference compiled from source (oracle/_ref), bounded sample
# ---------------------------------------------------------------------------

def reference_rate(procs: int, cap: int = 0) -> tuple:
    """Solves/s of the reference on `procs` cores of this host (independent
    solves, one per core), from its pinned complete solve scaled by this
    host's speed on a bounded sample (oracle/ref_timing.py); with the
    products per core-second of the sample and how the value was obtained."""
    from oracle import ref_timing  # the checker/baseline only
    s = ref_timing.speed_sample(procs, cap or ref_timing.CAP)
    secs, why = ref_timing.solve_seconds_here(s, strict=not cap or cap == ref_timing.CAP)
    sample = (f"one bulk site step per process of the reference's ground-state sweep of this workload "
              f"(oracle/_ref: the reference compiled from source; environments set up untimed; eigensolve stopped "
              f"after {s['cap']} products, then its QR gauge move and environment update), sites "
              f"{s['positions'][0]}..{s['positions'][-1]}, {s['procs']} single-threaded processes at once "
              f"({s['products']} products, {s['core_seconds']:.1f} core-s, {s['wall']:.1f} s wall)")
    detail = {"products_sample": s["products"], "core_seconds_sample": s["core_seconds"],
              "products_per_core_second": s["rate"], "wall_s": s["wall"]}
    if secs is None:
        return None, sample + f"; no value: {why}", detail
    detail["core_seconds_per_solve"] = secs
    return s["procs"] / secs, sample + f"; scaled to the complete solve: {why}", detail


def run_reference(args, rank: int, world: int) -> None:
    if rank != 0:
        return
    procs = min(os.cpu_count() or 1, 64)
    vals, walls, last = [], [], None
    for _ in range(max(1, args.steps)):  # no warm-up: nothing on the CPU path warms up
        try:
            v, sample, detail = reference_rate(procs, args.ref_iter_cap)
        except FileNotFoundError as e:  # the reference was not built here (no sources)
            v, sample = None, str(e)
        if v is None:
            print(json.dumps({"impl": "reference", "unavailable": sample}), flush=True)
            return
        if args.ref_iter_cap > 0:
            sample += f" [eigensolves stopped after {args.ref_iter_cap} products: plumbing test, not a measurement]"
        vals.append(v)
        walls.append(detail["wall_s"])
        last = (sample, detail)
    value = float(np.mean(vals))
    line = {"impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world,
            "steps": len(vals), "warmup": 0, "warmup_requested": args.warmup,
            "ms_per_step": 1e3 * float(np.mean(walls)),  # the sample's wall time; the solve's is in detail
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "c128",
            "data": "synthetic (seeded complex Gaussian initial MPS)",
            "config": {**WORKLOAD, "parallelism": f"replicas{world}", "l2": "n/a (CPU)"},
            "cpu_baseline": {"value": value, "unit": UNIT, "cores": procs, "kind": "reference", "sample": last[0]},
            "detail": last[1],
            "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


# ---------------------------------------------------------------------------
# GPU arm
# ---------------------------------------------------------------------------

def measured_peaks() -> dict:
    """HBM copy bandwidth and dense BF16 tensor throughput measured on this
    pool (MEASURED_PEAKS.json, driver-written), else the earlier measurement
    on this pool (fallback), with their sources."""
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            m = json.load(f)
        return {"hbm_gbs": float(m["hbm_gbs"]), "hbm_src": "MEASURED_PEAKS.json hbm_gbs (measured)",
                "bf16": float(m["bf16_tflops"]), "bf16_sustained": float(m.get("bf16_tflops_sustained",
                                                                              m["bf16_tflops"])),
                "bf16_src": "MEASURED_PEAKS.json bf16_tflops_sustained (measured)"}
    except Exception:
        return {"hbm_gbs": 6650.0, "hbm_src": "fallback 6.65 TB/s (earlier measurement on this pool)",
                "bf16": 1590.0, "bf16_sustained": 1400.0,
                "bf16_src": "fallback 1.4 PFLOP/s sustained (earlier measurement on this pool)"}


def bf16_peak() -> tuple:
    """Burst BF16 peak (for a kernel timed alone) and its source."""
    p = measured_peaks()
    return p["bf16"], p["bf16_src"].replace("_sustained", "").replace("sustained", "burst")


# dram__bytes_read.sum + dram__bytes_write.sum per launch from ncu captures of
# the same shapes, None where none was taken: the Lanczos step of eight D = 128
# Schwinger chains and the QR of a 256 x 128 site (one launch of the lockstep
# sample each), profiles/kernels_schwinger_sample_N40_D128_batch8.md
KERNEL_TRAFFIC = {"gemm_fp64_dmma": None, "gemm_split_tcgen05": None, "lanczos_step": 84.3e6, "qr": 0.613e6,
                  "split_operands": None}


def fp64_gemm_peak(torch) -> float:
    """Measured complex FP64 GEMM throughput of cuBLAS (torch.matmul on
    complex128, 4096^3, 8 n^3 flops), best of 5, TFLOP/s: the tensor-pipe
    FP64 denominator (the driver's MEASURED_PEAKS.json carries no FP64)."""
    n = 4096
    a = torch.randn(n, n, dtype=torch.complex128, device="cuda")
    b = torch.randn(n, n, dtype=torch.complex128, device="cuda")
    best = 0.0
    for _ in range(6):
        s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s.record()
        torch.matmul(a, b)
        e.record()
        torch.cuda.synchronize()
        best = max(best, 8.0 * n ** 3 / (s.elapsed_time(e) * 1e-3) / 1e12)
    del a, b
    return best


def attribution(form: str, value: float, arms: dict, plain_rate) -> dict:
    """Batched solves/s of the three forms, split into factors: the tolerance
    schedule (schedule / fp64), the tensor cores (mixed / schedule, the same
    schedule with split-precision products) and the batching (fp64 batched /
    one plain FP64 solve alone)."""
    v = {k: a["value"] for k, a in arms.items()}
    v[form] = value
    if not all(k in v for k in ("fp64", "schedule", "mixed")):
        return None
    return {"schedule": v["schedule"] / v["fp64"], "tensor_cores": v["mixed"] / v["schedule"],
            "concurrency": v["fp64"] / plain_rate if plain_rate else None}


def reduce_over_ranks(dist, x: float, op, device: str) -> float:
    """x combined over the ranks of the process group (MAX for times, SUM for
    work), or x itself without a group.  The only exchange the replicas make."""
    if dist is None:
        return x
    import torch
    t = torch.tensor([x], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=op)
    return float(t.item())


def run_gpu(args, rank: int, world: int, local_rank: int) -> None:
    import torch
    from mpsdyn_b200 import capi

    torch.cuda.set_device(local_rank)
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=600),
                                device_id=torch.device("cuda", local_rank))

    def barrier():
        if dist is not None:
            dist.barrier()

    def allreduce(x: float, op) -> float:
        return reduce_over_ranks(dist, x, op, "cuda")

    W = WORKLOAD
    B = args.batch
    lockstep = args.batch_form == "lockstep"
    # one library context (own CUDA stream) per concurrent solve; the
    # lockstep form runs the whole batch on the first one
    ctxs = [capi.Context(local_rank) for _ in range(B)]
    exts = [torch.cuda.ExternalStream(c.stream) for c in ctxs]
    flush_buf = torch.empty(256 * 1024 * 1024 // 4, dtype=torch.float32, device="cuda")
    mixed = args.precision == "mixed"
    prec = PRECISION[args.precision]
    opts = ctxs[0].options(convtol=W["convtol"], precision=prec)
    opts64 = ctxs[0].options(convtol=W["convtol"], precision=0)
    mpos = [c.mpo_schwinger(W["N"], MU, W["x"]) for c in ctxs]
    seeds = [(W["seed_gs"] + 1000 * (rank * B + i), W["seed_exc"] + 1000 * (rank * B + i)) for i in range(B)]
    G = max(1, min(args.groups, B)) if lockstep else 1
    members = [list(range(g * B // G, (g + 1) * B // G)) for g in range(G)]  # solves of each lockstep group
    lead = {i: mem[0] for mem in members for i in mem}                      # a group's context: its first solve's
    owner = [ctxs[lead[i]] if lockstep else ctxs[i] for i in range(B)]
    inits = [(c.mps_random(W["N"], 2, W["D"], sg), c.mps_random(W["N"], 2, W["D"], se))
             for c, (sg, se) in zip(owner, seeds)]
    hosts = [(g.download()[0], x.download()[0]) for g, x in inits]
    h2d_mps = sum(a.nbytes for a in hosts[0][0]) + sum(a.nbytes for a in hosts[0][1])
    mpo_bytes = 16 * (2 * 1 * 2 * 5 + 2 * 5 * 2 * 1 + (W["N"] - 2) * 2 * 5 * 2 * 5)
    results = [None] * B

    def solve_resident(i, o=None):
        o = o or opts
        c = ctxs[i]
        g, x = inits[i][0].copy(), inits[i][1].copy()
        e0, s0 = c.find_ground_state(mpos[i], W["D"], g, 0.0, o)
        e1, s1 = c.find_next_excited_state(mpos[i], W["D"], [g], x, 0.0, o)
        g.free()
        x.free()
        results[i] = {"E0": e0, "E1": e1, "gs": s0, "exc": s1}

    def solve_e2e(i):
        c = ctxs[i]
        m = c.mpo_schwinger(W["N"], MU, W["x"])           # host build + upload
        g, x = c.mps(hosts[i][0]), c.mps(hosts[i][1])      # host -> device
        e0, _ = c.find_ground_state(m, W["D"], g, 0.0, opts)
        e1, _ = c.find_next_excited_state(m, W["D"], [g], x, 0.0, opts)
        og, _ = g.download()                               # device -> host
        ox, _ = x.download()
        results[i] = {"E0": e0, "E1": e1, "d2h": sum(a.nbytes for a in og) + sum(a.nbytes for a in ox) + 16}
        g.free()
        x.free()
        m.free()

    def lockstep_solves(o, e2e=False, g=0):
        # the solves of group g swept in lockstep on the group's context:
        # their local eigenproblems share the grouped launches of every
        # Lanczos round
        mem = members[g]
        c = ctxs[mem[0]]
        if e2e:
            ms = [c.mpo_schwinger(W["N"], MU, W["x"]) for _ in mem]            # host build + upload
            gs = [c.mps(hosts[i][0]) for i in mem]                               # host -> device
            xs = [c.mps(hosts[i][1]) for i in mem]
        else:
            ms = [mpos[mem[0]]] * len(mem)
            gs = [inits[i][0].copy() for i in mem]
            xs = [inits[i][1].copy() for i in mem]
        e0, st0, s0 = c.find_ground_state_batch(ms, W["D"], gs, 0.0, o)
        if any(st0):
            raise RuntimeError(f"ground-state batch: statuses {st0}")
        e1, st1, s1 = c.find_next_excited_state_batch(ms, W["D"], [[x] for x in gs], xs, 0.0, o)
        if any(st1):
            raise RuntimeError(f"excited-state batch: statuses {st1}")
        for q, i in enumerate(mem):
            results[i] = {"E0": e0[q], "E1": e1[q], "gs": s0[q], "exc": s1[q]}
            if e2e:
                og, _ = gs[q].download()                                          # device -> host
                ox, _ = xs[q].download()
                results[i]["d2h"] = sum(a.nbytes for a in og) + sum(a.nbytes for a in ox) + 16
        for v in gs + xs:
            v.free()
        if e2e:
            for m in ms:
                m.free()

    def run_batch(fn, timed_events=True, o=None, e2e=False):
        if lockstep:
            # one host thread per group; the span runs from the earliest start
            # event to the latest end event on the groups' streams
            gev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(G)]
            errs = []

            def group(g):
                try:
                    gev[g][0].record(exts[members[g][0]])
                    lockstep_solves(o or opts, e2e, g)
                    gev[g][1].record(exts[members[g][0]])
                except Exception as ex:  # reported after the join
                    errs.append(ex)

            ths = [threading.Thread(target=group, args=(g,)) for g in range(G)]
            for t in ths:
                t.start()
            for t in ths:
                t.join()
            torch.cuda.synchronize()
            if errs:
                raise errs[0]
            if not timed_events:
                return None, None
            t0 = min(range(G), key=lambda g: 0.0 if g == 0 else gev[0][0].elapsed_time(gev[g][0]))
            span = max(gev[t0][0].elapsed_time(gev[g][1]) for g in range(G))
            per = []
            for g in range(G):
                per += [gev[g][0].elapsed_time(gev[g][1])] * len(members[g])  # a solve completes with its group
            return span, per
        evs = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(B)]
        go = threading.Barrier(B)

        def body(i):
            go.wait()
            if timed_events:
                evs[i][0].record(exts[i])
            fn(i)
            if timed_events:
                evs[i][1].record(exts[i])

        ths = [threading.Thread(target=body, args=(i,)) for i in range(B)]
        for t in ths:
            t.start()
        for t in ths:
            t.join()
        torch.cuda.synchronize()
        if not timed_events:
            return None, None
        # batch time on the device: earliest start to latest end (events of
        # different streams on one device are comparable)
        t0 = min(range(B), key=lambda i: 0.0 if i == 0 else evs[0][0].elapsed_time(evs[i][0]))
        span = max(evs[t0][0].elapsed_time(evs[i][1]) for i in range(B))
        per = [evs[i][0].elapsed_time(evs[i][1]) for i in range(B)]
        return span, per

    def flush_l2():
        with torch.cuda.stream(exts[0]):
            flush_buf.zero_()
        torch.cuda.synchronize()

    # ---- warm-up ----
    for _ in range(args.warmup):
        run_batch(solve_resident, timed_events=False)

    # ---- timed: inputs resident in HBM ----
    clocks = ClockSampler(local_rank)
    clocks.start()
    launches0 = sum(c.launches for c in ctxs)
    barrier()
    spans, lat = [], []
    energies = []
    for _ in range(args.steps):
        flush_l2()
        span, per = run_batch(solve_resident)
        spans.append(span)
        lat.extend(per)
        energies.append([(r["E0"], r["E1"]) for r in results])
    launches = sum(c.launches for c in ctxs) - launches0
    barrier()
    clk = clocks.stop()
    stats = results[0]
    total_ms = allreduce(float(sum(spans)), torch.distributed.ReduceOp.MAX if dist else None)
    solves = allreduce(float(args.steps * B), torch.distributed.ReduceOp.SUM if dist else None)
    value = solves / (total_ms * 1e-3)

    # ---- timed: end to end through the C ABI with host buffers ----
    barrier()
    e2e_ms = []
    for _ in range(args.steps):
        flush_l2()
        t0 = time.perf_counter()
        run_batch(solve_e2e, timed_events=False, e2e=True)
        e2e_ms.append((time.perf_counter() - t0) * 1e3)
    d2h = sum(r["d2h"] for r in results)
    e2e_total = allreduce(float(sum(e2e_ms)), torch.distributed.ReduceOp.MAX if dist else None)
    e2e_value = solves / (e2e_total * 1e-3)

    # ---- comparison arms, same seeds: the batch in FP64 throughout, and in
    # FP64 with the mixed form's schedule of tolerances (precision 2), which
    # splits mixed / FP64 into what the schedule saves and what the tensor
    # cores save ----
    def batch_arm(precision):
        o = ctxs[0].options(convtol=W["convtol"], precision=precision)
        barrier()
        spans_a, energies_a = [], []
        arm_steps = max(1, args.arm_steps)
        for _ in range(arm_steps):
            flush_l2()
            span, _ = run_batch(lambda i: solve_resident(i, o), o=o)
            spans_a.append(span)
            energies_a.append([(r["E0"], r["E1"]) for r in results])
        t = allreduce(float(sum(spans_a)), torch.distributed.ReduceOp.MAX if dist else None)
        dE = max(max(abs(a[0] - b[0]) / abs(b[0]), abs(a[1] - b[1]) / abs(b[1]))
                 for sa, sb in zip(energies, energies_a) for a, b in zip(sa, sb))
        arm_solves = allreduce(float(arm_steps * B), torch.distributed.ReduceOp.SUM if dist else None)
        return {"value": arm_solves / (t * 1e-3), "ms_per_step": t / arm_steps, "steps": arm_steps,
                "max_rel_dE_vs_line": dE,
                "products_per_solve": results[0]["gs"]["matvecs"] + results[0]["exc"]["matvecs"]}

    # the other two forms, same seeds (the line's own form is the line)
    arms = {}
    if prec != 0:
        arms["fp64"] = batch_arm(0)
        if prec == 2:
            arms["mixed"] = batch_arm(1)
        else:
            arms["schedule"] = batch_arm(2)

    # ---- with the library's kernel profiler on (events around 1 in 32
    # launches of each kernel class): one FP64 solve alone (the plain form),
    # and one lockstep group of the line alone (its first group's solves, the
    # line's precision; group work on other streams runs concurrently, so the
    # classes' shares of the group's time may add up to more than 1) ----
    def profiled_single(o):
        flush_l2()
        ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        ctxs[0].profile_begin()
        ev0.record(exts[0])
        solve_resident(0, o)
        ev1.record(exts[0])
        ev1.synchronize()
        prof = ctxs[0].profile_end()
        r = results[0]
        return ev0.elapsed_time(ev1), prof, r

    def profiled_group(o):
        flush_l2()
        lead0 = members[0][0]
        ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        ctxs[lead0].profile_begin()
        ev0.record(exts[lead0])
        lockstep_solves(o, False, 0)
        ev1.record(exts[lead0])
        ev1.synchronize()
        prof = ctxs[lead0].profile_end()
        return ev0.elapsed_time(ev1), prof

    plain_ms, prof64, r64 = profiled_single(opts64) if args.plain else (None, None, None)
    if args.plain and lockstep:
        line_ms, profln = profiled_group(opts)
    elif args.plain and prec != 0:
        line_ms, profln, _ = profiled_single(opts)
    else:
        line_ms, profln = None, None

    if rank != 0:
        for c in ctxs:
            c.close()
        if dist is not None:
            dist.destroy_process_group()
        return

    # ---- roofline of the dominant kernels, from the profiled single solves ----
    peak64 = fp64_gemm_peak(torch)
    peaks = measured_peaks()

    def kernel_table(prof, total_ms):
        out = {}
        for name, k in (prof or {}).get("kernels", {}).items():
            if not k["calls"] or k["ms"] <= 0:
                continue
            rate = k["work"] / (k["ms"] * 1e-3)
            if name in ("lanczos_step", "split_operands"):
                ach, pk, unit, bound, src = rate / 1e9, peaks["hbm_gbs"], "GB/s", "hbm", peaks["hbm_src"]
            elif name == "gemm_split_tcgen05":
                ach, pk, unit, bound, src = rate / 1e12, peaks["bf16_sustained"], "TFLOP/s", "tensor", peaks["bf16_src"]
            else:
                ach, pk, unit, bound = rate / 1e12, peak64, "TFLOP/s", "tensor"
                src = "cuBLAS complex128 GEMM 4096^3 measured in this run (FP64 tensor pipe)"
            out[name] = {"bound": bound, "achieved": ach, "peak": pk, "unit": unit, "frac": ach / pk,
                         "peak_source": src, "sampled_launches": k["calls"],
                         "work_per_launch": k["work"] / k["calls"],
                         "share_of_time": 32.0 * k["ms"] / total_ms if total_ms else None}
        return out

    table64 = kernel_table(prof64, plain_ms)
    tableln = kernel_table(profln, line_ms)

    def dominant(table, note):
        # the largest share among the kernels of the Lanczos rounds, which run
        # one after another on the group's stream; the QRs run on the chains'
        # own streams, up to a group's worth at once, so their summed event
        # time overstates their share of the wall time
        if not table:
            return None
        cand = [n for n in table if n != "qr"] or list(table)
        name = max(cand, key=lambda n: table[n]["share_of_time"] or 0.0)
        d = dict(table[name])
        d.update(kernel=name, traffic=KERNEL_TRAFFIC.get(name), traffic_unit="bytes per launch", note=note)
        return d

    roofline = dominant(tableln if (prec != 0 or lockstep) else table64,
                        "achieved = sampled launches' algorithmic work / their summed CUDA-event time, one "
                        "lockstep group of the line's form alone on the GPU (8 solves; one Lanczos round is one "
                        "grouped launch of each kernel for all of them); lanczos_step bytes: basis read twice + "
                        "work vector traffic; gemm_split_tcgen05 flops: 24 BF16 MMAs per complex k-step")

    cpu = None
    if not args.no_cpu_baseline and world == 1:
        try:
            procs = min(os.cpu_count() or 1, 64)
            cv, sample, detail = reference_rate(procs)
            cpu = {"value": cv, "unit": UNIT, "cores": procs, "kind": "reference", "sample": sample,
                   "detail": detail}
        except Exception as e:  # the baseline is reported, not required
            cpu = {"value": None, "unit": UNIT, "cores": 0, "kind": "reference", "sample": f"failed: {e}"}

    lat_s = np.array(lat) * 1e-3
    e0s = [e for step in energies for e in step]
    plain_rate = 1e3 / plain_ms if plain_ms else None
    s_gs, s_ex = stats["gs"], stats["exc"]
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": total_ms / args.steps, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "c128/bf16x3" if mixed else "c128",
        "data": "synthetic (seeded complex Gaussian initial MPS, model MPO built in-library)",
        "config": {**WORKLOAD, "mu": MU, "parallelism": f"replicas{world}",
                   "precision": f"{args.precision}: {PRECISION_TEXT[args.precision]}",
                   "batch": B,
                   "groups": G,
                   "batch_form": ("lockstep: the B solves swept together on one stream, their local "
                                  "eigenproblems in shared grouped launches" if lockstep else
                                  "concurrent independent solves, one stream and host thread each"),
                   "l2": "flushed between steps (256 MB write)"},
        "e2e": {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": B * (h2d_mps + mpo_bytes),
                "d2h_bytes_per_step": d2h, "ms_per_step": e2e_total / args.steps},
        "latency_s": {"p50": float(np.percentile(lat_s, 50)), "p99": float(np.percentile(lat_s, 99))},
        "plain_single_solve_ms": plain_ms,
        "plain_fp64_solves_per_s": plain_rate,
        "vs_plain_fp64": (value / plain_rate) if plain_rate else None,
        "line_form_profiled_ms": line_ms,
        "line_form_profiled": ("one lockstep group of the line (solves " + str(members[0]) + ") alone"
                               if lockstep else "one solve of the line's precision alone"),
        "arms": arms,
        "attribution": attribution(args.precision, value, arms, plain_rate),
        "roofline": roofline,
        "kernels_line_form": tableln,
        "kernels_fp64_single": table64,
        "cpu_baseline": cpu,
        "clocks": clk,
        "gpu_launches": launches,
        "results": {"E0": e0s[0][0], "E1": e0s[0][1], "gap": e0s[0][1] - e0s[0][0],
                    "gs": {k: s_gs[k] for k in ("rounds", "site_solves", "matvecs", "split_rounds", "split_matvecs",
                                                 "flops")},
                    "exc": {k: s_ex[k] for k in ("rounds", "site_solves", "matvecs", "split_rounds", "split_matvecs",
                                                  "flops")}},
    }
    print(json.dumps(line), flush=True)
    for c in ctxs:
        c.close()
    if dist is not None:
        dist.destroy_process_group()


# ---------------------------------------------------------------------------
# secondary workloads (single GPU, one JSON line each)
# ---------------------------------------------------------------------------

def run_grouped(args) -> None:
    """Grouped effective-Hamiltonian matvec over `--instances` instances of
    mixed shapes: D ~ U{32..1024}, w ~ U{3,5}, d = 2, entries i.i.d. complex
    N(0,1) (torch generator, seed 2); one grouped product = 3 launches
    captured once in a CUDA graph and replayed; TFLOP/s from CUDA events."""
    import torch
    from mpsdyn_b200 import capi
    n = args.instances
    g = torch.Generator(device="cuda").manual_seed(2)
    rs = np.random.default_rng(2)
    Ds = rs.choice([32, 64, 128, 256, 512, 1024], size=n)
    ws = rs.choice([3, 5], size=n)
    ctx = capi.Context(0)
    keep, inst = [], []

    def randn(k):
        return torch.randn(k, dtype=torch.complex128, device="cuda", generator=g)
    for D, w in zip(Ds.tolist(), ws.tolist()):
        d = 2
        L, W, R, x = randn(D * w * D), randn(d * w * d * w), randn(D * w * D), randn(D * d * D)
        y = torch.empty(D * d * D, dtype=torch.complex128, device="cuda")
        keep.append((D, w, L, W, R, x, y))
        inst.append(dict(d=d, wl=w, wr=w, Dl=D, Dr=D, L=L.data_ptr(), W=W.data_ptr(), Rt=R.data_ptr(),
                         x=x.data_ptr(), y=y.data_ptr()))
    torch.cuda.synchronize()
    ms, flops = capi.heff_matvec_grouped(ctx, inst, args.steps)
    # accuracy: relative error of a few instances against torch (cuBLAS) FP64
    errs = []
    check = list(range(min(n, 3))) + [int(np.argmax(Ds))]
    y64 = {k: keep[k][6].clone() for k in check}
    for k in check:
        D, w, L, W, R, x, y = keep[k]
        Lm = L.view(D, w, D).permute(2, 1, 0)            # column-major (bra, w, ket) -> [a', b, a]
        Wm = W.view(w, 2, w, 2).permute(3, 2, 1, 0)      # [s', b, s, c]
        Rt = R.view(D, w, D).permute(2, 1, 0)            # [r, c, r']  (ket, w, bra)
        X = x.view(D, 2, D).permute(2, 1, 0)             # [a, s, r]
        T1 = torch.einsum("pba,asr->pbsr", Lm, X)        # pairwise, the kernel's contraction order
        T2 = torch.einsum("pbsr,tbsc->ptcr", T1, Wm)
        ref = torch.einsum("ptcr,rcq->ptq", T2, Rt)
        Y = y.view(D, 2, D).permute(2, 1, 0)
        errs.append(float((Y - ref).abs().max() / ref.abs().max()))
    peak = fp64_gemm_peak(torch)
    tf = flops / (ms * 1e-3) / 1e12
    roof64 = {"bound": "tensor", "achieved": tf, "peak": peak, "unit": "TFLOP/s", "frac": tf / peak,
              "peak_source": "cuBLAS complex128 GEMM 4096^3 measured in this run"}
    split = None
    if args.precision != "fp64":
        # the same products in split precision (tcgen05, BF16 limbs); the
        # environments' limb planes are made once (ms_prepare), x and the
        # intermediate in every product
        ms_s, _, ms_prep = capi.heff_matvec_grouped_ex(ctx, inst, 1, args.steps)
        torch.cuda.synchronize()
        serr = max(float((keep[k][6] - y64[k]).abs().max() / y64[k].abs().max()) for k in check)
        gemm_flops = sum(8.0 * (D * w * D * 2 * D + D * 2 * D * w * D) for D, w in zip(Ds.tolist(), ws.tolist()))
        bpk, bsrc = bf16_peak()
        bf16_rate = 6.0 * gemm_flops / (ms_s * 1e-3) / 1e12
        split = {"ms_per_step": ms_s, "tflops_fp64_equivalent": flops / (ms_s * 1e-3) / 1e12,
                 "env_prepare_ms_once": ms_prep, "rel_error_vs_fp64": serr,
                 "speedup_vs_fp64": ms / ms_s,
                 "roofline": {"bound": "tensor", "achieved": bf16_rate, "peak": bpk, "unit": "TFLOP/s",
                              "frac": bf16_rate / bpk, "peak_source": bsrc,
                              "note": ("BF16 tensor flops (24 limb MMAs per complex k-step = 6x the complex "
                                       "GEMM flops) over the whole product time, prep and leg kernel included")}}
    line = {"metric": "grouped effective-Hamiltonian matvec TFLOP/s (512 instances)",
            "value": split["tflops_fp64_equivalent"] if split else tf,
            "unit": "TFLOP/s", "n_gpus": 1, "steps": args.steps, "warmup": 1,
            "ms_per_step": split["ms_per_step"] if split else ms,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "c128/bf16x3" if split else "c128",
            "data": "synthetic (complex N(0,1), torch generator seed 2)",
            "config": {"workload": "grouped_matvec_x512", "instances": n, "D": "U{32..1024}", "w": "U{3,5}",
                       "precision": "split (BF16 limbs, tcgen05); value in FP64-equivalent flops" if split else "fp64",
                       "graph": "grouped launches captured once, replayed", "l2": "inputs > 126 MB L2"},
            "roofline": split["roofline"] if split else roof64,
            "rel_error_vs_cublas_fp64": max(errs), "flops_per_step": flops,
            "fp64": {"tflops": tf, "ms_per_step": ms, "roofline": roof64}, "split": split}
    print(json.dumps(line), flush=True)
    ctx.close()


def run_serving(args) -> None:
    """Poisson stream of Ising ground-state requests (L ~ U[16,256],
    g ~ U[0.5,1.5], h ~ U[0,0.2], J = 1, D ~ U{32,64,128,256}, seed = request
    id, convergence 1e-10) at `--rate` req/s into the solve server, cut to
    `--requests` requests."""
    from mpsdyn_b200 import capi
    import torch
    rs = np.random.default_rng(4)
    n = args.requests
    Ls = rs.integers(16, 257, size=n)
    gs = rs.uniform(0.5, 1.5, size=n)
    hs = rs.uniform(0.0, 0.2, size=n)
    Ds = rs.choice([32, 64, 128, 256], size=n)
    gaps = rs.exponential(1.0 / args.rate, size=n)
    free, total = torch.cuda.mem_get_info(0)
    budget = int(free * 0.85)

    def stream(precision):
        with capi.Server(0, slots=args.batch, hbm_budget_bytes=budget) as srv:
            t0 = time.perf_counter()
            nxt = t0
            for i in range(n):
                nxt += gaps[i]
                dt = nxt - time.perf_counter()
                if dt > 0:
                    time.sleep(dt)
                srv.submit(0, int(Ls[i]), int(Ds[i]), 1.0, float(gs[i]), float(hs[i]), i + 1, 1e-10, precision)
            srv.drain()
            wall = time.perf_counter() - t0
            res = srv.poll()
        ok = [r for r in res if r["status"] == 0]
        bad = [r["status"] for r in res if r["status"] != 0]
        lat = np.array([r["t_end"] - r["t_submit"] for r in ok]) if ok else np.zeros(1)
        span = max(r["t_end"] for r in res) - min(r["t_submit"] for r in res)
        return {"value": len(ok) / span, "latency_s": {"p50": float(np.percentile(lat, 50)),
                                                       "p99": float(np.percentile(lat, 99))},
                "completed": len(ok), "failed": {str(k): bad.count(k) for k in sorted(set(bad))}, "wall_s": wall,
                "flops_total": float(sum(r["flops"] for r in ok)),
                "energies": {int(r["id"]): r["energy"] for r in ok}}

    mixed = args.precision == "mixed"
    prec = PRECISION[args.precision]
    main = stream(prec)
    fp64 = stream(0) if prec != 0 else None
    cmp = None
    if fp64:
        common = sorted(set(main["energies"]) & set(fp64["energies"]))
        rel = {k: abs(main["energies"][k] - fp64["energies"][k]) / abs(fp64["energies"][k]) for k in common}
        worst = sorted(common, key=lambda k: -rel[k])[:3]
        cmp = {"value": fp64["value"], "latency_s": fp64["latency_s"], "completed": fp64["completed"],
               "failed": fp64["failed"],
               "max_rel_dE_vs_fp64": max(rel.values(), default=None),
               "median_rel_dE_vs_fp64": float(np.median(list(rel.values()))) if rel else None,
               # the requests that differ most (request id = seed; index id - 1 of the stream)
               "largest_dE": [{"id": k, "L": int(Ls[k - 1]), "D": int(Ds[k - 1]), "g": float(gs[k - 1]),
                               "h": float(hs[k - 1]), "E_line": main["energies"][k], "E_fp64": fp64["energies"][k],
                               "rel": rel[k]} for k in worst],
               "line_over_fp64": main["value"] / fp64["value"] if fp64["value"] else None}
    line = {"metric": "served DMRG solves/s (Ising mix)", "value": main["value"], "unit": "solves/s",
            "n_gpus": 1, "steps": n, "warmup": 0, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "c128/bf16x3" if mixed else "c128",
            "data": "synthetic request stream (numpy seed 4)",
            "config": {"workload": "serving_ising_poisson", "requests": n, "rate_req_s": args.rate,
                       "slots": args.batch, "hbm_budget_bytes": budget, "L": "U[16,256]", "D": "U{32,64,128,256}",
                       "precision": f"{args.precision}: {PRECISION_TEXT[args.precision]}"},
            "latency_s": main["latency_s"], "completed": main["completed"], "failed": main["failed"],
            "wall_s": main["wall_s"], "flops_total": main["flops_total"], "fp64_stream": cmp}
    print(json.dumps(line), flush=True)


def run_quench(args) -> None:
    """Batched real-time quenches: L = 64, d = 2, from the D = 1 all-up
    product state, J = 1, g ~ U[0.2, 2.0], h = 0.1, second-order MPO time
    evolution (IsingHamiltonian::getUMPO + Contractor::optimize), dt = 0.01,
    bond dimension up to `--qD`; <sigma_x> at the centre and the centre
    entropy after every step.  `--quenches` chains x `--qsteps` steps, one
    context per chain, all chains concurrent; run in FP64 and, unless
    --precision fp64, again with split-precision local vectors (optimize with
    precision 1), reporting both rates and the observables' largest deviation
    of the split run from the FP64 one."""
    from mpsdyn_b200 import capi
    rs = np.random.default_rng(5)
    nq, ns, L, D = args.quenches, args.qsteps, 64, args.qD
    gvals = rs.uniform(0.2, 2.0, size=nq)
    sx = np.array([[0, 1], [1, 0]], dtype=complex)

    def run(precision):
        out = [None] * nq
        step_ms = [[] for _ in range(nq)]
        errors = []

        def chain(i):
            try:
                with capi.Context(0) as c:
                    U = c.mpo_ising_evolution(L, 1.0, float(gvals[i]), 0.1, 0.01, False)
                    st = c.mps_product(L, 2, 1)
                    o = c.options(convtol=1e-10, precision=precision)
                    obs = []
                    for _ in range(ns):
                        t = time.perf_counter()
                        aux = st.copy()
                        c.optimize(U, aux, st, D, o)
                        aux.free()
                        m = c.expectation_local(st, sx)[L // 2]
                        st.gauge("L")
                        s = c.entropy(st, L // 2)
                        step_ms[i].append((time.perf_counter() - t) * 1e3)
                        obs.append((m, s))
                    out[i] = np.array(obs, dtype=float)
            except Exception as e:  # reported in the line, not swallowed
                errors.append(f"chain {i}: {e}")
        t0 = time.perf_counter()
        ths = [threading.Thread(target=chain, args=(i,)) for i in range(nq)]
        for t in ths:
            t.start()
        for t in ths:
            t.join()
        wall = time.perf_counter() - t0
        per = np.array([x for s in step_ms for x in s]) if any(step_ms) else np.zeros(1)
        done = sum(len(s) for s in step_ms)
        return {"value": done / wall, "wall_s": wall,
                "latency_ms_per_step": {"p50": float(np.percentile(per, 50)), "p99": float(np.percentile(per, 99))},
                "errors": errors}, out

    r64, o64 = run(0)
    split = None
    if args.precision != "fp64":
        rsp, osp = run(1)
        ok = [i for i in range(nq) if o64[i] is not None and osp[i] is not None]
        dev = np.array([np.abs(osp[i] - o64[i]).max(axis=0) for i in ok]) if ok else np.zeros((1, 2))
        split = dict(rsp, max_abs_dev_vs_fp64={"sx_center": float(dev[:, 0].max()),
                                               "entropy_center": float(dev[:, 1].max())},
                     speedup_vs_fp64=rsp["value"] / r64["value"] if r64["value"] else None)
    line = {"metric": "batched quench time steps/s (L=64, D<=%d)" % D, "value": r64["value"],
            "unit": "steps/s", "n_gpus": 1, "steps": ns, "warmup": 0, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "c128", "data": "synthetic (g ~ U[0.2,2], numpy seed 5)",
            "config": {"workload": "quench_ising_L64", "quenches": nq, "steps": ns, "dt": 0.01, "D_max": D},
            "latency_ms_per_step": r64["latency_ms_per_step"], "errors": r64["errors"], "wall_s": r64["wall_s"],
            "split": split,
            "last": {"sx_center": float(o64[0][-1][0]), "entropy_center": float(o64[0][-1][1])}
            if o64[0] is not None else None}
    print(json.dumps(line), flush=True)
    if r64["errors"] or (split and split["errors"]):
        sys.exit(1)


def run_sample(args) -> None:
    """A bounded sample of the headline sweep for profilers: the ground-state
    sweep of the Schwinger chain (x = 100, m/g = 0.125, seed-1 initial MPS,
    convergence 1e-10) on --sites sites with D = 128, stopped after --rounds
    half-sweeps (the library returns MPSGPU_NOT_CONVERGED at the round limit,
    which ends the sample), in --precision.  With 40 sites, 26 bulk sites
    have the (128, 5, 128) shapes of the 100-site chain, so the kernel mix per
    site step is the headline's while the launch count stays small enough for
    a profiler that slows every launch down.  With --sample-batch B > 1, B
    chains (seeds 1, 1001, ...) are swept in lockstep, as the bench line's
    batches are."""
    from mpsdyn_b200 import capi
    B = max(1, args.sample_batch)
    with capi.Context(0) as ctx:
        H = ctx.mpo_schwinger(args.sites, MU, WORKLOAD["x"])
        psis = [ctx.mps_random(args.sites, 2, WORKLOAD["D"], 1 + 1000 * i) for i in range(B)]
        o = ctx.options(convtol=1e-10, max_rounds=args.rounds, precision=PRECISION[args.precision])
        l0 = ctx.launches
        t0 = time.perf_counter()
        status = "converged"
        if B == 1:
            try:
                ctx.find_ground_state(H, WORKLOAD["D"], psis[0], 0.0, o)
            except capi.MpsgpuError as e:
                if e.status != 2:  # anything but the round limit is a failure
                    raise
                status = "round limit"
        else:
            _, sts, _ = ctx.find_ground_state_batch([H] * B, WORKLOAD["D"], psis, 0.0, o)
            if any(st not in (0, 2) for st in sts):
                raise RuntimeError(f"sample batch: statuses {sts}")
            status = "round limit" if any(st == 2 for st in sts) else "converged"
        ctx.synchronize()
        print(json.dumps({"sample": f"schwinger N={args.sites} D={WORKLOAD['D']}, {args.rounds} half-sweep(s), "
                                    f"{args.precision}, {B} chain(s)", "status": status,
                          "launches": ctx.launches - l0, "seconds": time.perf_counter() - t0}), flush=True)


def run_split_gemm(args) -> None:
    """One split-precision complex GEMM C = A B (seeded complex Gaussian A,
    B) through mpsgpu_zgemm_split, timed over --steps runs with CUDA events,
    with its largest entrywise error relative to |A||B| on a 64 x 64 corner."""
    from mpsdyn_b200 import capi
    m, n, k = (int(v) for v in args.mnk.split(","))
    rng = np.random.default_rng(0)
    A = rng.standard_normal((m, k)) + 1j * rng.standard_normal((m, k))
    Bm = rng.standard_normal((k, n)) + 1j * rng.standard_normal((k, n))
    with capi.Context(0) as ctx:
        Cm, t_all, t_mma = capi.zgemm_split(ctx, A, Bm, repeats=args.steps)
    c = min(64, m, n)
    ref = A[:c] @ Bm[:, :c]
    rel = float(np.max(np.abs(Cm[:c, :c] - ref) / (np.abs(A[:c]) @ np.abs(Bm[:, :c]))))
    fl = 8.0 * m * n * k
    out = {"m": m, "n": n, "k": k, "max_rel_error_corner": rel}
    if args.steps:
        out.update(ms_total=t_all, ms_mma=t_mma, bf16_tflops_mma=6 * fl / (t_mma * 1e-3) / 1e12,
                   fp64_equivalent_tflops_mma=fl / (t_mma * 1e-3) / 1e12)
    print(json.dumps(out), flush=True)


def main():
    args = parse()
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        run_reference(args, rank, world)
        return
    if args.workload == "grouped":
        run_grouped(args)
    elif args.workload == "serving":
        run_serving(args)
    elif args.workload == "quench":
        run_quench(args)
    elif args.workload == "sample":
        run_sample(args)
    elif args.workload == "split_gemm":
        run_split_gemm(args)
    else:
        run_gpu(args, rank, world, local_rank)


if __name__ == "__main__":
    main()
