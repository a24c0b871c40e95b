#!/usr/bin/env python
"""Benchmark of the W4A4 int4 dual-scale hot path (decode-shaped GEMM sweep).

    python bench.py --gpus N --steps K --warmup W            # this library, on the GPU(s)
    python bench.py --impl reference --steps K --warmup W    # the CPU path, host cores

Workload (N=1): every linear of one Llama-3.1-8B-architecture layer (qkv 4096->6144,
o 4096->4096, gate+up 4096->28672, down 14336->4096) at M in {1, 8, 16, 32, 64, 128}, int4
weights in groups of 128 with fp16 group scales, DualQuant row scale r and column scale 1/c,
per-token int4 activations with an fp16 scale, fp32 output.  One "step" is one pass over all
24 (linear, M) pairs: activation quantiser + GEMM each.  The metric is decode GB/s: algorithmic
bytes of the step (packed weights + group scales + r + c + bf16 X + fp32 Y) divided by time.
Each M value uses its own copy of the four weight matrices (6 x 109 MB = 655 MB in rotation,
5x the 126 MB L2), so every launch streams its weights from HBM.

With N > 1 ranks each rank owns a contiguous N/ranks slice of the output rows of every weight
(column-parallel, no collective); the reported value is total bytes over the slowest rank.
"""
from __future__ import annotations

import argparse
import dataclasses
import json
import os
import statistics
import subprocess
import sys
import time

import torch

ROOT = os.path.dirname(os.path.abspath(__file__))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

from dualquant_b200 import sharding, synthetic  # noqa: E402

METRIC = "w4a4_int4_decode_gemm_sweep_GBps"
UNIT = "GB/s"
WORKLOAD = "config1: Llama-3.1-8B layer linears (qkv,o,gate_up,down) x M{1,8,16,32,64,128}, int4 dual-scale, G=128"


def _step_bytes(n_split: int = 1) -> int:
    total = 0
    for _, K, N in synthetic.LLAMA31_8B_LINEARS:
        for M in synthetic.DECODE_M:
            for rank in range(n_split):
                lo, hi = sharding.shard_rows(N, n_split, rank)
                total += synthetic.int4_gemm_bytes(M, hi - lo, K)
    return total


def bench_config(world: int) -> dict:
    """The workload description; both arms (this library and --impl reference) print exactly
    this object."""
    return {
        "workload": WORKLOAD,
        "linears": {name: [K, N] for name, K, N in synthetic.LLAMA31_8B_LINEARS},
        "M": list(synthetic.DECODE_M),
        "step": "one pass over all 24 (linear, M) pairs: per-token activation quantisation + dual-scale GEMM, "
                "bf16 X in, fp32 Y out",
        "seed": 0,
        "n_split": world,
        "parallelism": f"column-parallel over N x{world}, no collective",
        "step_algorithmic_bytes": _step_bytes(world),
    }


def _peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(path):
        with open(path) as f:
            return json.load(f), "measured"
    return {"hbm_gbs": 6650.0, "bf16_tflops": 1590.0}, "fallback"


class ClockSampler:
    """nvidia-smi clock / throttle-reason samples taken while the timed regions run.  A reader
    thread collects lines; start() returns once the first sample has arrived so that the (short)
    timed regions are covered."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.gpu_index = gpu_index
        self.proc = None
        self.lines = []
        self.stamps = []
        self.thread = None

    def start(self):
        import threading

        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-i", str(self.gpu_index), "-lms", "20"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except OSError:
            self.proc = None
            return

        def reader():
            for line in self.proc.stdout:
                self.lines.append(line)
                self.stamps.append(time.time())

        self.thread = threading.Thread(target=reader, daemon=True)
        self.thread.start()
        t0 = time.time()
        while not self.lines and time.time() - t0 < 5.0:
            time.sleep(0.01)

    def median_sm_mhz(self, t0: float, t1: float):
        """Median SM clock of the samples that arrived in the wall-clock window [t0, t1]."""
        vals = []
        for line, ts in zip(list(self.lines), list(self.stamps)):
            if t0 <= ts <= t1:
                p = [v.strip() for v in line.split(",")]
                try:
                    vals.append(float(p[1]))
                except (ValueError, IndexError):
                    pass
        return statistics.median(vals) if vals else None

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        if self.thread is not None:
            self.thread.join(timeout=2)
        sm, smax, reasons = [], [], set()
        names = ("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap")
        for line in list(self.lines):
            p = [v.strip() for v in line.split(",")]
            if len(p) < 9:
                continue
            try:
                sm.append(float(p[1]))
                smax.append(float(p[2]))
            except ValueError:
                continue
            for name, val in zip(names, p[5:9]):
                if val.lower() == "active":
                    reasons.add(name)
        return {"sm_mhz": statistics.median(sm) if sm else None,
                "sm_max_mhz": max(smax) if smax else None,
                "samples": len(sm), "reasons": sorted(reasons)}


# ------------------------------------------------------------------------------------------------
# GPU arm
# ------------------------------------------------------------------------------------------------
class Workload:
    def __init__(self, dev, rank: int, world: int, seed: int = 0):
        from dualquant_b200 import ops

        self.ops = ops
        self.dev = dev
        self.world = world
        g = torch.Generator(device=dev).manual_seed(seed)
        self.linears = []  # per linear: dict(name,K,N_local,a,r,weights[copy])
        n_copies = len(synthetic.DECODE_M)
        for name, K, N in synthetic.LLAMA31_8B_LINEARS:
            n_lo, n_hi = sharding.shard_rows(N, world, rank)
            nl = n_hi - n_lo
            r, c = synthetic.make_scales(N, K, seed)
            a = (1.0 / c).to(dev)
            r_local = r[n_lo:n_hi].contiguous().to(dev)
            copies = []
            for _ in range(n_copies):
                w = (torch.randn(nl, K, generator=g, device=dev) * 0.02).to(torch.bfloat16)
                codes, sw = ops.quant_w_int4(w)
                copies.append(ops.pack_w_int4(codes, sw))
                del w, codes, sw
            self.linears.append({"name": name, "K": K, "N": nl, "a": a, "r": r_local, "w": copies})
        # All activations of a step live in one device buffer (and one pinned host buffer), all
        # outputs in another, so that the end-to-end path moves them with one copy each way.
        self.x, self.x_host, self.y, self.y_host, self.scratch = {}, {}, {}, {}, {}
        x_keys = []
        for M in synthetic.DECODE_M:
            for lin in self.linears:
                if (M, lin["K"]) not in x_keys:
                    x_keys.append((M, lin["K"]))
        x_elems = sum(M * K for M, K in x_keys)
        y_elems = sum(M * lin["N"] for M in synthetic.DECODE_M for lin in self.linears)
        self.x_all_host = torch.empty(x_elems, dtype=torch.bfloat16).pin_memory()
        self.x_all = torch.empty(x_elems, dtype=torch.bfloat16, device=dev)
        self.y_all_host = torch.empty(y_elems, dtype=torch.float32).pin_memory()
        self.y_all = torch.empty(y_elems, dtype=torch.float32, device=dev)
        off = 0
        self.x_chunk, self.y_chunk = {}, {}  # per M: (offset, elements) of its slice of x_all / y_all
        self.x_off, self.y_off = {}, {}  # (M, K) / (M, linear): (offset, elements) in x_all / y_all
        for M, K in x_keys:
            self.x_off[(M, K)] = (off, M * K)
            lo, n = self.x_chunk.get(M, (off, 0))
            self.x_chunk[M] = (lo, n + M * K)
            self.x_all_host[off:off + M * K].copy_(synthetic.make_x(M, K, seed).reshape(-1))
            self.x_host[(M, K)] = self.x_all_host[off:off + M * K].view(M, K)
            self.x[(M, K)] = self.x_all[off:off + M * K].view(M, K)
            off += M * K
        self.x_all.copy_(self.x_all_host)
        off = 0
        for M in synthetic.DECODE_M:
            for lin in self.linears:
                K, nl = lin["K"], lin["N"]
                self.y_off[(M, lin["name"])] = (off, M * nl)
                lo, n = self.y_chunk.get(M, (off, 0))
                self.y_chunk[M] = (lo, n + M * nl)
                self.y[(M, lin["name"])] = self.y_all[off:off + M * nl].view(M, nl)
                self.y_host[(M, lin["name"])] = self.y_all_host[off:off + M * nl].view(M, nl)
                off += M * nl
                nbytes = ops.linear_scratch_bytes(M, nl, K)
                self.scratch[(M, lin["name"])] = torch.empty(nbytes, dtype=torch.uint8, device=dev)
        torch.cuda.synchronize(dev)

    def step_m(self, mi):
        """The four linears of one batch size M = DECODE_M[mi]."""
        ops = self.ops
        M = synthetic.DECODE_M[mi]
        for lin in self.linears:
            ops.linear_w4a4_int4(self.x[(M, lin["K"])], lin["a"], None, lin["w"][mi], lin["r"],
                                 scale_fp16=True, scratch=self.scratch[(M, lin["name"])],
                                 out=self.y[(M, lin["name"])])

    def step_unit(self, mi, li):
        """One (batch size, linear) pair."""
        M = synthetic.DECODE_M[mi]
        lin = self.linears[li]
        self.ops.linear_w4a4_int4(self.x[(M, lin["K"])], lin["a"], None, lin["w"][mi], lin["r"],
                                  scale_fp16=True, scratch=self.scratch[(M, lin["name"])],
                                  out=self.y[(M, lin["name"])])

    def step(self):
        """Device-resident pass: quantiser + GEMM for all 24 (linear, M) pairs."""
        for mi in range(len(synthetic.DECODE_M)):
            self.step_m(mi)

    def prequantise(self):
        ops = self.ops
        self.q = {}
        for M in synthetic.DECODE_M:
            for lin in self.linears:
                self.q[(M, lin["name"])] = ops.quant_act_int4(self.x[(M, lin["K"])], lin["a"], None, True)

    def gemm_only_step(self):
        ops = self.ops
        for mi, M in enumerate(synthetic.DECODE_M):
            for lin in self.linears:
                codes, sx = self.q[(M, lin["name"])]
                ops.gemm_w4a4_int4(codes, sx, lin["w"][mi], lin["r"], out=self.y[(M, lin["name"])])

    def e2e_units(self):
        """The step's (batch size, linear) pairs in end-to-end order: largest batch first and, inside
        a batch, the linear with the largest output first, so that the downloads (the 42.8 MB of fp32
        outputs are what bounds the step) start as early as possible and never pause."""
        lins = sorted(range(len(self.linears)), key=lambda li: -self.linears[li]["N"])
        return [(mi, li) for mi in reversed(range(len(synthetic.DECODE_M))) for li in lins]

    def e2e_setup(self, run_unit):
        """run_unit[(mi, li)]() launches one linear (quantiser + GEMM) on the current stream."""
        self.run_unit = run_unit
        self.units = self.e2e_units()
        self.s_in = torch.cuda.Stream(device=self.dev)
        self.s_out = torch.cuda.Stream(device=self.dev)
        self.ev_in = {key: torch.cuda.Event() for key in self.x_off}
        self.ev_done = {u: torch.cuda.Event() for u in self.units}

    def e2e_step(self):
        """Host buffers in, host buffers out, every step: each activation matrix goes up from pinned
        host memory on a copy stream, each linear runs (through the C ABI) on the compute stream as
        soon as its input has landed, and its output goes down to pinned host memory on a second
        copy stream while the following linears compute.  The step ends when the last output byte
        is in host memory."""
        cur = torch.cuda.current_stream(self.dev)
        self.s_in.wait_stream(cur)   # not before the previous step has ended
        self.s_out.wait_stream(cur)
        with torch.cuda.stream(self.s_in):
            seen = set()
            for mi, li in self.units:
                key = (synthetic.DECODE_M[mi], self.linears[li]["K"])
                if key in seen:
                    continue
                seen.add(key)
                lo, n = self.x_off[key]
                self.x_all[lo:lo + n].copy_(self.x_all_host[lo:lo + n], non_blocking=True)
                self.ev_in[key].record(self.s_in)
        for u in self.units:
            mi, li = u
            M, lin = synthetic.DECODE_M[mi], self.linears[li]
            cur.wait_event(self.ev_in[(M, lin["K"])])
            self.run_unit[u]()
            self.ev_done[u].record(cur)
            with torch.cuda.stream(self.s_out):
                self.s_out.wait_event(self.ev_done[u])
                lo, n = self.y_off[(M, lin["name"])]
                self.y_all_host[lo:lo + n].copy_(self.y_all[lo:lo + n], non_blocking=True)
        cur.wait_stream(self.s_out)

    def e2e_bytes(self):
        return self.x_all.numel() * 2, self.y_all.numel() * 4


def _capture(fn, dev):
    """CUDA graph of one call of fn (after a warm-up on a side stream)."""
    s = torch.cuda.Stream(device=dev)
    s.wait_stream(torch.cuda.current_stream(dev))
    with torch.cuda.stream(s):
        fn()
    torch.cuda.current_stream(dev).wait_stream(s)
    torch.cuda.synchronize(dev)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        fn()
    return graph


def _time_loop(run, steps, warmup, dev, barrier):
    for _ in range(warmup):
        run()
    torch.cuda.synchronize(dev)
    barrier()
    torch.cuda.synchronize(dev)
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(steps):
        run()
    e1.record()
    torch.cuda.synchronize(dev)
    barrier()
    return e0.elapsed_time(e1)  # ms


def _kernel_class(M: int) -> str:
    """Which GEMM kernel dq_gemm_w4a4_int4 runs for a batch of M tokens."""
    if M <= 8:
        return "gemv_w4a4_int4_kernel<1> (mma.sync.s8, 8-token capacity)"
    if M <= 16:
        return "gemv_w4a4_int4_kernel<2> (mma.sync.s8, 16-token capacity)"
    if M <= 32:
        return "gemm_w4a4_int4_tm_kernel<32> (tcgen05 kind::i8, weights via tensor memory)"
    if M <= 64:
        return "gemm_w4a4_int4_tm_kernel<64> (tcgen05 kind::i8, weights via tensor memory)"
    return "gemm_w4a4_int4_kernel<128> / gemm_w4a4_int4_tm_kernel<64> (tcgen05 kind::i8, by estimated cost)"


def _traffic_table():
    """ncu DRAM traffic per launch of each decode kernel class (profiles/decode_kernel_traffic.json,
    written from ncu captures of `bench.py --case NAME:M`); {} when the file is absent."""
    path = os.path.join(ROOT, "profiles", "decode_kernel_traffic.json")
    if not os.path.exists(path):
        return {}
    with open(path) as f:
        return json.load(f)


def _sustained(run, ms_per_step, dev, barrier, max_over_ranks, sampler, reps=5, target_s=0.2):
    """`reps` timed loops of at least `target_s` seconds of GPU time each (the K-step loop of the
    contract lasts a few milliseconds): ms/step of every repeat and the SM clock sampled during it."""
    n = max(10, int(target_s * 1e3 / max(ms_per_step, 1e-3)) + 1)
    out, clocks = [], []
    for _ in range(reps):
        t0 = time.time()
        ms = max_over_ranks(_time_loop(run, n, 1, dev, barrier)) / n
        t1 = time.time()
        out.append(ms)
        clocks.append(sampler.median_sm_mhz(t0, t1) if sampler is not None else None)
    return n, out, clocks


def run_gpu(args):
    import torch.distributed as dist

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    if world != args.gpus:
        if world == 1 and args.gpus > 1:
            raise SystemExit("launch with torch.distributed.run --nproc-per-node N for --gpus N")
    if not torch.cuda.is_available():
        raise SystemExit("bench.py: no CUDA device; the library has no CPU path "
                         "(use --impl reference for the CPU baseline)")
    torch.cuda.set_device(local_rank)
    dev = torch.device("cuda", local_rank)
    if world > 1:
        dist.init_process_group("nccl", device_id=dev)

    def barrier():
        if world > 1:
            dist.barrier(device_ids=[local_rank])

    def max_over_ranks(ms):
        if world == 1:
            return ms
        t = torch.tensor([ms], dtype=torch.float64, device=dev)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        return float(t.item())

    from dualquant_b200 import _lib

    wl = Workload(dev, rank, world, seed=0)
    step_bytes = _step_bytes(world)
    n_lin = len(wl.linears)
    n_m = len(synthetic.DECODE_M)
    launches_per_step = 2 * n_m * n_lin  # activation quantiser + GEMM per linear
    peaks, peak_kind = _peaks()
    hbm = peaks["hbm_gbs"]

    # ---- device-resident: CUDA graph of one step ---------------------------------------------
    graph = _capture(wl.step, dev) if not args.no_graph else None
    run = graph.replay if graph is not None else wl.step
    sampler = ClockSampler(local_rank) if rank == 0 else None
    if sampler is not None:
        sampler.start()
    ms = max_over_ranks(_time_loop(run, args.steps, args.warmup, dev, barrier))
    ms_per_step = ms / args.steps
    value = step_bytes / (ms_per_step * 1e-3) / 1e9
    n_rep, rep_ms, rep_clk = _sustained(run, ms_per_step, dev, barrier, max_over_ranks, sampler)
    sustained = {
        "steps_per_repeat": n_rep, "repeats": len(rep_ms),
        "value_median": round(step_bytes / (statistics.median(rep_ms) * 1e-3) / 1e9, 1),
        "value_min": round(step_bytes / (max(rep_ms) * 1e-3) / 1e9, 1),
        "value_max": round(step_bytes / (min(rep_ms) * 1e-3) / 1e9, 1),
        "ms_per_step": [round(v, 4) for v in rep_ms], "sm_mhz": rep_clk,
    }

    # ---- GEMM launches alone, per kernel class (one class per batch size) ---------------------
    wl.prequantise()
    traffic = _traffic_table()
    classes = []
    gemm_ms_total = 0.0
    for mi, M in enumerate(synthetic.DECODE_M):
        def gemm_m(mi=mi, M=M):
            for c in range(len(wl.linears[0]["w"])):  # cycle the weight copies: every launch reads HBM
                for lin in wl.linears:
                    codes, sx = wl.q[(M, lin["name"])]
                    wl.ops.gemm_w4a4_int4(codes, sx, lin["w"][(mi + c) % n_m], lin["r"], out=wl.y[(M, lin["name"])])
        gm = _capture(gemm_m, dev) if not args.no_graph else None
        n_launch = n_lin * n_m
        ms_m = max_over_ranks(_time_loop(gm.replay if gm is not None else gemm_m, max(args.steps // 2, 5),
                                         args.warmup, dev, barrier)) / max(args.steps // 2, 5)
        bytes_m = sum(synthetic.int4_gemm_bytes(M, lin["N"], lin["K"]) for lin in wl.linears)  # this rank, 4 launches
        us = ms_m * 1e3 / n_launch
        ach = bytes_m / n_lin / (us * 1e-6) / 1e9
        gemm_ms_total += ms_m / n_m  # one pass over the four linears of this M
        rec = {"kernel": _kernel_class(M), "M": M, "launches_per_step": n_lin,
               "algorithmic_bytes_per_launch": bytes_m // n_lin, "us_per_launch": round(us, 2),
               "achieved": round(ach, 1), "frac": round(ach / hbm, 4)}
        t = traffic.get(f"M{M}")
        if t is not None and world == 1:
            rec["traffic"] = t.get("dram_bytes_per_launch")
            rec["traffic_case"] = t.get("case")
            rec["traffic_case_algorithmic_bytes"] = t.get("algorithmic_bytes_per_launch")
        classes.append(rec)
        del gm
    n_gemm = n_m * n_lin
    achieved = step_bytes / world / (gemm_ms_total * 1e-3) / 1e9  # per GPU, all GEMM launches of a step
    dom = max(classes, key=lambda r: r["us_per_launch"] * r["launches_per_step"])
    roofline = {
        "bound": "hbm", "kernel": dom["kernel"], "achieved": dom["achieved"], "peak": hbm,
        "peak_kind": peak_kind, "unit": "GB/s", "frac": dom["frac"],
        "traffic": dom.get("traffic"), "traffic_case": dom.get("traffic_case"),
        "traffic_case_algorithmic_bytes": dom.get("traffic_case_algorithmic_bytes"),
        "algorithmic_bytes_per_launch": dom["algorithmic_bytes_per_launch"],
        "avg_launch_us": dom["us_per_launch"],
        "note": "the class with the largest share of the step's GEMM time; every class is listed in `classes`",
        "all_gemm_launches": {"achieved": round(achieved, 1), "frac": round(achieved / hbm, 4),
                              "avg_launch_us": round(gemm_ms_total * 1e3 / n_gemm, 2),
                              "algorithmic_bytes_per_launch": step_bytes // world // n_gemm},
        "quantiser": {"kernel": "act_quant_rows_kernel", "launches_per_step": n_gemm,
                      "us_per_launch": round(max(ms_per_step - gemm_ms_total, 0.0) * 1e3 / n_gemm, 2),
                      "note": "step time minus GEMM-only time, per launch (latency-bound at decode sizes)"},
        "classes": classes,
    }

    # ---- end to end through the C ABI with host buffers -----------------------------------------
    units = wl.e2e_units()
    if args.no_graph:
        run_unit = {u: (lambda u=u: wl.step_unit(*u)) for u in units}
    else:
        graphs_u = {u: _capture(lambda u=u: wl.step_unit(*u), dev) for u in units}
        run_unit = {u: g_.replay for u, g_ in graphs_u.items()}
    wl.e2e_setup(run_unit)
    ms3 = max_over_ranks(_time_loop(wl.e2e_step, args.steps, args.warmup, dev, barrier)) / args.steps
    h2d, d2h = wl.e2e_bytes()
    e2e = {"value": round(step_bytes / (ms3 * 1e-3) / 1e9, 1), "unit": UNIT,
           "ms_per_step": round(ms3, 4), "h2d_bytes_per_step": h2d * world,
           "d2h_bytes_per_step": d2h * world,
           "copies": "per linear, on two copy streams, overlapped with the other linears; largest outputs first"}
    # clock samples cover the timed regions above
    clocks = sampler.stop() if sampler is not None else None
    _lib.device_status(local_rank)

    per_shape = per_shape_detail(wl, dev, args) if (world == 1 and not args.no_detail) else None
    del wl, graph
    torch.cuda.empty_cache()

    # ---- the other benchmark configurations, as sub-records of the same line -------------------
    extras = {}
    if not args.no_extras:
        extras = run_extras(args, world, rank, local_rank, dev)

    if rank == 0:
        line = {
            "metric": METRIC, "value": round(value, 1), "unit": UNIT, "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(ms_per_step, 4),
            "higher_is_better": True, "scaling": "strong", "vs_baseline": None,
            "dtype": "int4xint4->int32 (kind::i8 / mma.sync.s8), fp32 epilogue",
            "data": "synthetic", "impl": "dualquant_b200",
            "config": bench_config(world),
            "arm": {"l2": "6 weight copies in rotation (655 MB > 5x L2): inputs larger than L2",
                    "launch": "CUDA graph replay of one step" if not args.no_graph else "stream launches"},
            "sustained": sustained,
            "roofline": roofline,
            "e2e": e2e,
            "gpu_launches": launches_per_step * args.steps,
            "clocks": clocks,
        }
        if per_shape is not None:
            line["per_shape_gemm_GBps"] = per_shape
            line["per_shape_frac_of_hbm"] = {k: [round(v / hbm, 3) for v in row] for k, row in per_shape.items()}
        line.update(extras)
        if not args.skip_cpu:
            line["cpu_baseline"] = cpu_baseline(budget_s=args.cpu_budget)
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.destroy_process_group()


def run_extras(args, world, rank, local_rank, dev):
    """Benchmark configurations 0, 2, 3 and 4 measured in the same run.  One GPU: prefill int4
    (TOPS), the config-2 MLP, block-scaled FP4 and the 32-layer decoder.  N GPUs: the decoder,
    tensor-parallel over the N ranks with the all-reduce fused into the decode GEMM.  A suite that
    fails reports its error text instead of numbers."""
    out = {}

    def guarded(name, fn):
        try:
            out[name] = fn()
        except Exception as exc:  # noqa: BLE001 - the headline line must still be printed
            out[name] = {"error": f"{type(exc).__name__}: {exc}"[:300]}
        torch.cuda.empty_cache()

    sub = argparse.Namespace(**vars(args))
    sub.steps = max(5, min(args.steps, 10))
    if world == 1:
        guarded("peaks_mma_only", lambda: run_peak_suite(sub, emit=False))
        guarded("prefill", lambda: run_prefill_suite(sub, emit=False))
        guarded("mlp", lambda: run_mlp_suite(sub, emit=False))
        guarded("fp4", lambda: run_fp4_suite(sub, emit=False))
        guarded("reference_gpu_kernels", lambda: run_reference_gpu(sub, emit=False))
        guarded("bcd", lambda: run_bcd_suite(sub, emit=False))
    sub.fused_allreduce = True
    try:
        out["decoder"] = run_decoder_suite(sub, emit=False, init_pg=False)
    except Exception as exc:  # noqa: BLE001
        out["decoder"] = {"error": f"{type(exc).__name__}: {exc}"[:300]}
    return out if rank == 0 else {}


def run_case(args):
    """One (linear, M) pair alone, a handful of launches: the small case profilers capture.
    --case NAME:M[:TN:SPLIT], e.g. gate_up:16 ; --iters launches after 3 warm-up launches.
    Other forms: e4m3:NAME:M, a16w4:NAME:M, linear:NAME:M, fp4:FMT:NAME:M, quant:M:K, quant_had:M:K,
    quant_fp4:FMT:M:K."""
    from dualquant_b200 import _lib, ops

    parts = args.case.split(":")
    if parts[0] in ("quant", "quant_had"):  # quant:M:K - the int4 activation quantiser alone
        from dualquant_b200 import _lib as _l, ops as _ops, quarot as _q

        M, K = int(parts[1]), int(parts[2])
        dev = torch.device("cuda", 0)
        torch.cuda.set_device(dev)
        had = None
        if parts[0] == "quant_had":  # with the full online Hadamard of size K (QuaRot R4)
            hk, kk = _q.get_hadK(K)
            had = _ops.Hadamard(_l.HAD_FULL, kk, 0, _q.full_hadamard_scale(K), None if hk is None else hk.to(dev))
        n_bufs = max(2, int(400e6 // (M * K * 2)) + 1)
        xs = [torch.randn(M, K, device=dev).to(torch.bfloat16) for _ in range(n_bufs)]
        a = torch.rand(K, device=dev) + 0.5
        for i in range(3):
            _ops.quant_act_int4(xs[i % n_bufs], a, had, True)
        torch.cuda.synchronize()
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record()
        for i in range(args.iters):
            _ops.quant_act_int4(xs[i % n_bufs], a, had, True)
        e1.record()
        torch.cuda.synchronize()
        ms = e0.elapsed_time(e1) / args.iters
        b = M * K * 3 + 4 * K + 4 * M
        print(json.dumps({"case": args.case, "us_per_launch": round(ms * 1e3, 2), "algorithmic_bytes": b,
                          "GBps": round(b / ms / 1e6, 1)}), flush=True)
        return
    if parts[0] == "quant_fp4":  # quant_fp4:FMT:M:K - the FP4 activation quantiser alone
        fmt = {"mxfp4": _lib.FP4_MXFP4, "nvfp4": _lib.FP4_NVFP4}[parts[1]]
        M, K = int(parts[2]), int(parts[3])
        dev = torch.device("cuda", 0)
        torch.cuda.set_device(dev)
        n_bufs = max(2, int(400e6 // (M * K * 2)) + 1)
        xs = [torch.randn(M, K, device=dev).to(torch.bfloat16) for _ in range(n_bufs)]
        a = torch.rand(K, device=dev) + 0.5
        for i in range(3):
            ops.quant_fp4(xs[i % n_bufs], fmt, a, None, atoms=True)
        torch.cuda.synchronize()
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record()
        for i in range(args.iters):
            ops.quant_fp4(xs[i % n_bufs], fmt, a, None, atoms=True)
        e1.record()
        torch.cuda.synchronize()
        ms = e0.elapsed_time(e1) / args.iters
        blk = 32 if fmt == _lib.FP4_MXFP4 else 16
        b = M * K * 2 + M * K // 2 + M * K // blk + 4 * K
        print(json.dumps({"case": args.case, "us_per_launch": round(ms * 1e3, 2), "algorithmic_bytes": b,
                          "GBps": round(b / ms / 1e6, 1)}), flush=True)
        return
    if parts[0] == "fp4":  # fp4:FMT:LINEAR:M - one block-scaled FP4 GEMM of the Qwen2.5-7B shapes alone
        fmt = {"mxfp4": _lib.FP4_MXFP4, "nvfp4": _lib.FP4_NVFP4}[parts[1]]
        K, N = {n: (k, nn) for n, k, nn in synthetic.QWEN25_7B_LINEARS}[parts[2]]
        M = int(parts[3])
        blk = 32 if fmt == _lib.FP4_MXFP4 else 16
        dev = torch.device("cuda", 0)
        torch.cuda.set_device(dev)
        g = torch.Generator(device=dev).manual_seed(0)
        w = (torch.randn(N, K, generator=g, device=dev) * 0.02).to(torch.bfloat16)
        pw = ops.pack_w_fp4(w, fmt)
        del w
        r, c = synthetic.make_scales(N, K, 0)
        r, a = r.to(dev), (1.0 / c).to(dev)
        x = torch.randn(M, K, generator=g, device=dev).to(torch.bfloat16)
        codes, sfa, rs = _fp4_prologue(ops, x, a, pw)
        y = torch.empty(M, N, dtype=torch.float32, device=dev)
        for _ in range(3):
            ops.gemm_w4a4_fp4(codes, sfa, rs, pw, r, out=y)
        torch.cuda.synchronize()
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(args.iters):
            ops.gemm_w4a4_fp4(codes, sfa, rs, pw, r, out=y)
        e1.record()
        torch.cuda.synchronize()
        _lib.device_status(0)
        ms = e0.elapsed_time(e1) / args.iters
        nbytes = N * K // 2 + N * K // blk + 2 * N + 2 * K + 2 * M * K + 4 * M * N
        print(json.dumps({"case": args.case, "iters": args.iters, "us_per_launch": round(ms * 1e3, 2),
                          "TFLOPS": round(2.0 * M * N * K / ms / 1e9, 1), "algorithmic_bytes": nbytes,
                          "GBps": round(nbytes / ms / 1e6, 1)}), flush=True)
        return
    if parts[0] == "e4m3":  # e4m3:NAME:M - the FP8-path int4 GEMM alone (E4M3 codes, bf16 out)
        name, M = parts[1], int(parts[2])
        K, N = {n: (k, nn) for n, k, nn in synthetic.LLAMA31_8B_LINEARS}[name]
        dev = torch.device("cuda", 0)
        torch.cuda.set_device(dev)
        g = torch.Generator(device=dev).manual_seed(0)
        w = (torch.randn(N, K, generator=g, device=dev) * 0.02).to(torch.bfloat16)
        cw, sw = ops.quant_w_int4(w)
        pw = ops.pack_w_int4(cw, sw)
        del w, cw, sw
        r, c = synthetic.make_scales(N, K, 0)
        x8, sx = ops.quant_act_int4(synthetic.make_x(M, K, 0).to(dev), (1.0 / c).to(dev), None, True, e4m3=True)
        w8, rr = pw.bytes_e4m3(), r.to(dev)
        y = torch.empty(M, N, dtype=torch.bfloat16, device=dev)
        for _ in range(3):
            ops.gemm_w4a4_int4_e4m3(x8, sx, w8, pw, rr, out=y)
        torch.cuda.synchronize()
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(args.iters):
            ops.gemm_w4a4_int4_e4m3(x8, sx, w8, pw, rr, out=y)
        e1.record()
        torch.cuda.synchronize()
        _lib.device_status(0)
        ms = e0.elapsed_time(e1) / args.iters
        print(json.dumps({"case": args.case, "iters": args.iters, "us_per_launch": round(ms * 1e3, 2),
                          "TOPS": round(2.0 * M * N * K / ms / 1e9, 1),
                          "operand_bytes": N * K + M * K + 2 * M * N}), flush=True)
        return
    if parts[0] in ("a16w4", "linear"):  # a16w4:NAME:M / linear:NAME:M - one whole linear alone
        name, M = parts[1], int(parts[2])
        K, N = {n: (k, nn) for n, k, nn in synthetic.LLAMA31_8B_LINEARS}[name]
        dev = torch.device("cuda", 0)
        torch.cuda.set_device(dev)
        g = torch.Generator(device=dev).manual_seed(0)
        n_copies = max(2, int(300e6 // (N * K // 2)) + 1) if M <= 128 else 1
        copies = []
        for _ in range(n_copies):
            w = (torch.randn(N, K, generator=g, device=dev) * 0.02).to(torch.bfloat16)
            cw, sw = ops.quant_w_int4(w)
            copies.append(ops.pack_w_int4(cw, sw))
            del w, cw, sw
        r, c = synthetic.make_scales(N, K, 0)
        r, a = r.to(dev), (1.0 / c).to(dev)
        x = synthetic.make_x(M, K, 0).to(dev)
        if parts[0] == "a16w4":
            y = torch.empty(M, N, dtype=torch.bfloat16, device=dev)
            scratch = torch.empty(M * K * 2 + 256, dtype=torch.uint8, device=dev)
            call = lambda pw: ops.linear_a16w4(x, a, pw, r, scratch=scratch, out=y)  # noqa: E731
        else:
            y = torch.empty(M, N, dtype=torch.float32, device=dev)
            scratch = torch.empty(max(256, ops.linear_scratch_bytes(M, N, K)), dtype=torch.uint8, device=dev)
            call = lambda pw: ops.linear_w4a4_int4(x, a, None, pw, r, scale_fp16=True, scratch=scratch, out=y)  # noqa: E731
        for i in range(3):
            call(copies[i % n_copies])
        torch.cuda.synchronize()
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record()
        for i in range(args.iters):
            call(copies[i % n_copies])
        e1.record()
        torch.cuda.synchronize()
        _lib.device_status(0)
        ms = e0.elapsed_time(e1) / args.iters
        print(json.dumps({"case": args.case, "iters": args.iters, "us_per_call": round(ms * 1e3, 2),
                          "TOPS": round(2.0 * M * N * K / ms / 1e9, 1),
                          "GBps": round(synthetic.int4_gemm_bytes(M, N, K) / ms / 1e6, 1)}), flush=True)
        return
    name, M = parts[0], int(parts[1])
    tn = int(parts[2]) if len(parts) > 2 else 0
    split = int(parts[3]) if len(parts) > 3 else 0
    K, N = {n: (k, nn) for n, k, nn in synthetic.LLAMA31_8B_LINEARS}[name]
    dev = torch.device("cuda", 0)
    torch.cuda.set_device(dev)
    g = torch.Generator(device=dev).manual_seed(0)
    copies = []
    n_copies = max(3, int(300e6 // (N * K // 2)) + 1)
    for _ in range(n_copies):
        w = (torch.randn(N, K, generator=g, device=dev) * 0.02).to(torch.bfloat16)
        codes, sw = ops.quant_w_int4(w)
        copies.append(ops.pack_w_int4(codes, sw))
        del w, codes, sw
    r, c = synthetic.make_scales(N, K, 0)
    x = synthetic.make_x(M, K, 0).to(dev)
    qx, sx = ops.quant_act_int4(x, (1.0 / c).to(dev), None, True)
    y = torch.empty(M, N, dtype=torch.float32, device=dev)
    rr = r.to(dev)
    for i in range(3):
        ops.gemm_w4a4_int4(qx, sx, copies[i % n_copies], rr, out=y, token_tile=tn, split_k=split)
    torch.cuda.synchronize()
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record()
    for i in range(args.iters):
        ops.gemm_w4a4_int4(qx, sx, copies[i % n_copies], rr, out=y, token_tile=tn, split_k=split)
    e1.record()
    torch.cuda.synchronize()
    _lib.device_status(0)
    ms = e0.elapsed_time(e1) / args.iters
    b = synthetic.int4_gemm_bytes(M, N, K)
    print(json.dumps({"case": args.case, "iters": args.iters, "us_per_launch": round(ms * 1e3, 2),
                      "algorithmic_bytes": b, "GBps": round(b / ms / 1e6, 1),
                      "weight_copies": n_copies}), flush=True)


PREFILL_SHAPES = (
    # (label, M, K, N)
    ("config0 linear", 2048, 4096, 4096),
    ("qkv", 4096, 4096, 6144),
    ("gate_up", 4096, 4096, 28672),
    ("down", 4096, 14336, 4096),
    ("config2 gate_up", 8192, 4096, 28672),
    ("config2 down", 8192, 14336, 4096),
)


def run_prefill_suite(args, emit=True):
    """Prefill-shaped linears (tensor-core bound): TOPS = 2*M*N*K / time of the GEMM launch and of
    quantiser + GEMM, against the dense 8-bit peak (nominal 4500 TOPS; 2x the measured bf16 peak;
    the MMA-only ceiling measured by the probe kernel)."""
    from dualquant_b200 import _lib, ops

    dev = torch.device("cuda", 0)
    torch.cuda.set_device(dev)
    peaks, kind = _peaks()
    int8_measured = 2.0 * peaks["bf16_tflops"]
    g = torch.Generator(device=dev).manual_seed(0)
    rows = []
    for label, M, K, N in PREFILL_SHAPES:
        w = (torch.randn(N, K, generator=g, device=dev) * 0.02).to(torch.bfloat16)
        codes_w, sw = ops.quant_w_int4(w)
        pw = ops.pack_w_int4(codes_w, sw)
        del w, codes_w, sw
        r, c = synthetic.make_scales(N, K, 0)
        r, a = r.to(dev), (1.0 / c).to(dev)
        x = (torch.randn(M, K, generator=g, device=dev)).to(torch.bfloat16)
        qx, sx = ops.quant_act_int4(x, a, None, True)
        x8, _ = ops.quant_act_int4(x, a, None, True, e4m3=True)
        w8 = pw.bytes_e4m3()
        # configuration 0 names an fp32 output; the other rows write bf16, the model's activation type
        ydt = torch.float32 if label.startswith("config0") else torch.bfloat16
        y = torch.empty(M, N, dtype=ydt, device=dev)
        scratch = torch.empty(ops.linear_scratch_bytes(M, N, K), dtype=torch.uint8, device=dev)
        # gemm: the FP8-path kernel (E4M3 operands, the weight's byte form resident); gemm_i8: the
        # kind::i8 kernel on the 4-bit artefact; linear: the one-call entry (quantiser + weight
        # expansion into scratch + FP8-path GEMM from 1024 tokens on)
        g_gemm = _capture(lambda: ops.gemm_w4a4_int4_e4m3(x8, sx, w8, pw, r, out=y), dev)
        g_i8 = _capture(lambda: ops.gemm_w4a4_int4(qx, sx, pw, r, out=y), dev)
        g_full = _capture(lambda: ops.linear_w4a4_int4(x, a, None, pw, r, scale_fp16=True,
                                                       scratch=scratch, out=y), dev)
        ms_gemm = _time_loop(g_gemm.replay, args.steps, args.warmup, dev, lambda: None) / args.steps
        ms_i8 = _time_loop(g_i8.replay, args.steps, args.warmup, dev, lambda: None) / args.steps
        ms_full = _time_loop(g_full.replay, args.steps, args.warmup, dev, lambda: None) / args.steps
        # the A16W4 variant (bf16 activations x int4 weights, tcgen05 kind::f16) on the same operands
        yb = torch.empty(M, N, dtype=torch.bfloat16, device=dev)
        s16 = torch.empty(M * K * 2 + 256, dtype=torch.uint8, device=dev)
        g_a16 = _capture(lambda: ops.linear_a16w4(x, a, pw, r, scratch=s16, out=yb), dev)
        ms_a16 = _time_loop(g_a16.replay, args.steps, args.warmup, dev, lambda: None) / args.steps
        del g_a16, yb, s16
        ops_ = 2.0 * M * N * K
        rows.append({"shape": label, "M": M, "K": K, "N": N, "y_dtype": "fp32" if ydt == torch.float32 else "bf16",
                     "a16w4_linear_us": round(ms_a16 * 1e3, 1), "a16w4_TFLOPS": round(ops_ / ms_a16 / 1e9, 1),
                     "gemm_kernel": "gemm_w4a4_e4m3_kernel (tcgen05 kind::f8f6f4, E4M3 codes)",
                     "gemm_us": round(ms_gemm * 1e3, 1), "gemm_TOPS": round(ops_ / ms_gemm / 1e9, 1),
                     "gemm_i8_us": round(ms_i8 * 1e3, 1), "gemm_i8_TOPS": round(ops_ / ms_i8 / 1e9, 1),
                     "linear_us": round(ms_full * 1e3, 1), "linear_TOPS": round(ops_ / ms_full / 1e9, 1),
                     "frac_int8_nominal": round(ops_ / ms_gemm / 1e9 / 4500.0, 4),
                     "frac_2x_measured_bf16": round(ops_ / ms_gemm / 1e9 / int8_measured, 4)})
        del x8, w8, g_gemm, g_i8, g_full
        del pw, x, qx, sx, y, scratch
    _lib.device_status(0)
    # "reference on this box": what the reference's PermLinear ends in - a bf16 F.linear (cuBLAS) on
    # de-quantised operands of the same shapes; a library call, timed for context after all int4
    # rows (a dense bf16 GEMM runs into the power cap and would colour the row timed after it)
    for row in rows:
        M, K, N = row["M"], row["K"], row["N"]
        xb = torch.empty(M, K, dtype=torch.bfloat16, device=dev).normal_(0, 1, generator=g)
        wb = torch.empty(N, K, dtype=torch.bfloat16, device=dev).normal_(0, 0.02, generator=g)
        yb = torch.empty(M, N, dtype=torch.bfloat16, device=dev)
        g_bf16 = _capture(lambda: torch.matmul(xb, wb.t(), out=yb), dev)
        ms_bf16 = _time_loop(g_bf16.replay, args.steps, args.warmup, dev, lambda: None) / args.steps
        row["bf16_matmul_us"] = round(ms_bf16 * 1e3, 1)
        row["bf16_matmul_TFLOPS"] = round(2.0 * M * N * K / ms_bf16 / 1e9, 1)
        del xb, wb, yb, g_bf16
    mma = _mma_peaks(args)
    if mma is not None and mma.get("e4m3_TFLOPS"):
        for row in rows:
            row["frac_e4m3_mma_only_measured"] = round(row["gemm_TOPS"] / mma["e4m3_TFLOPS"], 4)
    if mma is not None and mma.get("int8_TOPS"):
        for row in rows:
            row["gemm_i8_frac_int8_mma_only_measured"] = round(row["gemm_i8_TOPS"] / mma["int8_TOPS"], 4)
    rec = {"suite": "prefill", "unit": "TOPS (2*M*N*K/s)",
           "peaks": {"int8_nominal": 4500.0, "int8_2x_bf16_" + kind: int8_measured,
                     "int8_mma_only_measured": None if mma is None else mma.get("int8_TOPS"),
                     "e4m3_mma_only_measured": None if mma is None else mma.get("e4m3_TFLOPS")},
           "steps": args.steps, "rows": rows}
    if emit:
        print(json.dumps(rec), flush=True)
    return rec


def run_mlp_suite(args, emit=True):
    """Benchmark configuration 2: prefill MLP, M = 8192 tokens, int4 dual-scale.  gate+up 4096 -> 28672
    (bf16 out), SiLU(gate) * up in bf16, QuaRot R4 online Hadamard of size 14336 (28 x 512) fused
    with the activation quantiser, down 14336 -> 4096.  Stage times from CUDA-graph replays."""
    from dualquant_b200 import _lib, ops, quarot

    dev = torch.device("cuda", 0)
    torch.cuda.set_device(dev)
    M, H, I = 8192, 4096, 14336
    g = torch.Generator(device=dev).manual_seed(0)

    def packed(N, K):
        w = (torch.randn(N, K, generator=g, device=dev) * 0.02).to(torch.bfloat16)
        c, sw = ops.quant_w_int4(w)
        return ops.pack_w_int4(c, sw)

    w_gu, w_down = packed(2 * I, H), packed(H, I)
    r_gu, c_gu = synthetic.make_scales(2 * I, H, 0)
    r_dn, c_dn = synthetic.make_scales(H, I, 1)
    r_gu, a_gu, r_dn, a_dn = r_gu.to(dev), (1.0 / c_gu).to(dev), r_dn.to(dev), (1.0 / c_dn).to(dev)
    hk, kk = quarot.get_hadK(I)
    had = ops.Hadamard(_lib.HAD_FULL, kk, 0, quarot.full_hadamard_scale(I), hk.to(dev))
    x = torch.randn(M, H, generator=g, device=dev).to(torch.bfloat16)
    gu = torch.empty(M, 2 * I, dtype=torch.bfloat16, device=dev)
    y = torch.empty(M, H, dtype=torch.bfloat16, device=dev)
    s1 = torch.empty(ops.linear_scratch_bytes(M, 2 * I, H), dtype=torch.uint8, device=dev)
    w8_down = w_down.bytes_e4m3()  # the down projection runs on the FP8-path GEMM, byte form resident
    state = {}

    def st_gate_up():
        ops.linear_w4a4_int4(x, a_gu, None, w_gu, r_gu, scale_fp16=True, scratch=s1, out=gu)

    def st_act():
        state["h"] = torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]

    def st_quant():
        state["q"] = ops.quant_act_int4(state["h"], a_dn, had, True, e4m3=True)

    def st_down():
        ops.gemm_w4a4_int4_e4m3(state["q"][0], state["q"][1], w8_down, w_down, r_dn, out=y)

    def st_fused_quant():
        state["q"] = ops.quant_act_int4_gated(gu[:, :I], gu[:, I:], a_dn, had, True, e4m3=True)

    def whole():
        st_gate_up(); st_act(); st_quant(); st_down()

    def whole_fused():
        st_gate_up(); st_fused_quant(); st_down()

    whole()
    torch.cuda.synchronize()
    out = {"suite": "mlp", "M": M, "hidden": H, "intermediate": I}
    for name, fn in (("gate_up_linear", st_gate_up), ("silu_mul_bf16_torch", st_act),
                     ("hadamard_quant", st_quant), ("silu_mul_hadamard_quant_fused", st_fused_quant),
                     ("down_gemm", st_down), ("whole_mlp_unfused", whole), ("whole_mlp", whole_fused)):
        gr = _capture(fn, dev)
        ms = _time_loop(gr.replay, args.steps, args.warmup, dev, lambda: None) / args.steps
        out[name + "_us"] = round(ms * 1e3, 1)
    ops_total = 2.0 * M * (2 * I * H + H * I)
    out["whole_mlp_TOPS"] = round(ops_total / (out["whole_mlp_us"] * 1e-6) / 1e12, 1)
    out["hadamard_quant_GBps"] = round((M * I * 3) / (out["hadamard_quant_us"] * 1e-6) / 1e9, 1)
    _lib.device_status(0)
    if emit:
        print(json.dumps(out), flush=True)
    return out


def run_decoder_suite(args, emit=True, init_pg=True):
    """Benchmark configuration 4: random-init Llama-3.1-8B-architecture decoder, every linear W4A4 int4
    dual-scale with online Hadamards, bf16 attention; prefill batch x seqlen, then decode steps.
    Tensor-parallel over the ranks of the launch (torch.distributed.run) with an NCCL all-reduce
    after o_proj and down_proj.  Prints one JSON line on rank 0."""
    import torch.distributed as dist

    from dualquant_b200 import _lib, decoder

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local_rank)
    dev = torch.device("cuda", local_rank)
    group = None
    if world > 1:
        if init_pg:
            dist.init_process_group("nccl", device_id=dev)
        group = dist.group.WORLD
    cfg = decoder.DecoderConfig(num_hidden_layers=args.layers)
    B, S, steps = args.batch, args.seqlen, args.decode_steps
    fused = bool(args.fused_allreduce) and world > 1
    model = decoder.Decoder(cfg, dev, tp=world, rank=rank, seed=0, group=group, fused_allreduce=fused,
                            prefill_exchange=getattr(args, "prefill_exchange", "peer"))
    model.alloc_cache(B, S + steps)
    g = torch.Generator().manual_seed(0)
    ids = torch.randint(0, cfg.vocab_size, (B, S), generator=g).to(dev)

    def sync():
        torch.cuda.synchronize(dev)
        if world > 1:
            dist.barrier(device_ids=[local_rank])

    def timed(fn):
        sync()
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record()
        h0 = time.perf_counter()
        out = fn()
        host_ms[0] = (time.perf_counter() - h0) * 1e3  # how long the host took to enqueue the work
        e1.record()
        torch.cuda.synchronize(dev)
        ms = e0.elapsed_time(e1)
        if world > 1:
            t = torch.tensor([ms, host_ms[0]], dtype=torch.float64, device=dev)
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
            ms, host_ms[0] = float(t[0].item()), float(t[1].item())
        return out, ms

    host_ms = [0.0]

    with torch.no_grad():
        model.prefill(ids)  # warm-up at full size (allocator, kernel set-up, NCCL communicator)
        logits_eager, prefill_eager_ms = timed(lambda: model.prefill(ids))
        prefill_host_ms = host_ms[0]
        # The prompt pass as one CUDA graph, as the reference's harness times it
        # (ablation/real_int4_kernel/graph_bench_all.py:72-92); its logits must equal the eager pass's.
        # Over NCCL (tensor parallelism without the peer-memory exchange) the pass stays eager.
        prefill_launch = "eager"
        logits, prefill_ms = logits_eager, prefill_eager_ms
        prefill_graph_ok = None
        prefill_graph_ms = None
        if not args.no_graph:
            try:
                run_prefill = model.capture_prefill(ids)
                if hasattr(run_prefill, "graph"):
                    run_prefill()  # first replay untimed
                    logits_g, ms_g = timed(run_prefill)
                    prefill_graph_ok = bool(torch.equal(logits_g, logits_eager))
                    prefill_graph_ms = ms_g
                    if prefill_graph_ok and ms_g <= prefill_eager_ms:  # the faster of two equal results is reported
                        logits, prefill_ms, prefill_launch = logits_g, ms_g, "CUDA graph"
            except Exception as exc:  # noqa: BLE001
                sys.stderr.write(f"prefill graph capture failed, timing the eager pass: {exc}\n")
        tok = logits.argmax(-1)
        pos_t = torch.tensor([S], dtype=torch.int64, device=dev)
        static_tok = tok.clone()
        graph = None
        # With tensor parallelism and NCCL the step contains torch.distributed collectives, which
        # are not captured here (a first attempt to capture them did not terminate), so that
        # decode loop is launched eagerly.  With the all-reduce fused into the GEMM kernel the step
        # holds no library collective and is captured like the single-GPU one.
        if not args.no_graph and (world == 1 or fused):
            try:
                sync()
                model.decode_step(static_tok, pos_t)  # warm-up outside capture
                torch.cuda.synchronize(dev)
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph):
                    static_logits = model.decode_step(static_tok, pos_t)
            except Exception as exc:  # capture not possible (e.g. collective): run eagerly
                graph = None
                sys.stderr.write(f"decode graph capture failed, running eagerly: {exc}\n")

        # Correctness gate before any decode time is reported (the reference's harness does the same,
        # ablation/real_int4_kernel/graph_bench_all.py:84-92,142-153): the captured step must
        # reproduce the eagerly launched step on the same token and cache position.
        checks = {"graph_equals_eager": None}
        if graph is not None:
            pos_t.fill_(S)
            static_tok.copy_(tok)
            eager_logits = model.decode_step(static_tok, pos_t).clone()
            graph.replay()
            torch.cuda.synchronize(dev)
            diff = (static_logits.float() - eager_logits.float()).abs().max().item()
            ok = bool(torch.equal(static_logits, eager_logits))
            if world > 1:
                t = torch.tensor([0.0 if ok else 1.0], device=dev)
                dist.all_reduce(t, op=dist.ReduceOp.MAX)
                ok = t.item() == 0.0
            checks = {"graph_equals_eager": ok, "max_abs_logit_diff": diff}
        checks["prefill_logits_finite"] = bool(torch.isfinite(logits).all().item())
        checks["prefill_graph_equals_eager"] = prefill_graph_ok
        if fused:
            # One row-parallel linear (layer 0's o_proj) on the same decode-size input, reduced inside
            # the GEMM and by NCCL.  The fused path sums the ranks' fp32 partials and rounds once;
            # NCCL sums bf16 partials: agreement to bf16 rounding.  (Whole-stack logits are no
            # yardstick: 32 layers of 4-bit activations amplify a last-bit difference into
            # decorrelated codes, measured on the random-init stack.)
            lin = model.layers[0].o
            gx = torch.Generator(device=dev).manual_seed(1234 + rank)
            xin = torch.randn(B, lin.K, generator=gx, device=dev).to(torch.bfloat16)
            y_fused = lin(xin, ar=model.ar).float()
            y_nccl = lin(xin)
            dist.all_reduce(y_nccl, group=group)
            rel = ((y_fused - y_nccl.float()).abs().max() / y_nccl.float().abs().max()).item()
            checks["fused_allreduce_vs_nccl_max_rel_diff"] = round(rel, 5)
            checks["fused_allreduce_matches_nccl"] = bool(rel < 3e-2)

        if graph is None:
            for _ in range(2):  # untimed eager warm-up steps (allocator, lazy NCCL channels)
                model.decode_step(tok, pos_t)

        def decode_loop():
            cur = tok
            for i in range(steps):
                pos_t.fill_(S + i)
                if graph is not None:
                    static_tok.copy_(cur)
                    graph.replay()
                    cur = static_logits.argmax(-1)
                else:
                    cur = model.decode_step(cur, pos_t).argmax(-1)
            return cur

        _, decode_ms = timed(decode_loop)
    _lib.device_status(local_rank)
    rec = None
    if True:
        wbytes = decoder.linear_weight_bytes(cfg)
        step_ms = decode_ms / steps
        peaks, kind = _peaks()
        rec = ({
            "suite": "decoder", "n_gpus": world, "layers": cfg.num_hidden_layers, "batch": B, "seqlen": S,
            "decode_steps": steps, "parallelism": f"tp{world}: qkv/gate_up column-parallel, o/down row-parallel + "
                           + ("all-reduce fused into the decode GEMM over peer memory" if fused
                              else "NCCL all-reduce")
                           + (("; prefill with the residual stream sharded over tokens, "
                               + ("partial output tiles pushed to their owners from the GEMM epilogue and codes pushed "
                                  "to every rank over NVLink peer memory (no NCCL)" if model._exchange else
                                  "NCCL reduce-scatter of partial outputs and all-gather of activation codes"))
                              if world > 1 and model.token_sharded_prefill and (B * S) % world == 0 else ""),
            "prefill_ms": round(prefill_ms, 2), "prefill_tokens_per_s": round(B * S / prefill_ms * 1e3, 1),
            "prefill_launch": prefill_launch, "prefill_eager_ms": round(prefill_eager_ms, 2),
            "prefill_graph_ms": None if prefill_graph_ms is None else round(prefill_graph_ms, 2),
            "prefill_eager_host_enqueue_ms": round(prefill_host_ms, 2),
            "decode_ms_per_step": round(step_ms, 3) if checks.get("graph_equals_eager") is not False else None,
            "decode_tokens_per_s": round(B / step_ms * 1e3, 1),
            "decode_launch": "CUDA graph" if graph is not None else "eager",
            "linear_weight_GB": round(wbytes / 1e9, 3),
            "decode_weight_stream_GBps": round(wbytes / (step_ms * 1e-3) / 1e9, 1),
            "decode_weight_stream_frac_of_hbm_per_gpu": round(wbytes / world / (step_ms * 1e-3) / 1e9 / peaks["hbm_gbs"], 4),
            "checks": checks})
    del model
    torch.cuda.empty_cache()
    if emit and rank == 0:
        print(json.dumps(rec), flush=True)
    if world > 1 and init_pg:
        dist.destroy_process_group()
    return rec


def run_fp4_suite(args, emit=True):
    """Block-scaled FP4 linears on the Qwen2.5-7B-architecture shapes (benchmark configuration 3):
    MXFP4 and NVFP4, M = 16 (GB/s of algorithmic bytes) and M = 4096 (TFLOPS = 2*M*N*K/s)."""
    from dualquant_b200 import _lib, ops

    dev = torch.device("cuda", 0)
    torch.cuda.set_device(dev)
    peaks, kind = _peaks()
    fp4_measured = 4.0 * peaks["bf16_tflops"]
    g = torch.Generator(device=dev).manual_seed(0)
    rows = []
    for fmt_name, fmt in (("mxfp4", _lib.FP4_MXFP4), ("nvfp4", _lib.FP4_NVFP4)):
        blk = 32 if fmt == _lib.FP4_MXFP4 else 16
        for name, K, N in synthetic.QWEN25_7B_LINEARS:
            w = (torch.randn(N, K, generator=g, device=dev) * 0.02).to(torch.bfloat16)
            pw = ops.pack_w_fp4(w, fmt)
            del w
            r, c = synthetic.make_scales(N, K, 0)
            r, a = r.to(dev), (1.0 / c).to(dev)
            for M in (16, 4096):
                x = torch.randn(M, K, generator=g, device=dev).to(torch.bfloat16)
                codes, sf, rs = ops.quant_fp4(x, fmt, a, None)
                sfa = ops.fp4_sf_to_atoms(sf, K, fmt)
                # prefill rows write bf16 (the model's activation type; at M = 4096 an fp32 gate+up output is
                # 620 MB, a third of the GEMM's time in HBM writes alone), decode rows fp32
                ydt = torch.bfloat16 if M > 128 else torch.float32
                y = torch.empty(M, N, dtype=ydt, device=dev)
                # Decode batches stream the weights: the graph walks enough copies of the packed
                # weight (> 2x the 126 MB L2 in total) that every launch reads them from HBM.
                # At M = 4096 operands + output exceed L2 on their own or the GEMM is tensor-bound.
                w_bytes = pw.codes.numel() + pw.sf_atoms.numel()
                n_copies = 1 if M > 128 else int(2 * 126e6 // w_bytes) + 2
                pws = [pw] + [dataclasses.replace(pw, codes=pw.codes.clone(), sf_atoms=pw.sf_atoms.clone())
                              for _ in range(n_copies - 1)]

                def gemm_all():
                    for p_ in pws:
                        ops.gemm_w4a4_fp4(codes, sfa, rs, p_, r, out=y)

                def full_all():
                    for p_ in pws:
                        ops.gemm_w4a4_fp4(*_fp4_prologue(ops, x, a, p_), p_, r, out=y)

                g_gemm = _capture(gemm_all, dev)
                g_full = _capture(full_all, dev)
                ms_gemm = _time_loop(g_gemm.replay, args.steps, args.warmup, dev, lambda: None) / args.steps / n_copies
                ms_full = _time_loop(g_full.replay, args.steps, args.warmup, dev, lambda: None) / args.steps / n_copies
                del pws, g_gemm, g_full
                flops = 2.0 * M * N * K
                nbytes = N * K // 2 + N * K // blk + 2 * N + 2 * K + 2 * M * K + y.element_size() * M * N
                rows.append({"fmt": fmt_name, "linear": name, "M": M, "K": K, "N": N, "weight_copies": n_copies,
                             "y_dtype": "bf16" if ydt == torch.bfloat16 else "fp32",
                             "gemm_us": round(ms_gemm * 1e3, 1), "linear_us": round(ms_full * 1e3, 1),
                             "gemm_TFLOPS": round(flops / ms_gemm / 1e9, 1),
                             "gemm_GBps": round(nbytes / ms_gemm / 1e6, 1),
                             "frac_fp4_nominal": round(flops / ms_gemm / 1e9 / 9000.0, 4),
                             "frac_4x_measured_bf16": round(flops / ms_gemm / 1e9 / fp4_measured, 4),
                             "frac_hbm_measured": round(nbytes / ms_gemm / 1e6 / peaks["hbm_gbs"], 4)})
            del pw
    _lib.device_status(0)
    mma = _mma_peaks(args)
    if mma is not None:
        for row in rows:
            pk = mma.get(row["fmt"] + "_TFLOPS")
            if pk and row["M"] > 128:
                row["frac_fp4_mma_only_measured"] = round(row["gemm_TFLOPS"] / pk, 4)
    rec = {"suite": "fp4", "peaks": {"fp4_nominal_TFLOPS": 9000.0, "fp4_4x_bf16_" + kind: fp4_measured,
                                     "hbm_GBps_" + kind: peaks["hbm_gbs"],
                                     "mma_only_measured": mma},
           "steps": args.steps, "rows": rows}
    if emit:
        print(json.dumps(rec), flush=True)
    return rec


def _fp4_prologue(ops, x, a, pw):
    """Activation quantiser of the FP4 linear, as ops.linear_w4a4_fp4 runs it: one launch that
    writes the scale bytes in the order the GEMM streams."""
    return ops.quant_fp4(x, pw.fmt, a, None, atoms=True)


def per_shape_detail(wl, dev, args):
    """GEMM-only GB/s of each (linear, M), timed as a graph that cycles through the six weight
    copies of that linear (so each launch reads weights that left L2)."""
    ops = wl.ops
    out = {}
    for lin in wl.linears:
        row = []
        for M in synthetic.DECODE_M:
            codes, sx = wl.q[(M, lin["name"])]
            y = wl.y[(M, lin["name"])]

            def fn():
                for c in range(len(lin["w"])):
                    ops.gemm_w4a4_int4(codes, sx, lin["w"][c], lin["r"], out=y)

            g = _capture(fn, dev)
            ms = _time_loop(g.replay, 20, 5, dev, lambda: None) / 20 / len(lin["w"])
            b = synthetic.int4_gemm_bytes(M, lin["N"], lin["K"])
            row.append(round(b / (ms * 1e-3) / 1e9, 1))
        out[lin["name"]] = row
    return out


# ------------------------------------------------------------------------------------------------
# CPU arm (the oracle port of the reference's PyTorch path)
# ------------------------------------------------------------------------------------------------
class CpuWorkload:
    """The reference's CPU path for the same step: PermLinear.forward as fake-quant
    (activations/perm_linear.py:108-141) - scale, per-token int4 cast, bf16 F.linear against the
    fake-quant bf16 weight.  When the reference's own modules are staged under oracle/_ref
    (oracle/stage_reference.py) the step runs the reference's unmodified PermLinear
    (kind "reference"); otherwise the restatement in oracle/dq_oracle.py (kind "port").  Weights
    of the sample are built once (untimed), like the reference's offline weight quantisation."""

    def __init__(self, m_values, seed=0):
        from oracle import dq_oracle as O
        from oracle import stage_reference as SR

        self.O = O
        self.m_values = m_values
        self.kind = "port"
        ref = None
        if SR.available():
            try:
                ref = SR.import_reference()
                self.kind = "reference"
            except Exception as exc:  # noqa: BLE001 - fall back to the port, say why
                sys.stderr.write(f"staged reference not importable ({exc}); using the oracle port\n")
        self.linears = []
        for name, K, N in synthetic.LLAMA31_8B_LINEARS:
            w = synthetic.make_w(N, K, seed)
            qw, sw = O.quant_w_int4(w)
            r, c = synthetic.make_scales(N, K, seed)
            wdq = O.dequant_w(qw, sw, r).to(torch.bfloat16)
            entry = {"name": name, "K": K, "N": N, "a": 1.0 / c, "w": wdq, "module": None}
            if ref is not None:
                lin = torch.nn.Linear(K, N, bias=False).to(torch.bfloat16)
                lin.weight.data = wdq
                pl = ref.PermLinear(lin, ref.make_format("rtn_int4", block_size=-1))
                pl.set_act_scale(1.0 / c)
                entry["module"] = pl
            self.linears.append(entry)
        self.x = {(M, K): synthetic.make_x(M, K, seed) for M in m_values for _, K, _ in synthetic.LLAMA31_8B_LINEARS}

    def bytes(self):
        return sum(synthetic.int4_gemm_bytes(M, lin["N"], lin["K"]) for M in self.m_values for lin in self.linears)

    def describe(self):
        if self.kind == "reference":
            return ("the reference's own PermLinear (activations/perm_linear.py, staged unmodified under oracle/_ref) "
                    f"on CPU, torch {torch.__version__}")
        return ("oracle restatement of PermLinear's fake-quant forward (the staged reference is absent), "
                f"torch {torch.__version__} bf16 F.linear")

    def step(self):
        O = self.O
        out = None
        with torch.no_grad():
            for M in self.m_values:
                for lin in self.linears:
                    if lin["module"] is not None:
                        out = lin["module"](self.x[(M, lin["K"])])
                    else:
                        out = O.perm_linear_fakequant(self.x[(M, lin["K"])], lin["a"], None, lin["w"], False)
        return out


def cpu_baseline(budget_s: float = 15.0):
    cores = os.cpu_count() or 1
    torch.set_num_threads(cores)
    wl = CpuWorkload(synthetic.DECODE_M)
    wl.step()  # warm-up
    t0 = time.perf_counter()
    n = 0
    while True:
        wl.step()
        n += 1
        if time.perf_counter() - t0 > budget_s or n >= 500:
            break
    dt = (time.perf_counter() - t0) / n
    return {"value": round(wl.bytes() / dt / 1e9, 3), "unit": UNIT, "cores": cores, "kind": wl.kind,
            "sample": f"{n} pass(es) of the full step (24 linears), {dt:.3f} s each; {wl.describe()}",
            "ms_per_step": round(dt * 1e3, 1)}


def run_reference(args):
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    cores = os.cpu_count() or 1
    torch.set_num_threads(cores)
    wl = CpuWorkload(synthetic.DECODE_M)
    warmup = max(3, min(args.warmup, 20))
    for _ in range(warmup):
        wl.step()
    steps = max(1, min(args.steps, 100))
    t0 = time.perf_counter()
    for _ in range(steps):
        wl.step()
    dt = (time.perf_counter() - t0) / steps
    value = round(wl.bytes() / dt / 1e9, 3)
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": args.gpus,
        "steps": steps, "warmup": warmup, "ms_per_step": round(dt * 1e3, 2),
        "higher_is_better": True, "scaling": "strong", "vs_baseline": None,
        "dtype": "bf16 fake-quant (fp32 quantiser)", "data": "synthetic",
        "config": bench_config(args.gpus),
        "arm": {"path": wl.describe(), "threads": cores,
                "note": "the whole step on rank 0's host cores (the CPU path does not shard)"},
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": cores, "kind": wl.kind,
                         "sample": f"{steps} timed pass(es) of the full step (24 linears)"},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


# ------------------------------------------------------------------------------------------------
# The reference's own GPU kernels (Triton) on this GPU: context rows, never on the product path
# ------------------------------------------------------------------------------------------------
def run_bcd_suite(args, emit=True):
    """DualQuant's offline scale search + block quantisation of one 4096 x 4096 weight (32 column
    blocks of 128, row_column scales, five iterations, E8M0 row scales): dualquant_b200.bcd on the
    GPU (all blocks as one batch) next to the reference's wrap_dualquant_layer on the host cores
    (block after block; timed on the first four blocks and scaled to 32 - the blocks are
    independent and equally large)."""
    from dualquant_b200 import bcd

    dev = torch.device("cuda", 0)
    torch.cuda.set_device(dev)
    R, C, bs, iters = 4096, 4096, 128, 5
    cfg = dict(scale_option="row_column", row_init="max_abs", col_init="l1_norm", num_iter=iters, scale_format="e8m0")
    g = torch.Generator(device=dev).manual_seed(0)
    W = torch.randn(R, C, generator=g, device=dev) * 0.02
    for _ in range(2):
        bcd.dualquant_weight(W, block_size=bs, **cfg)
    torch.cuda.synchronize(dev)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    reps = 5
    e0.record()
    for _ in range(reps):
        mat_q, cs = bcd.dualquant_weight(W, block_size=bs, **cfg)
    e1.record()
    torch.cuda.synchronize(dev)
    gpu_ms = e0.elapsed_time(e1) / reps
    W3 = W.reshape(R, C // bs, bs)
    s = W3.abs().amax(dim=-1, keepdim=True) / 7.0
    rtn = ((W3 / s).round().clamp(-8, 7) * s).reshape(R, C)
    rec = {"suite": "bcd", "rows": R, "cols": C, "block_size": bs, "num_iter": iters, "scale_format": "e8m0",
           "gpu_ms": round(gpu_ms, 2),
           "mse_dualquant_over_rtn": round((((mat_q * cs - W) ** 2).mean() / ((rtn - W) ** 2).mean()).item(), 4)}
    try:
        from oracle import stage_reference as SR

        SR.import_reference()
        from layer_wrapper_dualquant import wrap_dualquant_layer

        nb = 4
        lin = torch.nn.Linear(nb * bs, R, bias=False)
        lin.weight.data.copy_(W[:, :nb * bs].cpu())
        ref_cfg = dict(num_splits=1, block_size=bs, dualquant_to_element_tensor=True, **cfg)
        t0 = time.time()
        ref_cs = wrap_dualquant_layer(lin, None, ref_cfg, "rtn_int4", act_quant_flag=True)
        cpu_s = time.time() - t0
        rec["reference_cpu"] = {"blocks_timed": nb, "seconds": round(cpu_s, 3),
                                "scaled_to_all_blocks_ms": round(cpu_s * (C // bs) / nb * 1e3, 1),
                                "threads": torch.get_num_threads()}
        rec["speedup_vs_reference_cpu"] = round(cpu_s * (C // bs) / nb * 1e3 / gpu_ms, 1)
        d = (mat_q[:, :nb * bs].cpu() - lin.weight.data).abs() / lin.weight.data.abs().max()
        # fp32 sums in another order: ulp-level differences everywhere, a code step at a rounding boundary
        rec["stored_weight_vs_reference"] = {"frac_elements_off_by_more_than_1e-5": round((d > 1e-5).float().mean().item(), 7),
                                             "max_rel_diff": round(d.max().item(), 6)}
        rec["max_rel_diff_column_scales"] = round(((cs[:nb * bs].cpu() - ref_cs).abs() / ref_cs.abs()).max().item(), 9)
    except Exception as exc:  # noqa: BLE001
        rec["reference_cpu"] = {"unavailable": f"{type(exc).__name__}: {exc}"[:200]}
    if emit:
        print(json.dumps(rec), flush=True)
    return rec


def run_reference_gpu(args, emit=True):
    """Times the reference's two Triton kernels on the same GPU with the same CUDA-event harness:
    `fused_w4a4_gemm` (ablation/real_int4_kernel/fused_w4a4_kernel.py:129-161, group 64, autotuned)
    and `fused_beta_int4_gemm` (vendor/dualscale_kernel_benchmark/fused_dual_scale_kernel.py:220-262,
    group 32), imported unmodified from oracle/_ref.  A kernel that cannot be imported, compiled or
    run reports its error text."""
    from oracle import stage_reference as SR

    rec = {"suite": "reference_gpu_kernels", "rows": []}
    if not SR.available():
        rec["unavailable"] = "oracle/_ref is not staged (run python oracle/stage_reference.py <reference checkout>)"
        if emit:
            print(json.dumps(rec), flush=True)
        return rec
    dev = torch.device("cuda", 0)
    torch.cuda.set_device(dev)
    try:
        SR.import_reference()
        import fused_dual_scale_kernel as fdk
        import fused_w4a4_kernel as fwk
    except Exception as exc:  # noqa: BLE001
        rec["unavailable"] = f"import failed: {type(exc).__name__}: {exc}"[:300]
        if emit:
            print(json.dumps(rec), flush=True)
        return rec
    from dualquant_b200 import ops

    g = torch.Generator(device=dev).manual_seed(0)
    cases = (("gate_up M=16", 16, 4096, 28672), ("o M=16", 16, 4096, 4096), ("config0 M=2048", 2048, 4096, 4096))
    for label, M, K, N in cases:
        w = (torch.randn(N, K, generator=g, device=dev) * 0.02)
        x = torch.randn(M, K, generator=g, device=dev).to(torch.bfloat16)
        beta = torch.exp(torch.randn(K, generator=g, device=dev) * 0.3).to(torch.bfloat16)
        row = {"shape": label, "M": M, "K": K, "N": N}
        # this library on the same shape (quantiser + GEMM), for the ratio
        codes, sw = ops.quant_w_int4(w.to(torch.bfloat16))
        pw = ops.pack_w_int4(codes, sw)
        a32 = beta.float()
        y = torch.empty(M, N, dtype=torch.float32, device=dev)
        scratch = torch.empty(max(256, ops.linear_scratch_bytes(M, N, K)), dtype=torch.uint8, device=dev)
        g_own = _capture(lambda: ops.linear_w4a4_int4(x, a32, None, pw, None, scratch=scratch, out=y), dev)
        row["dualquant_b200_linear_us"] = round(_time_loop(g_own.replay, 20, 5, dev, lambda: None) / 20 * 1e3, 1)
        yb = torch.empty(M, N, dtype=torch.bfloat16, device=dev)
        s16 = torch.empty(M * K * 2 + 256, dtype=torch.uint8, device=dev)
        g_a16 = _capture(lambda: ops.linear_a16w4(x, a32, pw, None, scratch=s16, out=yb), dev)
        row["dualquant_b200_a16w4_us"] = round(_time_loop(g_a16.replay, 20, 5, dev, lambda: None) / 20 * 1e3, 1)
        del g_a16, yb, s16
        for kname, fn, gs, mod in (("triton_fused_w4a4_gemm_g64", "fused_w4a4_gemm", 64, fwk),
                                   ("triton_fused_beta_int4_gemm_g32", "fused_beta_int4_gemm", 32, fdk)):
            try:
                wp, s1 = fdk.pack_int4_weights(w, gs)
                call = getattr(mod, fn)
                if fn == "fused_beta_int4_gemm":
                    run = lambda: call(x, beta, wp, s1, group_size=gs)  # noqa: E731
                else:
                    run = lambda: call(x, beta, wp, s1, group_size=gs)  # noqa: E731
                run()  # compile / autotune
                torch.cuda.synchronize()
                ms = _time_loop(run, 10, 3, dev, lambda: None) / 10
                row[kname + "_us"] = round(ms * 1e3, 1)
                row[kname + "_TOPS"] = round(2.0 * M * N * K / ms / 1e9, 1)
            except Exception as exc:  # noqa: BLE001
                row[kname + "_unavailable"] = f"{type(exc).__name__}: {exc}"[:200]
            torch.cuda.empty_cache()
        rec["rows"].append(row)
        del w, x, pw
    try:
        rec["decode_sweep"] = _reference_gpu_decode_sweep(SR, fdk, fwk, dev)
    except Exception as exc:  # noqa: BLE001
        rec["decode_sweep"] = {"error": f"{type(exc).__name__}: {exc}"[:300]}
    if emit:
        print(json.dumps(rec), flush=True)
    return rec


def _reference_gpu_decode_sweep(SR, fdk, fwk, dev, budget_s=90.0):
    """The headline step (the 24 (linear, M) pairs of the decode sweep) through the reference's own GPU
    code on this GPU: (a) its PermLinear - fake-quantised activations into a bf16 F.linear, the path the
    reference runs by default - and (b) its Triton W4A4 kernel (fused_w4a4_gemm, group 64, autotuned per
    shape; stops adding shapes once `budget_s` seconds are spent and says so).  One weight copy per
    linear, eager launches, CUDA events around the whole step; GB/s counts the same algorithmic int4
    bytes as the headline, so the figures compare like for like."""
    ref = SR.import_reference()
    g = torch.Generator(device=dev).manual_seed(0)
    out = {"step_algorithmic_bytes": _step_bytes(1)}
    lins = []
    for name, K, N in synthetic.LLAMA31_8B_LINEARS:
        w = torch.randn(N, K, generator=g, device=dev) * 0.02
        _, c = synthetic.make_scales(N, K, 0)
        lin = torch.nn.Linear(K, N, bias=False, device=dev, dtype=torch.bfloat16)
        lin.weight.data.copy_(w.to(torch.bfloat16))
        pl = ref.PermLinear(lin, ref.make_format("rtn_int4", block_size=-1))
        pl.set_act_scale((1.0 / c).to(dev))
        lins.append((name, K, N, w, pl, (1.0 / c).to(dev).to(torch.bfloat16)))
    xs = {(M, K): torch.randn(M, K, generator=g, device=dev).to(torch.bfloat16)
          for M in synthetic.DECODE_M for K in {k for _, k, _ in synthetic.LLAMA31_8B_LINEARS}}

    def step_permlinear():
        for M in synthetic.DECODE_M:
            for _name, K, _N, _w, pl, _b in lins:
                pl(xs[(M, K)])

    with torch.no_grad():
        step_permlinear()
        torch.cuda.synchronize(dev)
        ms = _time_loop(step_permlinear, 10, 3, dev, lambda: None) / 10
    out["reference_permlinear_bf16"] = {"ms_per_step": round(ms, 3),
                                        "GBps": round(out["step_algorithmic_bytes"] / ms / 1e6, 1),
                                        "what": "PermLinear.forward (fake-quant activations, bf16 F.linear), eager"}
    # Triton W4A4 kernel: autotune every shape first (inside the time budget), then time the shapes done
    t0 = time.time()
    packed, done = {}, []
    for name, K, N, w, _pl, beta in lins:
        packed[name] = fdk.pack_int4_weights(w, 64)
    for M in synthetic.DECODE_M:
        for name, K, N, _w, _pl, beta in lins:
            if time.time() - t0 > budget_s:
                break
            wp, s1 = packed[name]
            fwk.fused_w4a4_gemm(xs[(M, K)], beta, wp, s1, group_size=64)  # compile / autotune
            torch.cuda.synchronize(dev)
            done.append((M, name, K, N, beta))

    def step_triton():
        for M, name, K, _N, beta in done:
            wp, s1 = packed[name]
            fwk.fused_w4a4_gemm(xs[(M, K)], beta, wp, s1, group_size=64)

    if done:
        ms_t = _time_loop(step_triton, 10, 3, dev, lambda: None) / 10
        nbytes = sum(synthetic.int4_gemm_bytes(M, N, K) for M, _n, K, N, _b in done)
        out["reference_triton_w4a4_g64"] = {"pairs_timed": len(done), "of": 24, "ms": round(ms_t, 3),
                                            "GBps": round(nbytes / ms_t / 1e6, 1),
                                            "what": "fused_w4a4_gemm (per-(row, K tile) activation scales, group 64), eager"}
    return out


# ------------------------------------------------------------------------------------------------
# MMA-only tensor-core peaks (tcgen05 issue loops with resident operands)
# ------------------------------------------------------------------------------------------------
_MMA_PEAKS = {}


def _mma_peaks(args):
    """Measured once per process: {"int8_TOPS", "e4m3_TFLOPS", "mxfp4_TFLOPS", "nvfp4_TFLOPS"} or None."""
    if "v" not in _MMA_PEAKS:
        try:
            _MMA_PEAKS["v"] = run_peak_suite(args, emit=False)
        except Exception as exc:  # noqa: BLE001
            sys.stderr.write(f"MMA-only peak measurement failed: {exc}\n")
            _MMA_PEAKS["v"] = None
    return _MMA_PEAKS["v"]


def run_peak_suite(args, emit=True):
    """tcgen05.mma issue loops on operands that never leave shared / tensor memory: the rate the
    tensor pipe sustains with nothing else going on, for kind::i8 (128x256x32 per instruction)
    and kind::mxf4nvf4.block_scale (128x256x64, E8M0 block 32 and E4M3 block 16); and the E4M3 loop
    once more with its operands refilled from L2, the ceiling of a K loop that has to feed itself."""
    from dualquant_b200 import _lib, ops

    if "v" in _MMA_PEAKS and _MMA_PEAKS["v"] is not None:
        rec = _MMA_PEAKS["v"]
    else:
        dev = torch.device("cuda", 0)
        torch.cuda.set_device(dev)
        rec = {"suite": "peaks_mma_only"}
        for key, kind in (("int8_TOPS", 0), ("e4m3_TFLOPS", 3), ("e4m3_refill_TFLOPS", 4), ("mxfp4_TFLOPS", 1),
                          ("nvfp4_TFLOPS", 2)):
            best = 0.0
            for _ in range(3):
                best = max(best, ops.mma_peak(kind, iters=4096))
            rec[key] = round(best, 1)
        rec["how"] = ("one CTA per SM, one thread issuing back-to-back tcgen05.mma (UMMA 128x256, K = 32 bytes "
                      "per instruction for int8 / E4M3, 64 elements for FP4) on shared-memory operands that are "
                      "never reloaded; e4m3_refill: the same loop with a fresh 16 KB + 32 KB operand pair copied "
                      "in from L2 for every four instructions (three-stage ring); CUDA events; best of 3")
        _lib.device_status(0)
        _MMA_PEAKS["v"] = rec
    if emit:
        print(json.dumps(rec), flush=True)
    return rec


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=50)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="dualquant_b200", choices=["dualquant_b200", "reference"])
    ap.add_argument("--no-graph", action="store_true")
    ap.add_argument("--skip-cpu", action="store_true")
    ap.add_argument("--cpu-budget", type=float, default=15.0)
    ap.add_argument("--case", default=None, help="NAME:M[:TN:SPLIT] - run one (linear, M) GEMM alone")
    ap.add_argument("--iters", type=int, default=6)
    ap.add_argument("--layers", type=int, default=32)
    ap.add_argument("--batch", type=int, default=8)
    ap.add_argument("--seqlen", type=int, default=2048)
    ap.add_argument("--decode-steps", type=int, default=128)
    ap.add_argument("--prefill-exchange", choices=("peer", "nccl"), default="peer",
                    help="decoder suite on several GPUs: how the token-sharded prompt pass exchanges data")
    ap.add_argument("--fused-allreduce", action="store_true",
                    help="decoder suite, N>1: sum row-parallel partial outputs inside the decode GEMM over peer memory")
    ap.add_argument("--tune", action="append", default=[], metavar="NAME=VALUE",
                    help="launch-shape override passed to dq_set_tuning (measurement sweeps)")
    ap.add_argument("--no-extras", action="store_true",
                    help="only the decode sweep (skip the prefill / MLP / FP4 / decoder sub-records)")
    ap.add_argument("--no-detail", action="store_true", help="skip the per-(linear, M) GEMM table")
    ap.add_argument("--suite", default=None, choices=["prefill", "fp4", "mlp", "decoder", "peaks", "reference_gpu", "bcd"],
                    help="one measurement suite alone")
    args = ap.parse_args()
    args.warmup = max(args.warmup, 3) if args.impl != "reference" else args.warmup
    if args.tune:
        from dualquant_b200 import _lib as _tl

        for item in args.tune:
            name, _, val = item.partition("=")
            _tl.set_tuning(name, int(val))
    if args.suite == "prefill":
        run_prefill_suite(args)
    elif args.suite == "fp4":
        run_fp4_suite(args)
    elif args.suite == "mlp":
        run_mlp_suite(args)
    elif args.suite == "decoder":
        run_decoder_suite(args)
    elif args.suite == "peaks":
        run_peak_suite(args)
    elif args.suite == "reference_gpu":
        run_reference_gpu(args)
    elif args.suite == "bcd":
        run_bcd_suite(args)
    elif args.case:
        run_case(args)
    elif args.impl == "reference":
        run_reference(args)
    else:
        run_gpu(args)


if __name__ == "__main__":
    main()
