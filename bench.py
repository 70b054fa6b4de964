#!/usr/bin/env python
"""Benchmark of the counter-synapse linear path on B200.

    python bench.py --gpus N --steps K --warmup W [--impl reference] [--workload cfg2]

Metric: counter-linear train tokens/s.  A step is one pass of the hot path -- forward Y = X W^T,
backward-to-input dX, weight gradient dW = dY^T X and the fused counter update (writing the new
6-bit state, 2-bit packed weights, scale and v) -- over every counter linear of the workload.
Default workload `cfg2`: the stories15M-shaped stack (42 linears of 288/768 width, 8192 tokens).
Inputs are seeded synthetic tensors with the reference's shapes and distributions.

Prints ONE JSON line (rank 0).  `value` times the step with inputs resident in HBM; `e2e`
times it from pinned HOST buffers (host->device copies of X and dY, device->host copy of the
updated state / packed weights / scales) through the same C-ABI calls.  `--impl reference`
times the CPU checker's restatement of the reference kernels on the host cores instead.

The same line carries, under `also`, the other configurations of the metric: on one GPU the
1B-scale stack (cfg3), the decode-GEMV sweep at M = 1, 4, 16 with the reference's own host GEMV
beside it (cfg5) and the fused update at an HBM-resident size; on several GPUs the 8B-scale
data-parallel stack (cfg4), the tensor-parallel decode sweep and `dp_parity`, a byte comparison of every rank's updated row shards
with the CPU checker run on the reduce-scattered gradient that the rank downloaded.
"""
from __future__ import annotations

import argparse
import json
import os
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "counter-linear train tokens/s"
UNIT = "tokens/s"


def workload(name: str):
    from motifcl_b200 import synth
    if name == "cfg2":
        return dict(cfg=2, tokens=8192, sigma=0.02, linears=synth.stories15m_linears(),
                    desc="stories15M-shaped stack: dim 288, 6 layers, FFN 768, 42 counter linears, 8192 tokens")
    if name == "cfg3":
        return dict(cfg=3, tokens=16384, sigma=0.01, linears=synth.llama_linears(2048, 5632, 22),
                    desc="1B-scale: dim 2048, FFN 5632, 22 layers, 16384 tokens")
    if name == "cfg4":
        return dict(cfg=4, tokens=8192, sigma=0.01, linears=synth.llama_linears(4096, 14336, 32, kv_dim=1024),
                    desc="8B-scale: dim 4096, FFN 14336, 32 layers, k/v 4096x1024, 8192 tokens per GPU")
    if name == "cfg1":
        return dict(cfg=1, tokens=256, sigma=0.02, linears=[synth.LinearShape("single", 288, 288)],
                    desc="single 288x288 counter linear, 256 tokens")
    raise SystemExit(f"unknown workload {name}")


def algorithmic(wl):
    W = sum(l.out_features * l.in_features for l in wl["linears"])
    rows = sum(l.out_features for l in wl["linears"])
    feat = sum(l.out_features + l.in_features for l in wl["linears"])
    # products: X and dY read once, Y and dX written once (fp32), the 6-bit state read once, dW written once
    gemm_bytes = 8.0 * wl["tokens"] * feat + 0.75 * W + 4.0 * W
    return dict(weights=W, rows=rows, gemm_flop=6.0 * wl["tokens"] * W, gemm_bytes=gemm_bytes,
                update_bytes=5.75 * W + 16.0 * rows)


# dram__bytes_read.sum + dram__bytes_write.sum of the contraction kernel's launches for one step of a workload, from the ncu
# capture summarised in profiles/grouped_step_cfg2.md
MEASURED_TRAFFIC_BYTES = {"cfg2": 3.248e9}


class ClockSampler:
    """Samples SM clock and throttle reasons through NVML (read-only) while the timed region runs."""

    def __init__(self, index: int):
        self.samples, self.reasons, self.max_mhz = [], set(), None
        self._stop = threading.Event()
        self._thr = None
        try:
            import pynvml
            pynvml.nvmlInit()
            self.nv = pynvml
            self.h = pynvml.nvmlDeviceGetHandleByIndex(index)
            self.max_mhz = pynvml.nvmlDeviceGetMaxClockInfo(self.h, pynvml.NVML_CLOCK_SM)
        except Exception:
            self.nv = None

    def _run(self):
        nv = self.nv
        names = {nv.nvmlClocksThrottleReasonHwSlowdown: "hw_slowdown",
                 nv.nvmlClocksThrottleReasonHwThermalSlowdown: "hw_thermal_slowdown",
                 nv.nvmlClocksThrottleReasonSwThermalSlowdown: "sw_thermal_slowdown",
                 nv.nvmlClocksThrottleReasonSwPowerCap: "sw_power_cap"}
        while not self._stop.is_set():
            try:
                self.samples.append(nv.nvmlDeviceGetClockInfo(self.h, nv.NVML_CLOCK_SM))
                r = nv.nvmlDeviceGetCurrentClocksThrottleReasons(self.h)
                for bit, n in names.items():
                    if r & bit:
                        self.reasons.add(n)
            except Exception:
                pass
            self._stop.wait(0.004)

    def __enter__(self):
        if self.nv:
            self._thr = threading.Thread(target=self._run, daemon=True)
            self._thr.start()
        return self

    def __exit__(self, *a):
        self._stop.set()
        if self._thr:
            self._thr.join()

    def summary(self):
        return {"sm_mhz": float(np.median(self.samples)) if self.samples else None,
                "sm_max_mhz": self.max_mhz, "reasons": sorted(self.reasons), "samples": len(self.samples)}


def measured_peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.isfile(p):
        d = json.load(open(p))
        return d["hbm_gbs"], d["bf16_tflops_sustained"], "measured"
    return 6650.0, 1400.0, "fallback"


def base_config(name, wl, world):
    """The `config` object: identical in both arms (ours / reference) for the same command line."""
    alg = algorithmic(wl)
    in_bytes = sum(4 * wl["tokens"] * (l.in_features + l.out_features) for l in wl["linears"])
    return {"workload": f"{name}: {wl['desc']}", "tokens_per_gpu": wl["tokens"], "linears": len(wl["linears"]),
            "weights": alg["weights"], "parallelism": f"dp{world}" if world > 1 else "single",
            "l2": "inputs larger than L2 (X and dY of all linears: %.2f GB)" % (in_bytes / 1e9)}


class CpuSample:
    """A bounded sample of a workload for the CPU checker (the restatement of the reference kernels, all
    host cores): one linear of every distinct shape at up to `max_tokens` tokens.  One `pass_once()` runs
    forward, backward-to-input, weight gradient and the fused update of each; `scale` converts the time of
    a pass to the time of a full step (products by tokens x weights, update by weights)."""

    def __init__(self, wl, max_tokens: int = 8192):
        import oracle
        from motifcl_b200 import synth
        self.orc = oracle.port
        self.cores = len(os.sched_getaffinity(0))
        self.orc.set_threads(self.cores)
        self.wl = wl
        cfg, sigma = wl["cfg"], wl["sigma"]
        self.tokens = min(wl["tokens"], max_tokens)
        shapes = {}
        for idx, l in enumerate(wl["linears"]):
            shapes.setdefault((l.out_features, l.in_features), idx)
        self.data = []
        for (O, I), idx in shapes.items():
            sc, v = synth.scale_v(cfg, idx, O, I)
            self.data.append((O, I, synth.counters(cfg, idx, O, I).reshape(-1), sc, v,
                              synth.activations(cfg, idx, self.tokens, I),
                              synth.upstream_grad(cfg, idx, self.tokens, O, sigma)))
        self.weights = sum(d[0] * d[1] for d in self.data)
        self.t_gemm = self.t_upd = 0.0
        self.passes = 0

    def pass_once(self):
        o = self.orc
        for O, I, st, sc, v, x, dy in self.data:
            a = time.perf_counter()
            o.forward(x, st, sc, 11, O)
            o.backward_input(dy, st, sc, 11, I)
            gw = o.grad_w(dy, x)
            b = time.perf_counter()
            o.update_dense(st, sc, v, gw, 11, I, O, 0, 3e-3, 0.0, 0.9, 1e-3, 12345)
            c = time.perf_counter()
            self.t_gemm += b - a
            self.t_upd += c - b
        self.passes += 1

    def reset(self):
        self.t_gemm = self.t_upd = 0.0
        self.passes = 0

    def full_step_seconds(self):
        alg = algorithmic(self.wl)
        wr = alg["weights"] / self.weights
        return (self.t_gemm / self.passes) * (self.wl["tokens"] / self.tokens) * wr + (self.t_upd / self.passes) * wr

    def describe(self, seconds):
        return (f"{len(self.data)} distinct linear shapes ({self.weights} of {algorithmic(self.wl)['weights']} weights) at "
                f"{self.tokens} tokens, {self.passes} passes ({seconds:.1f} s of CPU work); scaled to the full workload by "
                f"tokens*weights (update by weights)")


def cpu_reference_rate(wl, min_seconds: float = 10.0, max_tokens: int = 8192):
    """The `cpu_baseline` object of the GPU arm: passes over the sample until `min_seconds` of CPU work."""
    smp = CpuSample(wl, max_tokens)
    t0 = time.perf_counter()
    while smp.passes == 0 or time.perf_counter() - t0 < min_seconds:
        smp.pass_once()
    full = smp.full_step_seconds()
    return dict(value=wl["tokens"] / full, unit=UNIT, cores=smp.cores, kind="port",
                sample=smp.describe(time.perf_counter() - t0)), full


def run_reference(args, wl):
    """The reference arm: the CPU restatement of the reference kernels, all host cores, on the same bounded sample
    as the GPU arm's cpu_baseline (every distinct linear shape at the full token count).  A step is a whole number of
    passes over that sample, sized from the warm-up so that the timed region holds at least 10 s of CPU work;
    `ms_per_step` is the MEASURED time of a step, `step_work_fraction` the work of such a step as a share of a full
    workload step, and `value` = tokens / (ms_per_step / step_work_fraction)."""
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    smp = CpuSample(wl)
    t0 = time.perf_counter()
    for _ in range(max(args.warmup, 1)):
        smp.pass_once()
    t_pass = (time.perf_counter() - t0) / smp.passes
    reps = max(1, int(np.ceil(10.0 / max(args.steps * t_pass, 1e-9))))
    reps = min(reps, max(1, int(120.0 / max(args.steps * t_pass, 1e-9))))      # and the run stays within minutes
    smp.reset()
    t0 = time.perf_counter()
    for _ in range(args.steps):
        for _ in range(reps):
            smp.pass_once()
    wall = time.perf_counter() - t0
    full = smp.full_step_seconds()
    val = wl["tokens"] / full
    ms_step = wall / args.steps * 1e3
    line = {"impl": "reference", "metric": METRIC, "value": val, "unit": UNIT, "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_step, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": base_config(args.workload, wl, args.gpus),
            "step_work_fraction": (wall / args.steps) / full,
            "passes_per_step": reps, "ms_per_full_step_scaled": full * 1e3,
            "arm": "CPU restatement of the reference kernels on the host cores (no GPU); the reference's own kernels "
                   "are OpenCL / Vulkan compute shaders with no host implementation of the contractions",
            "cpu_baseline": dict(value=val, unit=UNIT, cores=smp.cores, kind="port", sample=smp.describe(wall)),
            "e2e": {"value": val, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line))


def run_micro(args):
    """Single-kernel timing at an HBM-resident size, for roofline figures and profiler captures:
        --micro update:ROWSxIN[:lr_scale]   fused counter update (5.75 B/weight + 16 B/row)
        --micro gemv:OUTxIN:M               ternary GEMV (out*in/4 + 4*out + 4*M*(in+out) bytes)
        --micro step:TOKENSxINxOUT          one linear step (6*tokens*in*out flop)
        --micro stepmany:LAYERS[:TOKENS]    the grouped step of the first LAYERS linears of the stories15M stack
    Buffers are rotated so that consecutive launches never touch the same memory (sets larger
    than L2 in total)."""
    import torch
    from motifcl_b200 import Context
    torch.cuda.set_device(0)
    torch.cuda.set_stream(torch.cuda.Stream(device=0))
    ctx = Context.on_torch_stream(0)
    dev = "cuda:0"
    kind, shape, *rest = args.micro.split(":")
    dims = [int(v) for v in shape.split("x")]
    hbm_peak, tf_peak, peak_kind = measured_peaks()
    g = torch.Generator(device=dev).manual_seed(1)

    def timed(fn, iters, warm):
        for i in range(warm):
            fn(i)
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for i in range(iters):
            fn(warm + i)
        e1.record()
        torch.cuda.synchronize()
        return e0.elapsed_time(e1) / iters

    with ClockSampler(0) as clk:
        if kind == "update":
            O, I = dims
            lrs = float(rest[0]) if rest else 0.0
            per_set = O * I * 4.75
            nsets = max(2, int(300e6 // per_set) + 1)
            sets = []
            for _ in range(nsets):
                codes = torch.randint(0, 63, (O, I // 4, 4), device=dev, generator=g, dtype=torch.int32)
                w = codes[..., 0] | (codes[..., 1] << 6) | (codes[..., 2] << 12) | (codes[..., 3] << 18)
                st = torch.stack([w & 255, (w >> 8) & 255, (w >> 16) & 255], -1).to(torch.uint8).reshape(-1).contiguous()
                sets.append((st, torch.full((O,), 0.05, device=dev), torch.full((O,), 1e-3, device=dev),
                             torch.randn(O, I, device=dev, generator=g) * 0.5,
                             torch.zeros(O, I // 16, dtype=torch.int32, device=dev)))
            def fn(i):
                st, sc, v, gw, p2 = sets[i % nsets]
                ctx.counter_update_dense(st, sc, v, gw, p2, 11, I, O, 0, 3e-3, lrs, 0.9, 1e-3, 12345 + i)
            ms = timed(fn, args.steps, max(args.warmup, 3))
            nbytes = 5.75 * O * I + 16.0 * O
            out = {"kernel": "counter_update_dense_kernel", "bound": "hbm", "achieved": nbytes / ms / 1e6,
                   "peak": hbm_peak, "unit": "GB/s", "bytes_per_launch": nbytes}
        elif kind == "gemv":
            O, I = dims
            M = int(rest[0]) if rest else 1
            nsets = max(2, int(300e6 // (O * I / 4)) + 1)
            p2s = [torch.randint(-2 ** 31, 2 ** 31 - 1, (O, I // 16), dtype=torch.int32, device=dev, generator=g)
                   for _ in range(nsets)]
            sc = torch.full((O,), 0.05, device=dev)
            x = torch.randn(M, I, device=dev, generator=g)
            y = torch.empty(M, O, device=dev)
            ms = timed(lambda i: ctx.ternary_gemv(x, p2s[i % nsets], sc, y, M, I, O), args.steps, max(args.warmup, 3))
            nbytes = O * I / 4 + 4 * O + 4 * M * (I + O)
            out = {"kernel": "ternary_gemv_kernel", "bound": "hbm", "achieved": nbytes / ms / 1e6, "peak": hbm_peak,
                   "unit": "GB/s", "bytes_per_launch": nbytes, "tokens_per_s": M / (ms * 1e-3)}
        elif kind == "gemvsweep":
            # the decode-GEMV configuration: 32 layers of w1, w3 (14336x4096), w2 (4096x14336), q, o
            # (4096x4096) as 2-bit weights, every matrix distinct (1.68 GB), one recorded batch per sweep
            M = dims[0]
            layers = int(rest[0]) if rest else 32
            shapes = [(14336, 4096), (14336, 4096), (4096, 14336), (4096, 4096), (4096, 4096)]
            mats = []
            for _ in range(layers):
                for (O, I) in shapes:
                    mats.append((torch.randint(-2 ** 31, 2 ** 31 - 1, (O, I // 16), dtype=torch.int32, device=dev,
                                               generator=g), torch.full((O,), 0.05, device=dev), O, I))
            xs_ = {I: torch.randn(M, I, device=dev, generator=g) for I in (4096, 14336)}
            ys_ = {O: torch.empty(M, O, device=dev) for O in (4096, 14336)}

            def sweep():
                for p2, sc, O, I in mats:
                    ctx.ternary_gemv(xs_[I], p2, sc, ys_[O], M, I, O)
            sweep()
            ctx.finish()
            ctx.batch_begin()
            sweep()
            batch = ctx.batch_end()
            ms = timed(lambda i: batch.launch(), args.steps, max(args.warmup, 3))
            nbytes = sum(O * I / 4 + 4 * O + 4 * M * (I + O) for _, _, O, I in mats)
            out = {"kernel": "ternary GEMV sweep (%d layers x 5 matrices)" % layers, "bound": "hbm",
                   "achieved": nbytes / ms / 1e6, "peak": hbm_peak, "unit": "GB/s", "bytes_per_launch": nbytes,
                   "tokens_per_s": M / (ms * 1e-3), "us_per_matrix": ms * 1e3 / len(mats)}
        elif kind == "step":
            T, I, O = dims
            x = torch.randn(T, I, device=dev, generator=g)
            dy = torch.randn(T, O, device=dev, generator=g) * 0.02
            st = torch.randint(0, 255, (O * I // 4 * 3,), dtype=torch.uint8, device=dev, generator=g)
            sc, v = torch.full((O,), 0.05, device=dev), torch.zeros(O, device=dev)
            y, dx = torch.empty(T, O, device=dev), torch.empty(T, I, device=dev)
            gw, p2 = torch.empty(O, I, device=dev), torch.zeros(O, I // 16, dtype=torch.int32, device=dev)
            if rest:
                a, b = rest[0].split("/")
                ctx.set_gemm_mode("tensor", int(a), int(b))
            ms = timed(lambda i: ctx.counter_linear_step(x, dy, st, sc, v, y, dx, gw, p2, 11, I, O, T, O, 0, 3e-3,
                                                         0.0, 0.9, 1e-3, i), args.steps, max(args.warmup, 3))
            fl = 6.0 * T * I * O
            out = {"kernel": "linear step (split, expand, 3 contractions, update)", "bound": "tensor",
                   "achieved": fl / ms / 1e9, "peak": tf_peak, "unit": "TFLOP/s", "flop_per_launch": fl}
        elif kind == "stepmany":
            from motifcl_b200 import synth
            from motifcl_b200.runtime import linear_descs
            T = int(rest[0]) if rest else 8192
            shapes = synth.stories15m_linears()[:dims[0]]
            ents = []
            for sh in shapes:
                I, O = sh.in_features, sh.out_features
                ents.append(dict(x=torch.randn(T, I, device=dev, generator=g),
                                 grad_out=torch.randn(T, O, device=dev, generator=g) * 0.02,
                                 state=torch.randint(0, 255, (O * I // 4 * 3,), dtype=torch.uint8, device=dev, generator=g),
                                 scale=torch.full((O,), 0.05, device=dev), v=torch.zeros(O, device=dev),
                                 y=torch.empty(T, O, device=dev), grad_x=torch.empty(T, I, device=dev),
                                 grad_w=torch.empty(O, I, device=dev),
                                 packed2_out=torch.zeros(O, I // 16, dtype=torch.int32, device=dev),
                                 in_features=I, out_features=O, batch=T, update_rows=O, row_offset=0))
            descs = linear_descs(ents)
            ms = timed(lambda i: ctx.counter_linear_step_many(descs, 11, 3e-3, 0.0, 0.9, 1e-3, i), 5, 3)
            W = sum(sh.in_features * sh.out_features for sh in shapes)
            nbytes = 8.0 * T * sum(sh.in_features + sh.out_features for sh in shapes) + 4.75 * W
            out = {"kernel": "grouped step (digits, contractions, split-K reduction, update)", "bound": "hbm",
                   "achieved": nbytes / ms / 1e6, "peak": hbm_peak, "unit": "GB/s", "bytes_per_launch": nbytes,
                   "layers": len(shapes), "tokens": T}
        else:
            raise SystemExit("unknown --micro kind")
    ctx.finish()        # raises if a kernel of the timed region reported an abandoned wait
    out.update({"frac": out["achieved"] / out["peak"], "peak_kind": peak_kind, "ms": ms, "micro": args.micro,
                "steps": args.steps, "clocks": clk.summary(), "gpu_launches": ctx.launch_count})
    print(json.dumps(out))


# MotifCL's published records for the ops of this path (reports/vulkan-perf/*.json, Radeon RX 580, median
# wall time of dispatch + wait): op -> {shape: (median_us, throughput, unit)}
PUBLISHED_RX580 = {
    "counter_update_f32": {"in1024_out256_N8": (608.6, None, None)},
    "counter_decode_weight_f32": {"in1024_out256": (188.3, None, None)},
    "counter_backward_input_f32": {"in1024_out256_N8": (501.2, 8.37, "GFLOP/s")},
    "matmul_f32": {"512x512x512": (None, 609.5, "GFLOP/s")},
    "matmul_f32_nt": {"512x512x512": (None, 451.2, "GFLOP/s")},
    "matmul_f32_tn": {"512x512x512": (None, 538.2, "GFLOP/s")},
    "matmul_f32_m1": {"1x2048x2048": (497.9, 16.8, "GFLOP/s")},
}


def run_refperf(args):
    """--micro refperf  runs MotifCL's OWN micro-benchmark program (benchmarks/bench_vulkan_perf.cpp, compiled
    unmodified against the CUDA adapter: motifcl_b200/adapter/Makefile) for the ops of the counter-linear path and
    prints its records beside the numbers MotifCL publishes for them."""
    import glob
    import subprocess
    exe = os.path.join(ROOT, "motifcl_b200", "adapter", "_build", "bench_vulkan_perf")
    if not os.path.isfile(exe):
        print(json.dumps({"micro": "refperf", "unavailable": "adapter binaries are not built (make -C motifcl_b200/adapter "
                                                             "needs the MotifCL tree)"}))
        return
    import tempfile
    out_dir = tempfile.mkdtemp(prefix="motifcl-vulkan-perf-")
    rows = []
    for flt in ("counter_", "matmul_f32"):
        r = subprocess.run([exe, "--filter", flt, "--out", os.path.join(out_dir, flt.strip("_"))], capture_output=True,
                           text=True, timeout=600)
        if r.returncode != 0:
            print(json.dumps({"micro": "refperf", "filter": flt, "returncode": r.returncode,
                              "stderr": r.stderr[-400:]}))
            continue
        for f in sorted(glob.glob(os.path.join(out_dir, flt.strip("_"), "*.json"))):
            rec = json.load(open(f))
            for row in rec["rows"]:
                pub = PUBLISHED_RX580.get(rec["op"], {}).get(row["shape"])
                if row.get("result") == "ERROR" or pub is None:
                    continue
                rows.append({"op": rec["op"], "shape": row["shape"], "device": rec["vulkan_device"],
                             "median_us": row["median_us"], "min_us": row["min_us"],
                             "throughput": row.get("achieved_gflops", row.get("achieved_gbs")),
                             "published_rx580_median_us": pub[0], "published_rx580_throughput": pub[1],
                             "speedup_wall": (pub[0] / row["median_us"]) if pub[0] else
                             (row.get("achieved_gflops", 0.0) / pub[1] if pub[1] else None)})
    print(json.dumps({"micro": "refperf", "program": "MotifCL benchmarks/bench_vulkan_perf.cpp (unmodified)",
                      "methodology": "median wall time of 50 runs after 5 warm-ups, dispatch + wait", "rows": rows}))


def run_trainer15m(args):
    """--micro trainer15m[:BATCH[:STEPS]]  runs MotifCL's OWN harnesses for its headline tokens/s, compiled unmodified
    against the CUDA adapter (motifcl_b200/adapter/Makefile): tests/bench_ternary15m.cpp (the 6-block ternary15m stack,
    forward + backward + counter updates + sgd, one submit per step) and tools/train_ternary15m.cpp (the trainer itself,
    on seeded synthetic records: the tokenised corpus of the published run is in neither tree).  BATCH x 256 tokens per
    step; MotifCL's published run is BATCH = 16 on a Radeon RX 580 (docs/TERNARY15M_PRETRAIN_RESULTS.md:3,24-26)."""
    import re
    import subprocess
    import tempfile
    build = os.path.join(ROOT, "motifcl_b200", "adapter", "_build")
    parts = args.micro.split(":")
    batch = int(parts[1]) if len(parts) > 1 else 16
    steps = int(parts[2]) if len(parts) > 2 else 100
    rec = {"micro": "trainer15m", "batch": batch, "seq": 256, "tokens_per_step": batch * 256, "data": "synthetic",
           "published_rx580_tokens_per_s": 4152}
    if not os.path.isfile(os.path.join(build, "bench_ternary15m")):
        rec["unavailable"] = "adapter binaries are not built (make -C motifcl_b200/adapter needs the MotifCL tree)"
        print(json.dumps(rec))
        return
    env = dict(os.environ, BENCH_BATCHED="1", BENCH_B=str(batch), BENCH_STEPS=str(steps))
    r = subprocess.run([os.path.join(build, "bench_ternary15m")], capture_output=True, text=True, timeout=900, env=env)
    m = re.search(r"ms/step=([0-9.]+)\s+tokens/step=(\d+)\s+tok/s=([0-9.e+]+)", r.stdout)
    rec["bench_ternary15m"] = ({"ms_per_step": float(m.group(1)), "tokens_per_s": float(m.group(3))} if r.returncode == 0 and m
                               else {"returncode": r.returncode, "stderr": r.stderr[-300:]})
    sys.path.insert(0, os.path.join(ROOT, "motifcl_b200", "adapter"))
    import make_synthetic_records as msr
    with tempfile.TemporaryDirectory() as tmp:
        msr.write_dataset(os.path.join(tmp, "data"), seq=256, train_records=4096, val_records=96, seed=1)
        env = dict(os.environ, DATA_DIR=os.path.join(tmp, "data"), OUT_DIR=os.path.join(tmp, "out"), STEPS=str(2 * steps),
                   BATCH=str(batch), SEQ="256", LOG_EVERY=str(steps), EVAL_EVERY="1000000", CKPT_EVERY="1000000", RESUME="0")
        r = subprocess.run([os.path.join(build, "train_ternary15m")], capture_output=True, text=True, timeout=900, env=env)
    logs = re.findall(r"^step (\d+) loss ([0-9.]+) .*?([0-9]+) tok/s", r.stdout, flags=re.M)
    # the second window is free of first-step allocations
    rec["train_ternary15m"] = ({"tokens_per_s": float(logs[-1][2]), "loss_first_window": float(logs[0][1]),
                                "loss_last_window": float(logs[-1][1]), "steps": int(logs[-1][0])}
                               if r.returncode == 0 and logs else {"returncode": r.returncode, "stderr": r.stderr[-300:]})
    print(json.dumps(rec))


def gemv_tp_sweep(ctx, dev, local, rank, world, M, layers, steps, warmup, use_nccl=False):
    """The decode-GEMV sweep with the weights sharded over the ranks of the job (q, w1, w3 split by output features;
    o, w2 split by input features + one sum over the ranks each): what a tensor-parallel decoder does per token.  The
    sums run as the library's one-shot peer kernel (motifcl_b200.peer; the sweep is then one recorded batch per rank)
    or, with use_nccl, as NCCL all-reduces launched eagerly.  Returns the record (the same on every rank)."""
    import torch
    import torch.distributed as dist
    from motifcl_b200 import gemv_tp
    from motifcl_b200.peer import PeerReducer
    dim, ffn = 4096, 14336
    red = None if (use_nccl or world == 1) else PeerReducer(ctx, M * dim)
    g = torch.Generator(device=dev).manual_seed(1234)          # every rank draws the same full matrices
    rnd = lambda O, I: torch.randint(-2 ** 31, 2 ** 31 - 1, (O, I // 16), dtype=torch.int32, device=dev, generator=g)
    sc = lambda O: torch.full((O,), 0.05, device=dev)
    blocks = []
    for _ in range(layers):
        q = gemv_tp.ColumnParallelGemv(rnd(dim, dim), sc(dim), dim, rank, world)
        o = gemv_tp.RowParallelGemv(rnd(dim, dim), sc(dim), dim, rank, world)
        mlp = gemv_tp.TensorParallelMlp(rnd(ffn, dim), sc(ffn), rnd(ffn, dim), sc(ffn), rnd(dim, ffn), sc(dim), dim, ffn,
                                        rank, world)
        blocks.append((q, o, mlp))
        torch.cuda.empty_cache()
    x = torch.randn(M, dim, device=dev, generator=g)
    fn = lambda a, p2, s_, y_, m, i, o_: ctx.ternary_gemv(a, p2, s_, y_, m, i, o_)
    yq = torch.empty(M, blocks[0][0].rows, device=dev)
    xo = torch.randn(M, blocks[0][1].cols, device=dev, generator=g)
    yo, ym = torch.empty(M, dim, device=dev), torch.empty(M, dim, device=dev)
    h1, h3 = torch.empty(M, blocks[0][2].cols, device=dev), torch.empty(M, blocks[0][2].cols, device=dev)

    def sweep():
        for q, o, mlp in blocks:
            q(fn, x, yq)
            o(fn, xo, yo, reducer=red)
            mlp(fn, x, h1, h3, ym, reducer=red, gate=False)

    parity = None
    if red is not None:
        # the peer sum against NCCL's, on the first o layer and the first FFN
        q0, o0, mlp0 = blocks[0]
        o0(fn, xo, yo, reducer=red)
        mlp0(fn, x, h1, h3, ym, reducer=red, gate=False)
        ctx.finish()
        a_o, a_m = yo.clone(), ym.clone()
        o0(fn, xo, yo)
        mlp0(fn, x, h1, h3, ym, gate=False)
        torch.cuda.synchronize()
        err = max(float((a_o - yo).abs().max() / yo.abs().max()), float((a_m - ym).abs().max() / ym.abs().max()))
        parity = {"peer_sum_vs_nccl_max_rel": err, "ok": err <= 1e-6}

    def timed(steps, warm):
        for _ in range(warm):
            sweep()
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(steps):
            sweep()
        e1.record()
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()
        ms = e0.elapsed_time(e1) / steps
        if world > 1:
            t = torch.tensor([ms], device=dev)
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
            ms = float(t.item())
        return ms
    # One recorded batch per sweep when no collective library call is inside it (one rank, or the peer kernel, whose
    # call counter lives in device memory: an even number of sums per sweep keeps the two partial areas alternating
    # across replays).  With NCCL all-reduces the sweep is launched eagerly: a batch is a stream capture of the context's
    # stream, and torch's NCCL collectives run on the process group's own stream behind event hand-offs, which must not
    # be captured by this library's thread-local capture.  Every rank takes the same path: the ranks agree on whether
    # recording worked before any of them replays.
    recorded = False
    batch = None
    if not (use_nccl and world > 1):
        try:
            sweep()
            ctx.finish()
            ctx.batch_begin()
            try:
                sweep()
            finally:
                batch = ctx.batch_end()
        except Exception as exc:      # noqa: BLE001
            print(f"[rank {rank}] recording refused ({exc}); timing eager launches", file=sys.stderr)
            batch = None
        if red is not None:
            red.seq = 2 * layers        # the sums that really ran so far (the recorded ones did not): same on every rank
        ok = torch.tensor([1 if batch is not None else 0], device=dev)
        if world > 1:
            torch.cuda.synchronize()
            dist.all_reduce(ok, op=dist.ReduceOp.MIN)
        if int(ok.item()) == 1:
            sweep = batch.launch
            sweep()
            ctx.finish()
            recorded = True
    launches0 = ctx.launch_count
    with ClockSampler(local) as clk:
        ms = timed(steps, max(warmup, 3))
    hbm_peak, _, peak_kind = measured_peaks()
    nbytes = layers * (2 * (dim * dim / 4) + 3 * (dim * ffn / 4))          # 2-bit weights of the whole model
    rec = {"kernel": "tensor-parallel ternary GEMV sweep", "n_gpus": world, "M": M,
           "layers": layers, "ms_per_sweep": ms, "tokens_per_s": M / (ms * 1e-3),
           "weight_bytes": nbytes, "achieved": nbytes / ms / 1e6, "unit": "GB/s (all ranks)",
           "peak": hbm_peak * world, "frac": nbytes / ms / 1e6 / (hbm_peak * world),
           "peak_kind": peak_kind, "sums_per_sweep": 2 * layers if world > 1 else 0,
           "recorded_batch": recorded, "sum": "nccl" if (use_nccl and world > 1) else ("peer kernel" if world > 1 else None),
           "parity": parity, "clocks": clk.summary(), "gpu_launches": ctx.launch_count - launches0}
    ctx.finish()
    if batch is not None:
        batch.close()
    if red is not None:
        red.close()
    return rec


def run_gemv_tp(args):
    """--micro gemvtp:M[:LAYERS[:nccl]]  the tensor-parallel decode-GEMV sweep (gemv_tp_sweep).  Run under torchrun; with
    one rank it is the plain sweep."""
    import torch
    import torch.distributed as dist
    from motifcl_b200 import Context
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    dev = f"cuda:{local}"
    if world > 1:
        dist.init_process_group("nccl", device_id=torch.device(dev))
    torch.cuda.set_stream(torch.cuda.Stream(device=local))
    ctx = Context.on_torch_stream(local)
    _, shape, *rest = args.micro.split(":")
    M = int(shape)
    layers = int(rest[0]) if rest else 32
    use_nccl = len(rest) > 1 and rest[1] == "nccl"
    rec = gemv_tp_sweep(ctx, dev, local, rank, world, M, layers, args.steps, args.warmup, use_nccl)
    rec["micro"] = args.micro
    if rank == 0:
        print(json.dumps(rec))
    if world > 1:
        dist.destroy_process_group()


def time_wide_workload(ctx, wl, dev, steps, warmup, group=None):
    """Times WideStack steps of a wide-layer workload (cfg3 on one GPU, cfg4 data-parallel) with CUDA events on
    the launching stream; returns the record for the `also` object.  Inputs of one layer (X and dY of 16384 x 2048
    floats and more) exceed L2, and consecutive layers use other buffers."""
    import torch
    import torch.distributed as dist
    from motifcl_b200.step import Hyper, WideStack
    world = 1 if group is None else dist.get_world_size(group)
    stack = WideStack(ctx, wl["linears"], wl["tokens"], Hyper(), dev, wl["sigma"], group)
    l0 = ctx.launch_count
    for _ in range(warmup):
        stack.step()
    stack.sync_streams()
    if world > 1:
        dist.barrier()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    l1 = ctx.launch_count
    e0.record()
    for _ in range(steps):
        stack.step()
    stack.sync_streams()
    e1.record()
    if world > 1:
        dist.barrier()
    torch.cuda.synchronize()
    ms = e0.elapsed_time(e1) / steps
    if world > 1:
        t = torch.tensor([ms], device=dev)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms = float(t.item())
    ctx.finish()
    alg = algorithmic(wl)
    hbm_peak, tf_peak, peak_kind = measured_peaks()
    tf = alg["gemm_flop"] / (ms * 1e-3) / 1e12           # per GPU: the whole step (pre-passes and update included)
    rec = {"workload": wl["desc"], "n_gpus": world, "tokens_per_gpu": wl["tokens"], "linears": len(wl["linears"]),
           "weights": alg["weights"], "steps": steps, "warmup": warmup, "ms_per_step": ms,
           "tokens_per_s": wl["tokens"] * world / (ms * 1e-3), "gpu_launches_per_step": (ctx.launch_count - l1) // steps,
           "roofline": {"kernel": "whole step per GPU: operand splits, tc_gemm_kernel contractions (fp16 terms, 2 / 2 / 3 "
                                  "products), fused update" + (", collectives overlapped" if world > 1 else ""),
                        "bound": "tensor", "achieved": tf, "peak": tf_peak, "unit": "TFLOP/s", "frac": tf / tf_peak,
                        "peak_kind": f"{peak_kind} bf16 sustained", "flop_per_step": alg["gemm_flop"],
                        "pass_adjusted": {"bf16_pass_units_per_3_useful": 7.0, "ceiling": tf_peak * 3.0 / 7.0,
                                          "frac": tf / (tf_peak * 3.0 / 7.0)}}}
    if world > 1:
        rec["collectives_per_step"] = {"reduce_scatter_bytes_in": 4.0 * alg["weights"],
                                       "all_gather_bytes_out": alg["weights"] / 4.0 + 4.0 * alg["rows"]}
    del stack
    torch.cuda.empty_cache()
    return rec


def gemv_cpu_baseline():
    """The reference's host GEMV, native::matmul_f32_m1 (MotifCL src/runtime/native_matmul.cpp:110-133: one thread, SSE,
    dense fp32 [in, out] weights), compiled from the reference's own source where that library was built, timed on
    one 4096 x 14336 matrix of the decode sweep and scaled by weights to the 32-layer sweep."""
    import oracle
    kind, fn = ("reference", oracle.ref.matmul_m1) if oracle.ref is not None else ("port", oracle.port.matmul_m1)
    K, N = 4096, 14336
    rng = np.random.default_rng(5)
    b = rng.integers(-1, 2, size=(K, N)).astype(np.float32)
    a = rng.standard_normal(K).astype(np.float32)
    fn(a, b)
    reps, t0 = 0, time.perf_counter()
    while reps < 3 or time.perf_counter() - t0 < 3.0:
        fn(a, b)
        reps += 1
    t = (time.perf_counter() - t0) / reps
    sweep_weights = 32 * (3 * 4096 * 14336 + 2 * 4096 * 4096)
    t_sweep = t * sweep_weights / (K * N)
    return {"value": 1.0 / t_sweep, "unit": "tokens/s at M = 1", "cores": 1, "kind": kind,
            "sample": f"matmul_f32_m1 on one dense fp32 [4096, 14336] matrix ({K * N * 4 / 1e6:.0f} MB), {reps} calls of "
                      f"{t * 1e3:.1f} ms; scaled by weights to the 160 matrices of the sweep",
            "ms_per_sweep_scaled": t_sweep * 1e3, "gb_per_s": K * N * 4 / t / 1e9}


def run_also(args):
    """--micro also: the other single-GPU configurations of the metric, each timed like its --micro form; one JSON
    object.  Run by the default benchmark in a child process so that a failure here cannot take the main line down."""
    import io
    import contextlib
    out = {}

    def micro(spec, steps, warmup):
        a = argparse.Namespace(**vars(args))
        a.micro, a.steps, a.warmup = spec, steps, warmup
        buf = io.StringIO()
        with contextlib.redirect_stdout(buf):
            run_micro(a)
        return json.loads(buf.getvalue().strip().splitlines()[-1])

    try:
        import torch
        from motifcl_b200 import Context
        torch.cuda.set_device(0)
        torch.cuda.set_stream(torch.cuda.Stream(device=0))
        ctx = Context.on_torch_stream(0)
        out["cfg3"] = time_wide_workload(ctx, workload("cfg3"), "cuda:0", 2, 1)
        ctx.close()
    except Exception as exc:       # noqa: BLE001
        out["cfg3"] = {"error": repr(exc)[:300]}
    try:
        sweeps = {f"M{m}": micro(f"gemvsweep:{m}", 20, 5) for m in (1, 4, 16)}
        out["cfg5"] = {"workload": "decode GEMV sweep: 32 layers x (w1, w3 14336x4096; w2 4096x14336; q, o 4096x4096) as 2-bit "
                                   "words, every matrix distinct (1.68 GB: larger than L2)",
                       "sweeps": {k: {"ms_per_sweep": v["ms"], "tokens_per_s": v["tokens_per_s"], "us_per_matrix": v["us_per_matrix"],
                                      "roofline": {"bound": "hbm", "achieved": v["achieved"], "peak": v["peak"], "unit": "GB/s",
                                                   "frac": v["frac"], "peak_kind": v["peak_kind"],
                                                   "bytes_per_sweep": v["bytes_per_launch"]}}
                                  for k, v in sweeps.items()}}
        out["cfg5"]["cpu_baseline"] = gemv_cpu_baseline()
    except Exception as exc:       # noqa: BLE001
        out["cfg5"] = {"error": repr(exc)[:300]}
    try:
        u = micro("update:8192x4096", 50, 5)
        out["update_hbm"] = {"workload": "fused counter update of an 8192 x 4096 layer, buffer sets rotated (larger than L2)",
                             "ms": u["ms"], "roofline": {"bound": "hbm", "achieved": u["achieved"], "peak": u["peak"],
                                                         "unit": "GB/s", "frac": u["frac"], "peak_kind": u["peak_kind"],
                                                         "bytes_per_launch": u["bytes_per_launch"]}}
    except Exception as exc:       # noqa: BLE001
        out["update_hbm"] = {"error": repr(exc)[:300]}
    print(json.dumps(out))


def also_in_child(timeout_s: int = 420):
    import subprocess
    try:
        r = subprocess.run([sys.executable, os.path.abspath(__file__), "--micro", "also"], capture_output=True, text=True,
                           timeout=timeout_s)
        lines = [ln for ln in r.stdout.strip().splitlines() if ln.startswith("{")]
        if r.returncode == 0 and lines:
            return json.loads(lines[-1])
        return {"error": f"child exited {r.returncode}: {r.stderr[-300:]}"}
    except Exception as exc:       # noqa: BLE001
        return {"error": repr(exc)[:300]}


def dp_parity_check(stack, xs, dys, dev, group):
    """After the timed region, on every rank: snapshot the local row shards, run ONE more data-parallel step, download
    the reduce-scattered gradient shard and the updated shard, run the CPU checker's update on the downloaded gradient
    with the shard's row offset and the step's seed, and compare bytes.  Also: the all-gathered 2-bit words equal the
    checker's pack2 of the gathered states, and the replicated scales equal the gathered shard scales."""
    import torch
    import torch.distributed as dist
    import oracle
    o = oracle.port
    o.set_threads(max(1, len(os.sched_getaffinity(0)) // dist.get_world_size(group)))
    h = stack.h
    stack.sync_streams()
    torch.cuda.synchronize()
    pre = []
    for l in stack.linears:
        sh = l.sharded
        sl = slice(sh.off, sh.off + sh.rows)
        pre.append((sh.state.cpu().numpy().copy(), sh.scale[sl].cpu().numpy().copy(), sh.v.cpu().numpy().copy()))
    seed = (12345 + stack.step_index) & 0xFFFFFFFF
    stack.step(xs, dys)
    stack.sync_streams()
    torch.cuda.synchronize()
    bad = 0
    checked = 0
    for l, (st0, sc0, v0) in zip(stack.linears, pre):
        sh = l.sharded
        I = l.shape.in_features
        sl = slice(sh.off, sh.off + sh.rows)
        gw = sh.gw_shard[:sh.rows].cpu().numpy()
        e = o.update_dense(st0, sc0, v0, gw, h.C, I, sh.rows, sh.off, h.lr, h.lr_scale, h.rms_beta, h.rms_eps, seed)
        bad += int(not np.array_equal(sh.state.cpu().numpy(), e[0]))
        bad += int(not np.array_equal(sh.scale[sl].cpu().numpy().view(np.uint32), e[1].view(np.uint32)))
        bad += int(not np.array_equal(sh.v.cpu().numpy().view(np.uint32), e[2].view(np.uint32)))
        bad += int(not np.array_equal(sh.packed2[sl].cpu().numpy().view(np.uint32), e[3]))
        # replicated tensors: gather every rank's state shard, pack on the host, compare with the local full copy
        world = dist.get_world_size(group)
        parts = [torch.empty_like(sh.state) for _ in range(world)]
        dist.all_gather(parts, sh.state, group=group)
        full_state = torch.cat(parts).cpu().numpy()
        bad += int(not np.array_equal(sh.packed2.cpu().numpy().view(np.uint32), o.pack2(full_state, h.C, I, sh.O)))
        checked += 5
    t = torch.tensor([bad, checked], device=dev, dtype=torch.int64)
    dist.all_reduce(t, op=dist.ReduceOp.SUM, group=group)
    bad, checked = int(t[0].item()), int(t[1].item())
    return {"result": "bit-exact" if bad == 0 else f"{bad} tensors differ", "tensors_compared": checked,
            "what": "per rank and linear: state / scale / v / 2-bit shard after one step vs the CPU checker's update of the "
                    "downloaded reduce-scattered gradient (row_offset, seed of the step); all-gathered 2-bit words vs "
                    "pack2 of the gathered states", "seed": seed}


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=50)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default="cfg2")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-also", action="store_true", help="skip the other configurations (cfg3 / cfg5 / update; cfg4 and "
                                                            "dp_parity on several GPUs)")
    ap.add_argument("--lanes", type=int, default=8, help="contexts (streams) that independent linears are spread over")
    ap.add_argument("--no-group", action="store_true", help="one call per linear (spread over --lanes) instead of the grouped step call")
    ap.add_argument("--eager", action="store_true", help="do not record the step into one batch (for per-kernel profiling)")
    ap.add_argument("--micro", default=None, help="single-kernel timing, see run_micro()")
    args = ap.parse_args()
    if args.micro and args.micro.startswith("gemvtp"):
        return run_gemv_tp(args)
    if args.micro == "refperf":
        return run_refperf(args)
    if args.micro == "also":
        return run_also(args)
    if args.micro and args.micro.startswith("trainer15m"):
        return run_trainer15m(args)
    if args.micro:
        return run_micro(args)
    wl = workload(args.workload)
    if args.impl == "reference":
        return run_reference(args, wl)

    import torch
    import torch.distributed as dist
    from motifcl_b200 import Context, synth
    from motifcl_b200.step import CounterLinearState, CounterStack, Hyper

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    assert world == args.gpus or world == 1, "launch with torchrun --nproc-per-node N for N > 1"
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    group = None
    if world > 1:
        dist.init_process_group("nccl", device_id=dev)
        group = dist.group.WORLD
    torch.cuda.set_stream(torch.cuda.Stream(device=local))   # a recordable (non-default) stream
    ctx = Context.on_torch_stream(local)
    cfg, T, sigma = wl["cfg"], wl["tokens"], wl["sigma"]
    if any(l.in_features > 1024 or l.out_features > 1024 for l in wl["linears"]):
        # wide-layer workloads keep activations per shape, not per layer
        rec = time_wide_workload(ctx, wl, dev, args.steps, max(args.warmup, 1), group)
        if rank == 0:
            print(json.dumps({"metric": METRIC, "value": rec["tokens_per_s"], "unit": UNIT, "n_gpus": world, "steps": args.steps,
                              "warmup": max(args.warmup, 1), "ms_per_step": rec["ms_per_step"], "higher_is_better": True,
                              "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
                              "config": base_config(args.workload, wl, world), "roofline": rec["roofline"],
                              "gpu_launches": rec["gpu_launches_per_step"] * args.steps, "e2e": None, "cpu_baseline": None}))
        if world > 1:
            dist.destroy_process_group()
        return

    # ---- inputs: pinned host copies (for e2e) and device-resident copies (for value) ----------
    lin_states, xs_h, dys_h = [], [], []
    for idx, l in enumerate(wl["linears"]):
        O, I = l.out_features, l.in_features
        sc, v = synth.scale_v(cfg, idx, O, I)
        lin_states.append(CounterLinearState(l, synth.counters(cfg, idx, O, I), sc, v, dev, rank, world))
        # every rank draws its own tokens (data parallel): offset the linear index by rank
        xs_h.append(torch.from_numpy(synth.activations(cfg, idx + 100 * rank, T, I)).pin_memory())
        dys_h.append(torch.from_numpy(synth.upstream_grad(cfg, idx + 100 * rank, T, O, sigma)).pin_memory())
    stack = CounterStack(ctx, lin_states, Hyper(), T, group, lanes=args.lanes, grouped=not args.no_group)
    xs = [t.to(dev, non_blocking=True) for t in xs_h]
    dys = [t.to(dev, non_blocking=True) for t in dys_h]
    torch.cuda.synchronize()
    in_bytes = sum(t.numel() * 4 for t in xs_h + dys_h)

    def barrier():
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()

    def timed(fn, steps, warmup):
        """K steps between two events on the launching stream (the figure that is reported), with an event after every
        step for the median."""
        for _ in range(warmup):
            fn()
        stack.sync_streams()
        barrier()
        evs = [torch.cuda.Event(enable_timing=True) for _ in range(steps + 1)]
        l0 = ctx.launch_count
        evs[0].record()
        for i in range(steps):
            fn()
            if i + 1 < steps:
                evs[i + 1].record()
        stack.sync_streams()            # several GPUs: the tail of the last step runs on the communication stream
        evs[steps].record()
        barrier()
        ms = evs[0].elapsed_time(evs[steps])
        per = sorted(evs[i].elapsed_time(evs[i + 1]) for i in range(steps))
        if world > 1:
            t = torch.tensor([ms], device=dev)
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
            ms = float(t.item())
        return ms / steps, (ctx.launch_count - l0), per[len(per) // 2]

    # ---- device-resident throughput ------------------------------------------------------
    with ClockSampler(local) as clk:
        ms_step, launches, ms_median = timed(lambda: stack.step(xs, dys, recorded=not args.eager), args.steps,
                                             max(args.warmup, 3))
    clocks = clk.summary()
    if world > 1:
        launches += stack.comm_launches()

    # ---- roofline of the dominant kernel: timed alone on the launching stream ---------------
    alg = algorithmic(wl)
    hbm_peak, tf_peak, peak_kind = measured_peaks()

    ms_upd, n_upd, _ = timed(stack.update_only, args.steps, 3)
    if args.eager or args.no_group:
        ms_gemm, n_gemm, _ = timed(lambda: stack.products_only(xs, dys), args.steps, 3)
    else:
        # recorded like the step itself, so that the figure is the kernels' time and not the host's per-call work
        # (an eager grouped call encodes ~170 tensor maps and builds its tables before it launches)
        prod_batch = stack._record(lambda: stack.products_only(xs, dys))
        ms_gemm, n_gemm, _ = timed(prod_batch.launch, args.steps, 3)
        prod_batch.close()
    gemm_tf = alg["gemm_flop"] / (ms_gemm * 1e-3) / 1e12
    gemm_gbs = alg["gemm_bytes"] / (ms_gemm * 1e-3) / 1e9
    upd_gbs = alg["update_bytes"] / world / (ms_upd * 1e-3) / 1e9      # each rank updates its row shard
    # The scope table counts the three products as 6*tokens*weights flop against the dense bf16 rate.  Two more
    # views explain the number: the pass-adjusted ceiling (fp32 fidelity costs 2 + 2 passes of fp16 terms for Y and
    # dX and 3 for dW = 7 per 3 useful) and the HBM view
    # (algorithmic bytes of the products at the copy bandwidth), which is the larger ideal time when layers are narrow.
    units = 7.0
    traffic = MEASURED_TRAFFIC_BYTES.get(args.workload)
    roofline = {"kernel": "counter-linear contractions (Y, dX, dW) of all linears: tc_gemm_kernel (two fp16 terms per "
                          "fp32 operand, CTA pairs)",
                "bound": "tensor", "achieved": gemm_tf, "peak": tf_peak, "unit": "TFLOP/s", "frac": gemm_tf / tf_peak,
                "peak_kind": f"{peak_kind} bf16 sustained", "traffic": traffic,
                "flop_per_step": alg["gemm_flop"], "ms": ms_gemm,
                "pass_adjusted": {"bf16_pass_units_per_3_useful": units, "ceiling": tf_peak * 3.0 / units,
                                  "frac": gemm_tf / (tf_peak * 3.0 / units)},
                "hbm_view": {"bytes_per_step": alg["gemm_bytes"], "achieved": gemm_gbs, "peak": hbm_peak, "unit": "GB/s",
                             "frac": gemm_gbs / hbm_peak,
                             "ideal_ms": alg["gemm_bytes"] / (hbm_peak * 1e9) * 1e3,
                             "ideal_ms_tensor_single_pass": alg["gemm_flop"] / (tf_peak * 1e12) * 1e3},
                "update": {"bound": "hbm", "achieved": upd_gbs, "peak": hbm_peak, "unit": "GB/s",
                           "frac": upd_gbs / hbm_peak, "bytes_per_step": alg["update_bytes"], "ms": ms_upd,
                           "note": "all 42 state tensors fit in L2 at this workload; the HBM-resident figure is "
                                   "also.update_hbm"}}

    # ---- end to end from pinned host memory --------------------------------------------------
    out_h = [(torch.empty_like(l.state, device="cpu").pin_memory(),
              torch.empty_like(l.packed2, device="cpu").pin_memory(),
              torch.empty_like(l.scale, device="cpu").pin_memory(),
              torch.empty_like(l.v, device="cpu").pin_memory()) for l in stack.linears]
    out_bytes = sum(sum(t.numel() * t.element_size() for t in o) for o in out_h)

    copy_stream = torch.cuda.Stream(device=local)
    main_stream = torch.cuda.current_stream(local)
    ready = [torch.cuda.Event() for _ in xs]
    consumed = torch.cuda.Event()
    consumed.record(main_stream)
    e2e_seed = [0]

    def e2e_step():
        # host->device copies run on their own stream, linear by linear; the step of linear i
        # starts as soon as its X and dY have landed, so transfer and compute overlap
        copy_stream.wait_event(consumed)          # the previous step has finished reading xs / dys
        with torch.cuda.stream(copy_stream):
            for i in range(len(xs)):
                xs[i].copy_(xs_h[i], non_blocking=True)
                dys[i].copy_(dys_h[i], non_blocking=True)
                ready[i].record(copy_stream)
        if world == 1:
            for i in range(len(xs)):
                main_stream.wait_event(ready[i])
                stack.step_linear(i, xs[i], dys[i], 12345 + e2e_seed[0])
        else:
            main_stream.wait_event(ready[-1])
            stack.step(xs, dys)
        e2e_seed[0] += 1
        consumed.record(main_stream)
        stack.sync_streams()                      # the updated shards come from the communication stream
        for l, o in zip(stack.linears, out_h):
            o[0].copy_(l.state, non_blocking=True)
            o[1].copy_(l.packed2, non_blocking=True)
            o[2].copy_(l.scale, non_blocking=True)
            o[3].copy_(l.v, non_blocking=True)
    ms_e2e, _, _ = timed(e2e_step, max(2, args.steps // 4), 2)

    cpu = None
    also = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        cpu, _ = cpu_reference_rate(wl)
    if world == 1 and not args.no_also:
        also = also_in_child()
    dp_parity = None
    if world > 1 and not args.no_also:
        try:
            dp_parity = dp_parity_check(stack, xs, dys, dev, group)
        except Exception as exc:       # noqa: BLE001
            dp_parity = {"result": "not run", "error": repr(exc)[:300]}
        del stack, xs, dys, lin_states
        torch.cuda.empty_cache()
        try:
            also = {"cfg4": time_wide_workload(ctx, workload("cfg4"), dev, 2, 1, group)}
        except Exception as exc:       # noqa: BLE001
            also = {"cfg4": {"error": repr(exc)[:300]}}
        torch.cuda.empty_cache()
        try:
            # the decode sweep with the 8B-scale matrices sharded over the ranks (sums through the peer kernel)
            also["cfg5_tensor_parallel"] = gemv_tp_sweep(ctx, dev, local, rank, world, 1, 32, 20, 5)
        except Exception as exc:       # noqa: BLE001
            also["cfg5_tensor_parallel"] = {"error": repr(exc)[:300]}

    if rank == 0:
        line = {"metric": METRIC, "value": T * world / (ms_step * 1e-3), "unit": UNIT, "n_gpus": world,
                "steps": args.steps, "warmup": max(args.warmup, 3), "ms_per_step": ms_step,
                "ms_per_step_median": ms_median,
                "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
                "data": "synthetic",
                "config": base_config(args.workload, wl, world),
                "arm": {"precision": "fp32 in/out; tcgen05 fp16 on two scaled fp16 terms per fp32 tensor (24 bits): "
                                     "Y and dX 2 products against exact fp16 ternary digits, dW 3; fp32 accumulate in TMEM; relative L2 <= 1e-5 vs the "
                                     "fp32 reference sums (tested; measured <= 6e-6); counter update bit-exact",
                        "grouped_call": not args.no_group, "lanes": 1 if not args.no_group else args.lanes,
                        "recorded_batch": not args.eager,
                        "collectives": ("reduce-scatter under the row products, update + all-gather under the next "
                                        "step's weight gradients (communication stream)") if world > 1 else None},
                "gpu_launches": launches, "clocks": clocks, "roofline": roofline,
                "e2e": {"value": T * world / (ms_e2e * 1e-3), "unit": UNIT, "ms_per_step": ms_e2e,
                        "h2d_bytes_per_step": in_bytes, "d2h_bytes_per_step": out_bytes},
                "cpu_baseline": cpu, "also": also}
        if dp_parity is not None:
            line["dp_parity"] = dp_parity
        print(json.dumps(line))
    if world > 1:
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
