#!/usr/bin/env python
"""Benchmark of the ragged-dot hot path on B200.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
                    [--only fwd|dlhs|drhs] [--no-e2e] [--no-cpu-baseline]

One JSON line on stdout (rank 0).  N = 1: one step is ragged_dot forward + its full backward
(dlhs through the transposed grouped GEMM, drhs through tgmm) on the Mixtral-8x7B-shaped
workload, m=8192, k=4096, n=14336, g=8, bf16 with fp32 accumulation; `value` counts useful
flops, 2*m*k*n per GEMM.  N > 1 (torchrun): the expert-parallel workload -- per GPU 8192
tokens x top-4 routing over 64 experts sharded 64/N per GPU, the rows exchanged over NVLink, the
local ragged_dot, and its backward (dlhs on the owner + the return exchange, drhs per local
expert): forward + backward, the same three GEMMs per row as at N = 1.

`--impl reference` times the CPU oracle (oracle/ragged_dot_oracle.py, the restatement of the
reference semantics; jax is not installed, so jax.lax.ragged_dot on XLA-CPU cannot run) on a
bounded sample of the same workload with all host threads.
"""

from __future__ import annotations

import argparse
import json
import os
import statistics
import sys
import threading
import time

import numpy as np
import torch

ROOT = os.path.dirname(os.path.abspath(__file__))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)



def captured_launches():
    """Per product of the bf16 Mixtral workload, from the profiler captures whose figures are kept in a small JSON file
    beside their summaries: the kernel's name and dram__bytes_read.sum + dram__bytes_write.sum of one launch."""
    path = os.path.join(ROOT, "profiles", "ragged_gemm_mixtral_dram_traffic.json")
    try:
        with open(path) as f:
            d = json.load(f)
        return {k: (v["kernel"], float(v["dram_read_bytes"]) + float(v["dram_write_bytes"]))
                for k, v in d["kernels"].items()}
    except Exception:
        return {}


METRIC = "ragged_dot fwd+bwd TFLOP/s (2*m*k*n useful flops per GEMM)"
UNIT = "TFLOP/s"


# ---------------------------------------------------------------------------- helpers
def measured_peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(path):
        with open(path) as f:
            p = json.load(f)
        return {
            "bf16_tflops": float(p["bf16_tflops"]),
            "bf16_tflops_sustained": float(p.get("bf16_tflops_sustained", p["bf16_tflops"])),
            "hbm_gbs": float(p["hbm_gbs"]),
            "source": "measured",
        }
    return {"bf16_tflops": 1590.0, "bf16_tflops_sustained": 1400.0, "hbm_gbs": 6650.0, "source": "fallback"}


class ClockSampler:
    """Samples SM clock and throttle reasons through NVML while the timed region runs."""

    def __init__(self, index: int, period_s: float = 0.004):
        self.index = index
        self.period = period_s
        self.samples = []
        self.power_w = []
        self.power_limit_w = None
        self.reasons = set()
        self.max_mhz = None
        self._stop = threading.Event()
        self._thread = None
        self._nvml = None

    def start(self):
        try:
            import pynvml

            pynvml.nvmlInit()
            self._nvml = pynvml
            self._h = pynvml.nvmlDeviceGetHandleByIndex(self.index)
            self.max_mhz = pynvml.nvmlDeviceGetMaxClockInfo(self._h, pynvml.NVML_CLOCK_SM)
            try:
                self.power_limit_w = pynvml.nvmlDeviceGetEnforcedPowerLimit(self._h) / 1000.0
            except Exception:
                self.power_limit_w = None
        except Exception:
            self._nvml = None
            return self
        self._thread = threading.Thread(target=self._run, daemon=True)
        self._thread.start()
        return self

    def _run(self):
        nv = self._nvml
        names = {
            "hw_slowdown": getattr(nv, "nvmlClocksThrottleReasonHwSlowdown", 0x8),
            "hw_thermal_slowdown": getattr(nv, "nvmlClocksThrottleReasonHwThermalSlowdown", 0x40),
            "sw_thermal_slowdown": getattr(nv, "nvmlClocksThrottleReasonSwThermalSlowdown", 0x20),
            "sw_power_cap": getattr(nv, "nvmlClocksThrottleReasonSwPowerCap", 0x4),
            "hw_power_brake": getattr(nv, "nvmlClocksThrottleReasonHwPowerBrakeSlowdown", 0x80),
        }
        while not self._stop.is_set():
            try:
                self.samples.append(nv.nvmlDeviceGetClockInfo(self._h, nv.NVML_CLOCK_SM))
                mask = nv.nvmlDeviceGetCurrentClocksThrottleReasons(self._h)
                for k, bit in names.items():
                    if mask & bit:
                        self.reasons.add(k)
                self.power_w.append(nv.nvmlDeviceGetPowerUsage(self._h) / 1000.0)
            except Exception:
                pass
            time.sleep(self.period)

    def stop(self):
        self._stop.set()
        if self._thread is not None:
            self._thread.join(timeout=1.0)
        return {
            "sm_mhz": statistics.median(self.samples) if self.samples else None,
            "sm_max_mhz": self.max_mhz,
            "reasons": sorted(self.reasons),
            "samples": len(self.samples),
            # board power beside the clock: these kernels pull the board to its power limit within
            # milliseconds, and the clock drops with it before NVML's reason bits show the cap
            "power_w": statistics.median(self.power_w) if self.power_w else None,
            "power_max_w": max(self.power_w) if self.power_w else None,
            "power_limit_w": self.power_limit_w,
        }


def physical_gpu_index(local_index: int) -> int:
    vis = os.environ.get("CUDA_VISIBLE_DEVICES")
    if vis:
        try:
            return int(vis.split(",")[local_index])
        except Exception:
            return local_index
    return local_index


def bind_to_gpu_numa_node(local_index: int) -> str:
    """Pins this process to the CPUs NVML reports as local to its GPU, so that the pinned host
    buffers it allocates afterwards (first touch) and the threads that drive the copies sit on the
    GPU's own NUMA node.  What a deployment does with numactl; returns a note for the JSON line."""
    try:
        import pynvml

        pynvml.nvmlInit()
        h = pynvml.nvmlDeviceGetHandleByIndex(physical_gpu_index(local_index))
        ncpu = os.cpu_count() or 1
        words = pynvml.nvmlDeviceGetCpuAffinity(h, (ncpu + 63) // 64)
        local = {64 * w + b for w, word in enumerate(words) for b in range(64) if (int(word) >> b) & 1}
        allowed = os.sched_getaffinity(0)
        cpus = local & allowed
        if not cpus:
            return "not bound: the GPU's local CPUs are outside this process's CPU set"
        if cpus == allowed:
            return f"all {len(allowed)} CPUs of this process are local to the GPU"
        os.sched_setaffinity(0, cpus)
        return f"bound to the {len(cpus)} CPUs local to the GPU (of {len(allowed)})"
    except Exception as e:  # no NVML, no permission: run unbound
        return f"not bound ({type(e).__name__})"


def dist_env():
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return rank, world, local


# ---------------------------------------------------------------------------- reference arm (CPU)
def mixtral_config(shape, only, rows_per_step):
    """`config` of the N = 1 line, identical for both arms when both run the whole workload."""
    return {
        "workload": shape.name + ("_fwd_bwd" if only is None else "_" + only),
        "m": shape.m, "k": shape.k, "n": shape.n, "g": shape.g,
        "group_sizes": "fwd: multinomial(Dirichlet(2)); bwd: same, each group at a random offset mod 128",
        "rows_per_step": rows_per_step,
        "l2": "inputs larger than L2 (weights %d MB per GEMM)" % (shape.g * shape.k * shape.n * 2 // 1000000),
    }


def cpu_oracle_sample(shape, rows, threads, seed=0):
    """Inputs for a CPU run on the first `rows` rows of the workload: the forward's and the
    backward's group sizes of our arm, scaled when rows < m."""
    from gpu_ragged_dot_b200 import workloads

    def scaled(gs_full):
        gs = (gs_full.astype(np.int64) * rows) // shape.m
        gs[-1] += rows - gs.sum()
        return torch.from_numpy(gs.astype(np.int32))

    gs_fwd, gs_bwd = scaled(workloads.group_sizes_mixtral(seed)), scaled(workloads.group_sizes_mixtral_ragged(seed))
    x = workloads.normal_tensor((rows, shape.k), 1.0, 11, "cpu")
    A = workloads.normal_tensor((shape.g, shape.k, shape.n), shape.k ** -0.5, 12, "cpu")
    dout = workloads.normal_tensor((rows, shape.n), 1.0, 13, "cpu")
    return x, A, dout, (gs_fwd, gs_bwd)


def cpu_oracle_step(x, A, dout, gs, only=None):
    from oracle import ragged_dot_oracle as oracle

    gs_fwd, gs_bwd = gs if isinstance(gs, tuple) else (gs, gs)
    if only in (None, "fwd"):
        oracle.ragged_dot(x, A, gs_fwd, native_16bit=True)
    if only in (None, "dlhs"):
        oracle.ragged_dot(dout, A, gs_bwd, trans_rhs=True, native_16bit=True)
    if only in (None, "drhs"):
        oracle.trans_ragged_dot(x, dout, gs_bwd, native_16bit=True)


def run_reference(args):
    from gpu_ragged_dot_b200 import workloads

    rank, world, _ = dist_env()
    if rank != 0:
        return
    # All the host threads this process may use (torchrun presets OMP_NUM_THREADS=1 for its ranks).
    threads = len(os.sched_getaffinity(0)) if hasattr(os, "sched_getaffinity") else (os.cpu_count() or 1)
    torch.set_num_threads(threads)
    if max(world, args.gpus) > 1:
        return run_reference_expert_parallel(args, max(world, args.gpus), threads)
    shape = workloads.MIXTRAL
    gemms = 3 if args.only is None else 1
    # The whole workload (all 8192 rows) per step whenever warm-up + steps fit about two and a half
    # minutes; otherwise the largest multiple of 128 rows that does.  The probe runs twice: the
    # first call pays for oneDNN's set-up and the first touch of 940 MB of weights.
    x, A, dout, gs = cpu_oracle_sample(shape, 1024, threads)
    cpu_oracle_step(x, A, dout, gs, args.only)
    t0 = time.perf_counter()
    cpu_oracle_step(x, A, dout, gs, args.only)
    t_probe = time.perf_counter() - t0
    budget = 150.0 / max(args.steps + args.warmup, 1)
    rows = int(min(shape.m, max(128, 1024 * budget / max(t_probe, 1e-3))))
    rows = shape.m if rows >= shape.m else max(128, (rows // 128) * 128)
    x, A, dout, gs = cpu_oracle_sample(shape, rows, threads)
    for _ in range(args.warmup):
        cpu_oracle_step(x, A, dout, gs, args.only)
    t0 = time.perf_counter()
    for _ in range(args.steps):
        cpu_oracle_step(x, A, dout, gs, args.only)
    dt = (time.perf_counter() - t0) / max(args.steps, 1)
    flops = 2.0 * rows * shape.k * shape.n * gemms
    value = flops / dt / 1e12
    sample = (("the whole workload: " if rows == shape.m else "") +
              f"rows 0..{rows - 1} of {shape.m} (group sizes {'as in our arm' if rows == shape.m else 'scaled'}), all {shape.g} experts' weights, "
              f"{'fwd+dlhs+drhs' if args.only is None else args.only} per step; torch CPU bf16 matmul (oneDNN, fp32 accumulate) per group")
    line = {
        "impl": "reference",
        "metric": METRIC,
        "value": value,
        "unit": UNIT,
        "n_gpus": args.gpus,
        "steps": args.steps,
        "warmup": args.warmup,
        "ms_per_step": dt * 1e3,
        "higher_is_better": True,
        "scaling": "weak",
        "vs_baseline": None,
        "dtype": "bf16",
        "data": "synthetic",
        "config": mixtral_config(shape, args.only, rows),
        "method": "CPU restatement of jax.lax.ragged_dot semantics (jax not installed); wall clock around the steps",
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": threads, "kind": "port", "sample": sample,
                         "host_cpus": os.cpu_count()},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "gpu_launches": 0,
    }
    print(json.dumps(line), flush=True)


def ep_config(shape, world, tokens, top_k, experts, tokens_per_step):
    """`config` of the N > 1 line, identical for both arms when the CPU arm runs every token."""
    return {"workload": f"expert_parallel_fwd_bwd_{shape.name}_w{world}", "tokens_per_gpu": tokens,
            "top_k": top_k, "experts": experts, "experts_per_gpu": experts // world, "k": shape.k, "n": shape.n,
            "tokens_per_step": tokens_per_step,
            "l2": "inputs larger than L2 (268 MB of rows per GPU)"}


def run_reference_expert_parallel(args, world, threads):
    """Reference arm of the N > 1 workload (expert-parallel forward + backward): the same routing,
    permutation by expert, ragged_dot over all 64 experts, and its VJP as the reference wires it
    (dlhs through the transposed product, summed over a token's copies; drhs through tgmm), on
    the host cores of rank 0.  There is no exchange on one host.  A step covers every token of the
    job when warm-up + steps fit about two and a half minutes, else a bounded sample of them."""
    from gpu_ragged_dot_b200 import workloads
    from oracle import ragged_dot_oracle as oracle

    shape = workloads.EP_PREFILL
    tokens_gpu, top_k, experts = 8192, 4, shape.g
    tokens_job = tokens_gpu * world
    A = workloads.normal_tensor((experts, shape.k, shape.n), shape.k ** -0.5, 12, "cpu")

    def make(tokens):
        x = workloads.normal_tensor((tokens, shape.k), 1.0, 11, "cpu")
        routing = torch.from_numpy(workloads.topk_routing(tokens, experts, top_k, seed=3000)).to(torch.int64)
        dy = workloads.normal_tensor((tokens * top_k, shape.n), 1.0, 13, "cpu")
        return x, routing, dy

    def step(x, routing, dy):
        flat = routing.reshape(-1)
        order = torch.argsort(flat, stable=True)
        gs = torch.bincount(flat, minlength=experts).to(torch.int32)
        token_of_row = order // top_k
        rows = x.index_select(0, token_of_row)
        y = oracle.ragged_dot(rows, A, gs, native_16bit=True)
        d_rows = oracle.ragged_dot(dy, A, gs, trans_rhs=True, native_16bit=True)
        dx = torch.zeros((x.shape[0], shape.k), dtype=torch.float32).index_add_(0, token_of_row, d_rows.float())
        dA = oracle.trans_ragged_dot(rows, dy, gs, native_16bit=True)
        return y, dx.to(torch.bfloat16), dA

    probe = make(2048)
    step(*probe)
    t0 = time.perf_counter()
    step(*probe)
    t_probe = time.perf_counter() - t0
    budget = 150.0 / max(args.steps + args.warmup, 1)
    tokens = int(min(tokens_job, max(256, 2048 * budget / max(t_probe, 1e-3))))
    tokens = tokens_job if tokens >= tokens_job else max(256, (tokens // 256) * 256)
    data = make(tokens)
    for _ in range(args.warmup):
        step(*data)
    t0 = time.perf_counter()
    for _ in range(args.steps):
        step(*data)
    dt = (time.perf_counter() - t0) / max(args.steps, 1)
    value = 3 * 2.0 * tokens * top_k * shape.k * shape.n / dt / 1e12
    sample = (("every token of the job: " if tokens == tokens_job else "") +
              f"{tokens} of the job's {tokens_job} tokens x top-{top_k} per step: sort by expert, gather rows, "
              f"ragged_dot over all {experts} experts' weights, dlhs + top-k combine, drhs; torch CPU bf16 matmul "
              "(oneDNN, fp32 accumulate) per group")
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": dt * 1e3, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "bf16", "data": "synthetic",
        "config": ep_config(shape, world, tokens_gpu, top_k, experts, tokens),
        "method": "CPU restatement of jax.lax.ragged_dot semantics (jax not installed), one host; wall clock",
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": threads, "kind": "port", "sample": sample,
                         "host_cpus": os.cpu_count()},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "gpu_launches": 0,
    }
    print(json.dumps(line), flush=True)


# ---------------------------------------------------------------------------- our arm, N = 1
def run_single(args):
    from gpu_ragged_dot_b200 import _lib, ops, workloads
    import gpu_ragged_dot_b200 as rd

    _lib.load()  # fail loudly if the CUDA library is missing
    dev = torch.device("cuda", 0)
    torch.cuda.set_device(dev)
    shape = {"mixtral": workloads.MIXTRAL, "decode": workloads.EP_DECODE,
             "deepseek": workloads.DEEPSEEK_V3, "deepseek_quarter": workloads.DEEPSEEK_QUARTER}[args.workload]
    fp8 = args.dtype == "e4m3"
    if fp8 and args.only != "fwd":
        raise SystemExit("bench.py: --dtype e4m3 exists for the forward product only (--only fwd)")
    dt = {"bf16": torch.bfloat16, "f32": torch.float32, "e4m3": torch.bfloat16}[args.dtype]
    peaks = measured_peaks()
    kernels = ["fwd", "dlhs", "drhs"] if args.only is None else [args.only]
    # Allocate only what the selected kernels touch (keeps profiler captures small).
    x, A, dout = workloads.make_inputs(shape, dev, seed=0, dtype=dt, with_dout=kernels != ["fwd"])
    if kernels == ["dlhs"]:
        x = None
    if kernels == ["drhs"]:
        A = None
    if args.workload == "mixtral":
        gs_fwd_np, gs_bwd_np = workloads.group_sizes_mixtral(0), workloads.group_sizes_mixtral_ragged(0)
    elif args.workload == "decode":
        gs_fwd_np = gs_bwd_np = workloads.group_sizes_from_routing(workloads.topk_routing(64, 64, 4, seed=5), 64)
    elif args.workload == "deepseek_quarter":
        gs_fwd_np = gs_bwd_np = workloads.group_sizes_deepseek_quarter(0)
    else:
        gs_fwd_np = gs_bwd_np = workloads.group_sizes_deepseek(0)
    gs_fwd = torch.from_numpy(gs_fwd_np).to(dev)
    gs_bwd = torch.from_numpy(gs_bwd_np).to(dev)
    y = torch.empty((shape.m, shape.n), dtype=dt, device=dev) if "fwd" in kernels else None
    dx = torch.empty((shape.m, shape.k), dtype=dt, device=dev) if "dlhs" in kernels else None
    dA = torch.empty((shape.g, shape.k, shape.n), dtype=dt, device=dev) if "drhs" in kernels else None
    esz = 2 if dt == torch.bfloat16 else 4
    ws = ops._workspace(shape.m, shape.g, dev)
    if fp8:  # e4m3 operands, weights stored [g, n, k]; the result stays bf16
        x = x.to(torch.float8_e4m3fn)
        A = A.transpose(1, 2).contiguous().to(torch.float8_e4m3fn)

    def launch(name):
        if name == "fwd" and fp8:
            ops.gmm_fp8_forward(x, A, gs_fwd, out=y, workspace=ws)
        elif name == "fwd":
            ops.gmm_forward(x, A, gs_fwd, out=y, workspace=ws)
        elif name == "dlhs":
            ops.gmm_forward(dout, A, gs_bwd, trans_rhs=True, out=dx, workspace=ws)
        else:
            ops.tgmm_forward(x, dout, gs_bwd, out=dA, workspace=ws)

    for _ in range(max(args.warmup, 3)):
        for name in kernels:
            launch(name)
    torch.cuda.synchronize()

    stream = torch.cuda.current_stream(dev)
    marks = [[torch.cuda.Event(enable_timing=True) for _ in range(len(kernels) + 1)] for _ in range(args.steps)]
    sampler = ClockSampler(physical_gpu_index(0)).start()
    torch.cuda.synchronize()
    for s in range(args.steps):
        marks[s][0].record(stream)
        for i, name in enumerate(kernels):
            launch(name)
            marks[s][i + 1].record(stream)
    torch.cuda.synchronize()
    clocks = sampler.stop()
    status = ops.device_status(ws)
    if status != 0:
        raise RuntimeError(f"device status {status} after the timed region")

    total_ms = marks[0][0].elapsed_time(marks[-1][-1])
    ms_per_step = total_ms / args.steps
    per_kernel_ms = {
        name: sum(marks[s][i].elapsed_time(marks[s][i + 1]) for s in range(args.steps)) / args.steps
        for i, name in enumerate(kernels)
    }
    gemm_flops = 2.0 * shape.m * shape.k * shape.n
    value = gemm_flops * len(kernels) / (ms_per_step * 1e-3) / 1e12

    # roofline of the dominant (slowest) kernel; every GEMM here is tensor-bound (AI ~ 775 flop/B)
    dom = max(per_kernel_ms, key=per_kernel_ms.get)
    per_kernel = {}
    for name, ms in per_kernel_ms.items():
        tf = gemm_flops / (ms * 1e-3) / 1e12
        per_kernel[name] = {"ms": ms, "tflops": tf, "frac_of_measured_burst": tf / peaks["bf16_tflops"],
                            "frac_of_measured_sustained": tf / peaks["bf16_tflops_sustained"]}
    captured = captured_launches() if args.workload == "mixtral" and args.dtype == "bf16" else {}
    kernel, traffic = captured.get(dom, ({"fwd": "gmm", "dlhs": "gmm, trans_rhs", "drhs": "tgmm"}[dom]
                                         + ": the kernel that the rules of rd_api.cu pick", None))
    gplus_f, gplus_b = int((gs_fwd_np > 0).sum()), int((gs_bwd_np > 0).sum())
    alg_bytes = {
        "fwd": (1.0 * (shape.m * shape.k + gplus_f * shape.k * shape.n) + 2.0 * shape.m * shape.n) if fp8 else
               esz * 1.0 * (shape.m * shape.k + gplus_f * shape.k * shape.n + shape.m * shape.n),
        "dlhs": esz * 1.0 * (shape.m * shape.n + gplus_b * shape.k * shape.n + shape.m * shape.k),
        "drhs": esz * 1.0 * (shape.m * shape.k + shape.m * shape.n + shape.g * shape.k * shape.n),
    }
    for name, ms in per_kernel_ms.items():
        gbs = alg_bytes[name] / (ms * 1e-3) / 1e9
        per_kernel[name]["algorithmic_GBps"] = gbs
        per_kernel[name]["frac_of_measured_hbm"] = gbs / peaks["hbm_gbs"]
    hbm_bound = alg_bytes[dom] / (peaks["hbm_gbs"] * 1e9) > gemm_flops / (peaks["bf16_tflops"] * 1e12)
    if hbm_bound:
        roofline = {
            "bound": "hbm",
            "kernel": kernel,
            "achieved": per_kernel[dom]["algorithmic_GBps"], "peak": peaks["hbm_gbs"],
            "peak_source": f"{peaks['source']} (copy bandwidth)", "unit": "GB/s",
            "frac": per_kernel[dom]["frac_of_measured_hbm"], "traffic": None,
            "algorithmic_bytes_per_launch": alg_bytes[dom], "algorithmic_flops_per_launch": gemm_flops,
            "per_kernel": per_kernel,
        }
    else:
        roofline = {
            "bound": "tensor",
            "kernel": kernel,
            "achieved": per_kernel[dom]["tflops"],
            "peak": peaks["bf16_tflops"],
            "peak_source": f"{peaks['source']} (burst cuBLAS bf16); sustained {peaks['bf16_tflops_sustained']}",
            "unit": "TFLOP/s",
            "frac": per_kernel[dom]["tflops"] / peaks["bf16_tflops"],
            "frac_of_sustained": per_kernel[dom]["tflops"] / peaks["bf16_tflops_sustained"],
            "traffic": traffic,
            "algorithmic_flops_per_launch": gemm_flops,
            "algorithmic_bytes_per_launch": alg_bytes[dom],
            "per_kernel": per_kernel,
        }

    line = {
        "metric": METRIC,
        "value": value,
        "unit": UNIT,
        "n_gpus": 1,
        "steps": args.steps,
        "warmup": max(args.warmup, 3),
        "ms_per_step": ms_per_step,
        "higher_is_better": True,
        "scaling": "weak",
        "vs_baseline": None,
        "dtype": {"bf16": "bf16", "f32": "f32 in/out, TF32 products, fp32 accumulate (the bf16 peak is NOT its roof)",
                  "e4m3": "e4m3 in, fp32 accumulate, bf16 out (the bf16 peak is NOT its roof)"}[args.dtype],
        "data": "synthetic",
        "config": (mixtral_config(shape, args.only, shape.m) if args.workload == "mixtral" else {
            "workload": shape.name + ("_fwd_bwd" if args.only is None else "_" + args.only),
            "m": shape.m, "k": shape.k, "n": shape.n, "g": shape.g,
            "group_sizes": {"decode": "64 tokens x uniform top-4 of 64 experts",
                            "deepseek": "multinomial(Dirichlet(0.3)), ~20% empty",
                            "deepseek_quarter": "multinomial(Dirichlet(0.3)) over 64 experts"}[args.workload],
            "l2": "inputs larger than L2 (weights %d MB per GEMM)" % (shape.g * shape.k * shape.n * 2 // 1000000),
        }),
        "method": "CUDA events on the launch stream; per-kernel events inside the timed region",
        "clocks": clocks,
        # one launch per GEMM; above 256 groups the group metadata is a launch of its own
        "gpu_launches": (1 if shape.g <= 256 else 2) * len(kernels) * args.steps,
        "roofline": roofline,
    }

    if not args.no_e2e and args.only is None and args.workload == "mixtral":
        line["e2e"] = run_e2e(args, shape, dev, rd, x, A, dout, gs_fwd, kernels)
    if args.only is None and not args.no_other_workloads and args.workload == "mixtral":
        del x, A, dout, y, dx, dA
        torch.cuda.empty_cache()
        line["other_workloads"] = run_other_workloads(dev, peaks)
    if not args.no_cpu_baseline and args.workload == "mixtral":
        line["cpu_baseline"] = run_cpu_baseline(shape, kernels)
    print(json.dumps(line), flush=True)


def run_permute(args):
    """`--workload permute`: the MoE-layer use of the path on the Mixtral shape (4096 tokens, top-2
    routing over 8 experts -> 8192 sorted rows): y[out_rows[r]] = x[in_rows[r]] @ A[expert of r].
    Times the permutation-fused kernels (rd_gmm_permuted / rd_tgmm_permuted) against
    rd_gather_rows + rd_gmm / rd_tgmm + rd_gather_rows, variants interleaved in one process."""
    import random
    import statistics

    from gpu_ragged_dot_b200 import _lib, ops, workloads

    _lib.load()
    dev = torch.device("cuda", 0)
    torch.cuda.set_device(dev)
    shape = workloads.MIXTRAL
    top_k = 2
    tokens = shape.m // top_k
    routing = workloads.topk_routing(tokens, shape.g, top_k, seed=0)  # [tokens, top_k]
    flat = routing.reshape(-1)
    order = np.argsort(flat, kind="stable")
    gs = torch.from_numpy(np.bincount(flat, minlength=shape.g).astype(np.int32)).to(dev)
    in_rows = torch.from_numpy((order // top_k).astype(np.int32)).to(dev)
    out_rows = torch.from_numpy(order.astype(np.int32)).to(dev)
    inv_rows = torch.empty_like(out_rows)
    inv_rows[out_rows.long()] = torch.arange(shape.m, dtype=torch.int32, device=dev)
    x = workloads.normal_tensor((tokens, shape.k), 1.0, 1, dev)
    A = workloads.normal_tensor((shape.g, shape.k, shape.n), shape.k ** -0.5, 2, dev)
    dy = workloads.normal_tensor((shape.m, shape.n), 1.0, 3, dev)
    ws = ops._workspace(shape.m, shape.g, dev)
    xs = torch.empty((shape.m, shape.k), dtype=torch.bfloat16, device=dev)
    ys = torch.empty((shape.m, shape.n), dtype=torch.bfloat16, device=dev)
    y = torch.empty((shape.m, shape.n), dtype=torch.bfloat16, device=dev)
    dys = torch.empty((shape.m, shape.n), dtype=torch.bfloat16, device=dev)
    dA = torch.empty_like(A)

    def fwd_fused():
        ops.gmm_permuted_forward(x, A, gs, in_rows=in_rows, out_rows=out_rows, out=y, y_rows=shape.m, workspace=ws)

    def fwd_fused_gather_only():
        ops.gmm_permuted_forward(x, A, gs, in_rows=in_rows, out=ys, workspace=ws)

    def fwd_two_pass():
        ops.gather_rows(x, in_rows, out=xs)
        ops.gmm_forward(xs, A, gs, out=ys, workspace=ws)
        ops.gather_rows(ys, inv_rows, out=y)

    def fwd_two_pass_gather_only():
        ops.gather_rows(x, in_rows, out=xs)
        ops.gmm_forward(xs, A, gs, out=ys, workspace=ws)

    def drhs_fused():
        ops.tgmm_permuted_forward(x, dy, gs, x_rows_index=in_rows, y_rows_index=out_rows, out=dA, workspace=ws)

    def drhs_two_pass():
        ops.gather_rows(x, in_rows, out=xs)
        ops.gather_rows(dy, out_rows, out=dys)
        ops.tgmm_forward(xs, dys, gs, out=dA, workspace=ws)

    variants = {"fwd_fused": fwd_fused, "fwd_two_pass": fwd_two_pass,
                "fwd_fused_gather_only": fwd_fused_gather_only,
                "fwd_two_pass_gather_only": fwd_two_pass_gather_only,
                "drhs_fused": drhs_fused, "drhs_two_pass": drhs_two_pass}
    for fn in variants.values():
        for _ in range(max(args.warmup, 3)):
            fn()
    torch.cuda.synchronize()
    sampler = ClockSampler(physical_gpu_index(0))
    sampler.start()
    times = {name: [] for name in variants}
    rng = random.Random(0)
    for _ in range(5):
        names = list(variants)
        rng.shuffle(names)
        for name in names:
            times[name].append(_time_ms(variants[name], args.steps))
    clocks = sampler.stop()
    assert ops.device_status(ws) == 0, "device reported an expired wait"
    flops = 2.0 * shape.m * shape.k * shape.n
    res = {name: {"ms": round(statistics.median(v), 4),
                  "tflops": round(flops / statistics.median(v) / 1e9, 1)} for name, v in times.items()}
    ms = res["fwd_fused"]["ms"]
    print(json.dumps({
        "metric": "ragged_dot_permuted_fwd_tflops", "value": res["fwd_fused"]["tflops"], "unit": UNIT,
        "n_gpus": 1, "steps": args.steps, "warmup": max(args.warmup, 3), "ms_per_step": ms,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "bf16", "data": "synthetic",
        "config": {"workload": "permute: mixtral shape, 4096 tokens x top-2 of 8 experts, gather + scatter "
                               "fused into the GEMM", "m": shape.m, "k": shape.k, "n": shape.n, "g": shape.g,
                   "l2": "operands larger than L2"},
        "variants": res, "clocks": clocks, "gpu_launches": 2 * args.steps,
    }), flush=True)


def _time_ms(fn, reps):
    for _ in range(3):
        fn()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(reps):
        fn()
    e1.record()
    torch.cuda.synchronize()
    return e0.elapsed_time(e1) / reps


def run_other_workloads(dev, peaks):
    """Short device-resident measurements of the bandwidth-bound configurations (not part of the
    headline `value`): the decode shape (m=256 over 64 experts) and the DeepSeek-V3 shape."""
    from gpu_ragged_dot_b200 import ops, workloads

    out = {}
    hbm = peaks["hbm_gbs"]

    def entry(ms, flops, nbytes):
        gbs = nbytes / (ms * 1e-3) / 1e9
        return {"ms": ms, "tflops": flops / (ms * 1e-3) / 1e12, "algorithmic_GBps": gbs,
                "frac_of_measured_hbm": gbs / hbm}

    # decode: 64 tokens x top-4 over 64 experts -> m = 256, weights 805 MB (larger than L2)
    s = workloads.EP_DECODE
    gs_np = workloads.group_sizes_from_routing(workloads.topk_routing(64, 64, 4, seed=5), 64)
    gplus = int((gs_np > 0).sum())
    x, A, _ = workloads.make_inputs(s, dev, with_dout=False)
    gs = torch.from_numpy(gs_np).to(dev)
    ws = ops._workspace(s.m, s.g, dev)
    y = torch.empty((s.m, s.n), dtype=torch.bfloat16, device=dev)
    ms = _time_ms(lambda: ops.gmm_forward(x, A, gs, out=y, workspace=ws), 30)
    out[s.name + "_fwd"] = entry(ms, 2.0 * s.m * s.k * s.n, 2.0 * (s.m * s.k + gplus * s.k * s.n + s.m * s.n))
    out[s.name + "_fwd"]["nonempty_groups"] = gplus
    # the same product with e4m3 operands (rd_gmm_fp8; weights stored [g, n, k]): half the weight bytes
    f8 = torch.float8_e4m3fn
    x8, A8 = x.to(f8), A.transpose(1, 2).contiguous().to(f8)
    ms8 = _time_ms(lambda: ops.gmm_fp8_forward(x8, A8, gs, out=y, workspace=ws), 30)
    out[s.name + "_fwd_e4m3"] = entry(ms8, 2.0 * s.m * s.k * s.n, 1.0 * (s.m * s.k + gplus * s.k * s.n) + 2.0 * s.m * s.n)
    del x, A, y, x8, A8
    torch.cuda.empty_cache()

    # the headline shape's forward with e4m3 operands (tensor-bound: kind::f8f6f4 has twice the bf16 rate)
    s = workloads.MIXTRAL
    gs_np = workloads.group_sizes_mixtral(0)
    x, A, _ = workloads.make_inputs(s, dev, with_dout=False)
    x8, A8 = x.to(f8), A.transpose(1, 2).contiguous().to(f8)
    del x, A
    gs = torch.from_numpy(gs_np).to(dev)
    ws = ops._workspace(s.m, s.g, dev)
    y = torch.empty((s.m, s.n), dtype=torch.bfloat16, device=dev)
    ms8 = _time_ms(lambda: ops.gmm_fp8_forward(x8, A8, gs, out=y, workspace=ws), 20)
    out[s.name + "_fwd_e4m3"] = entry(ms8, 2.0 * s.m * s.k * s.n, 1.0 * (s.m * s.k + s.g * s.k * s.n) + 2.0 * s.m * s.n)
    out[s.name + "_fwd_e4m3"]["note"] = "tensor-bound; no measured 8-bit peak on this pool (nominal dense 4500 TFLOP/s)"
    del y, x8, A8
    torch.cuda.empty_cache()

    # DeepSeek-V3 shaped: heavy-tailed groups, ~20 % empty
    s = workloads.DEEPSEEK_V3
    gs_np = workloads.group_sizes_deepseek(0)
    gplus = int((gs_np > 0).sum())
    x, A, dout = workloads.make_inputs(s, dev)
    gs = torch.from_numpy(gs_np).to(dev)
    ws = ops._workspace(s.m, s.g, dev)
    y = torch.empty((s.m, s.n), dtype=torch.bfloat16, device=dev)
    dx = torch.empty((s.m, s.k), dtype=torch.bfloat16, device=dev)
    dA = torch.empty_like(A)
    fl = 2.0 * s.m * s.k * s.n
    b_gmm = 2.0 * (s.m * s.k + gplus * s.k * s.n + s.m * s.n)
    b_tgmm = 2.0 * (s.m * s.k + s.m * s.n + s.g * s.k * s.n)
    out[s.name + "_fwd"] = entry(_time_ms(lambda: ops.gmm_forward(x, A, gs, out=y, workspace=ws), 8), fl, b_gmm)
    out[s.name + "_dlhs"] = entry(
        _time_ms(lambda: ops.gmm_forward(dout, A, gs, trans_rhs=True, out=dx, workspace=ws), 8), fl, b_gmm)
    out[s.name + "_drhs"] = entry(_time_ms(lambda: ops.tgmm_forward(x, dout, gs, out=dA, workspace=ws), 8), fl, b_tgmm)
    out[s.name + "_fwd"]["nonempty_groups"] = gplus
    # drhs writes 7.5 GB and reads 0.6 GB: it is bound by the WRITE bandwidth, which on these parts
    # is well below the read+write copy figure.  A memset of the same output measured here is its ceiling.
    ms_set = _time_ms(lambda: dA.zero_(), 5)
    out[s.name + "_drhs"]["memset_of_the_output_ms"] = ms_set
    out[s.name + "_drhs"]["write_GBps_of_memset"] = dA.numel() * 2 / (ms_set * 1e-3) / 1e9
    out[s.name + "_drhs"]["time_vs_memset_of_the_output"] = out[s.name + "_drhs"]["ms"] / ms_set
    return out


def run_e2e(args, shape, dev, rd, x, A, dout, gs, kernels):
    """Same step with HOST buffers, everything inside the timed region: pinned H2D of x, A,
    group_sizes and dout, ragged_dot + backward on the device, D2H of y, dlhs and drhs.

    `value` goes through `HostRaggedDot` (the host-buffer entry of the package: expert chunks are
    copied in, multiplied and copied out on three streams, so both directions of the PCIe link and
    the GPU work at once).  `one_stream_ms` is the plain way beside it: `ragged_dot` + autograd
    on device tensors with the copies around it on one stream."""
    full = len(kernels) == 3
    hx, hA, hd = (t.cpu().pin_memory() for t in (x, A, dout))
    hgs = gs.cpu().pin_memory()
    hy = torch.empty((shape.m, shape.n), dtype=torch.bfloat16).pin_memory()
    hdx = torch.empty_like(hx).pin_memory()
    hdA = torch.empty_like(hA).pin_memory()
    steps = max(2, min(args.steps, 5))

    def step_one_stream():
        dx_ = hx.to(dev, non_blocking=True)
        dA_ = hA.to(dev, non_blocking=True)
        dg_ = hgs.to(dev, non_blocking=True)
        if full:
            dd_ = hd.to(dev, non_blocking=True)
            dx_.requires_grad_(True)
            dA_.requires_grad_(True)
        yv = rd.ragged_dot(dx_, dA_, dg_)
        if full:
            yv.backward(dd_)
            hdx.copy_(dx_.grad, non_blocking=True)
            hdA.copy_(dA_.grad, non_blocking=True)
        hy.copy_(yv.detach(), non_blocking=True)

    pipe = rd.HostRaggedDot(shape.m, shape.k, shape.n, shape.g, device=dev, backward=full)

    def step_pipelined():
        if full:
            pipe(hx, hA, hgs, hd, y=hy, dlhs=hdx, drhs=hdA)
        else:
            pipe(hx, hA, hgs, y=hy)

    def timed(step, reps):
        for _ in range(2):
            step()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(reps):
            step()
        e1.record()
        torch.cuda.synchronize()
        return e0.elapsed_time(e1) / reps

    ms_serial = timed(step_one_stream, steps)
    torch.cuda.empty_cache()
    ms = timed(step_pipelined, steps)
    nbytes = lambda t: t.numel() * t.element_size()
    h2d = nbytes(hx) + nbytes(hA) + nbytes(hgs) + (nbytes(hd) if full else 0)
    d2h = nbytes(hy) + ((nbytes(hdx) + nbytes(hdA)) if full else 0)
    flops = 2.0 * shape.m * shape.k * shape.n * (3 if full else 1)
    return {"value": flops / (ms * 1e-3) / 1e12, "unit": UNIT, "ms_per_step": ms, "steps": steps,
            "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
            "h2d_GBps": h2d / (ms * 1e-3) / 1e9, "d2h_GBps": d2h / (ms * 1e-3) / 1e9,
            "api": "gpu_ragged_dot_b200.HostRaggedDot (pinned host buffers; chunks of experts copied in, "
                   "multiplied by rd_gmm/rd_tgmm and copied out on three streams)",
            "one_stream_ms": ms_serial, "one_stream_value": flops / (ms_serial * 1e-3) / 1e12,
            "one_stream_api": "gpu_ragged_dot_b200.ragged_dot + autograd backward, copies on the same stream"}


def run_cpu_baseline(shape, kernels):
    threads = torch.get_num_threads()
    rows = 4096
    x, A, dout, gs = cpu_oracle_sample(shape, rows, threads)
    only = None if len(kernels) == 3 else kernels[0]
    cpu_oracle_step(x[:128], A, dout[:128], torch.tensor([16] * shape.g, dtype=torch.int32), only)  # warm-up
    cpu_oracle_step(x, A, dout, gs, only)
    t0 = time.perf_counter()
    reps = 0
    while reps < 3 and time.perf_counter() - t0 < 20.0:
        cpu_oracle_step(x, A, dout, gs, only)
        reps += 1
    dt = (time.perf_counter() - t0) / reps
    flops = 2.0 * rows * shape.k * shape.n * len(kernels)
    return {"value": flops / dt / 1e12, "unit": UNIT, "cores": threads, "kind": "port",
            "host_cpus": os.cpu_count(),
            "sample": f"rows 0..{rows - 1} of {shape.m} (group sizes scaled 1/{shape.m // rows}), all {shape.g} "
                      f"experts' weights, {'+'.join(kernels)} x{reps}; oracle = torch CPU bf16 matmul (oneDNN, fp32 accumulate) per group"}


# ---------------------------------------------------------------------------- our arm, N > 1
EP_MODES = ("nccl", "p2p", "fused")
EP_COLLECTIVE = {
    "nccl": "NCCL all-to-all (rows, both directions) + all-to-all (counts)",
    "p2p": "NCCL all-gather (counts) + peer stores over NVLink + symmetric-memory barrier; gradient rows pulled "
           "back with peer loads",
    "fused": "NCCL all-gather (counts) + ONE kernel whose sender CTAs store rows to the peers over NVLink (ring "
             "phases) while its other CTAs multiply the rows that have arrived (ready flags); gradient rows pulled "
             "back with peer loads after a symmetric-memory barrier",
}
# our kernels per step (forward + backward), collectives and torch's own kernels not counted
EP_LAUNCHES = {"nccl": 1 + 1 + 1 + 2, "p2p": 4 + 1 + 1 + 2 + 1, "fused": 6 + 1 + 2 + 1}  # fused: count+share,
# plan, assign, own rows, metadata, send+GEMM; dlhs; metadata + drhs; pull


def ep_parity_check(layer, mode, out, dy, dx, dW, routing, world, dev, sample_tokens=48):
    """Outside the timed region: does this rank's result agree with an independent computation?
    Every segment of the receive buffer is copied into an ordinary tensor and multiplied with torch
    in fp32 on this GPU: y and the gradient rows (dlhs) of ALL received rows and the dW of every
    local expert must agree within rtol/atol 2e-2.  The return exchange is checked on the first
    `sample_tokens` tokens: their top_k gradient rows are fetched from the owners' buffers with
    peer memcpys and summed in fp32 in slot order, which dx must equal bit for bit.  Returns a
    dict, all-reduced over the ranks (worst case)."""
    import torch.distributed as dist

    El, W = layer.local_experts, world
    sv = layer._saved
    seg = sv["plan"].segment_sizes if mode == "nccl" else sv["seg"]
    recv, y = sv["recv"], out[0]
    d_rows = None if mode == "nccl" else layer._grad["buf"]
    offs = np.concatenate([[0], np.cumsum(seg.cpu().tolist())])
    ratio = lambda got, want: float(((got.float() - want).abs() / (2e-2 + 2e-2 * want.abs())).max()) if want.numel() else 0.0
    worst = [0.0, 0.0, 0.0, 0.0]  # y, dlhs, dW, dx mismatches
    for j in range(El):
        wj = layer.weights[j].float()
        want_dW = torch.zeros((layer.k, layer.n), dtype=torch.float32, device=dev)
        for q in range(W):
            lo, hi = int(offs[q * El + j]), int(offs[q * El + j + 1])
            rows = recv[lo:hi].clone().float()
            g_rows = dy[lo:hi].float()
            want_dW += rows.T @ g_rows
            worst[0] = max(worst[0], ratio(y[lo:hi], (rows @ wj).to(torch.bfloat16).float()))
            if d_rows is not None:
                worst[1] = max(worst[1], ratio(d_rows[lo:hi], (g_rows @ wj.T).to(torch.bfloat16).float()))
        worst[2] = max(worst[2], ratio(dW[j], want_dW.to(torch.bfloat16).float()))
    dx_checked = 0
    if mode != "nccl":
        hdl, cap = layer._grad["hdl"], layer._grad["capacity"]
        peers = [layer._grad["buf"] if (hdl is None or r == layer.rank) else
                 hdl.get_buffer(r, (cap, layer.k), layer.dtype) for r in range(W)]
        r_cpu = sv["routing"].cpu()
        p_cpu = sv["dest_pos"].reshape(r_cpu.shape).cpu()
        top_k = r_cpu.shape[1]
        for t in range(min(sample_tokens, r_cpu.shape[0])):
            acc = torch.zeros(layer.k, dtype=torch.float32, device=dev)
            for s_ in range(top_k):
                e, pos = int(r_cpu[t, s_]), int(p_cpu[t, s_])
                row = torch.empty((1, layer.k), dtype=layer.dtype, device=dev)
                row.copy_(peers[e // El][pos:pos + 1])  # a peer-to-peer memcpy of one row
                acc += row[0].float()
            worst[3] += float(not torch.equal(acc.to(layer.dtype).view(torch.int16), dx[t].view(torch.int16)))
            dx_checked += 1
    w = torch.tensor(worst, dtype=torch.float64, device=dev)
    dist.all_reduce(w, op=dist.ReduceOp.MAX)
    res = {"y_worst_ratio": float(w[0]), "dlhs_worst_ratio": float(w[1]) if d_rows is not None else None,
           "dW_worst_ratio": float(w[2]), "dx_tokens_checked_per_rank": dx_checked,
           "dx_mismatching_tokens": int(w[3]) if dx_checked else None,
           "tolerance": "|a-b| <= 2e-2 + 2e-2|b| against torch fp32 on the same GPU; dx bit-exact on the sample"}
    res["ok"] = bool(float(w[0]) <= 1.0 and float(w[1]) <= 1.0 and float(w[2]) <= 1.0 and float(w[3]) == 0.0)
    return res


def run_expert_parallel(args):
    """N > 1: expert-parallel forward + backward.  Three dispatch modes are timed on the same
    inputs: "nccl" (sort + gather + NCCL all-to-all with host-known split sizes; the baseline),
    "p2p" (device-side plan + rows stored straight into the owners' receive buffers through peer
    memory, no host round trip) and "fused" (the exchange inside the GEMM launch).  `value` is the
    fastest; all are reported, each with a parity check made outside the timed region."""
    import torch.distributed as dist
    from gpu_ragged_dot_b200 import _lib, ep, ops, workloads

    _lib.load()
    rank, world, local = dist_env()
    numa_note = bind_to_gpu_numa_node(local)
    dev = torch.device("cuda", local)
    torch.cuda.set_device(dev)
    dist.init_process_group("nccl", device_id=dev)
    shape = workloads.EP_PREFILL
    tokens, top_k, experts = 8192, 4, shape.g
    x_tokens = workloads.normal_tensor((tokens, shape.k), 1.0, 1000 + rank, dev)
    routing = torch.from_numpy(workloads.topk_routing(tokens, experts, top_k, seed=3000 + rank)).to(dev)
    peaks = measured_peaks()
    results, parity, local_only = {}, {}, None
    clocks = None
    warm = max(args.warmup, 3)
    for mode in EP_MODES:
        try:
            layer = ep.ExpertParallelRaggedDot(experts, shape.k, shape.n, dev, seed=2000 + rank, dispatch=mode)
            out = layer.forward(x_tokens, routing)
            dy = workloads.normal_tensor(tuple(out[0].shape), 1.0, 4000 + rank, dev)
            for _ in range(warm):
                out = layer.forward(x_tokens, routing)
                dx, dW = layer.backward(dy)
            torch.cuda.synchronize()
            ok = torch.ones(1, device=dev)
        except Exception as e:  # e.g. no peer access for symmetric memory
            if rank == 0:
                sys.stderr.write(f"bench: dispatch mode {mode} unavailable: {e!r}\n")
            ok = torch.zeros(1, device=dev)
        dist.all_reduce(ok, op=dist.ReduceOp.MIN)
        if float(ok) == 0:
            continue
        parity[mode] = ep_parity_check(layer, mode, out, dy, dx, dW, routing, world, dev)
        dist.barrier()
        torch.cuda.synchronize()
        sampler = ClockSampler(physical_gpu_index(local)).start()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(args.steps):
            layer.forward(x_tokens, routing)
            layer.backward(dy)
        e1.record()
        torch.cuda.synchronize()
        dist.barrier()
        clocks = sampler.stop()
        ms = e0.elapsed_time(e1) / args.steps
        # the breakdown comes from a second, untimed pass with events between the parts of a step
        layer.reset_timers()
        for _ in range(args.steps):
            layer.forward(x_tokens, routing, timed=True)
            layer.backward(dy, timed=True)
        torch.cuda.synchronize()
        dist.barrier()
        parts = layer.timers_ms(args.steps)
        bparts = layer.backward_timers_ms(args.steps)
        bad = torch.tensor([float(layer.device_status() != 0)], device=dev)
        dist.all_reduce(bad, op=dist.ReduceOp.MAX)
        if float(bad) != 0:
            raise RuntimeError(f"dispatch mode {mode}: a device-side wait expired inside the timed region")
        t = torch.tensor([ms, parts["gemm"], parts["a2a"], parts["permute"], parts.get("own_rows", 0.0),
                          bparts["dlhs_gemm"], bparts["drhs_tgmm"], bparts["return_exchange_and_combine"]],
                         dtype=torch.float64, device=dev)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        results[mode] = t.tolist()
        if mode == "fused":
            # The same per-GPU work with nothing to exchange: the three GEMMs over the rows that are in
            # the receive buffer, on this GPU alone (what a step would cost if the exchange were free).
            sv, cfg = layer._saved, _lib.TileCfg(0, 0, 0, 0, _lib.RD_CFG_NO_ZERO_TAIL)
            ybuf, dbuf = layer._ring["y"], layer._grad["buf"]
            ws1, ws2 = layer._grad["ws"], layer._grad["ws_tgmm"]

            def local_step():
                ops.gmm_forward(sv["recv"], layer.weights, sv["seg"], group_to_weight=sv["seg2e"], cfg=cfg,
                                out=ybuf, workspace=ws1)
                ops.gmm_forward(dy, layer.weights, sv["seg"], trans_rhs=True, group_to_weight=sv["seg2e"], cfg=cfg,
                                out=dbuf, workspace=ws1)
                ops.tgmm_forward(sv["recv"], dy, sv["seg"], seg_count=world, workspace=ws2)

            lt = torch.tensor([_time_ms(local_step, max(args.steps, 5))], dtype=torch.float64, device=dev)
            dist.all_reduce(lt, op=dist.ReduceOp.MAX)
            local_only = float(lt[0])
        del layer, out, dy, dx, dW
        torch.cuda.empty_cache()
    # Decode-shaped case of the same expert layout: 64 tokens x top-4 per GPU (m = 256 rows per rank),
    # weight-bandwidth bound on every rank.  Forward only, timed with the two host-sync-free modes.
    decode = {}
    d_tokens = 64
    xd = workloads.normal_tensor((d_tokens, shape.k), 1.0, 5000 + rank, dev)
    rd_ = torch.from_numpy(workloads.topk_routing(d_tokens, experts, top_k, seed=6000 + rank)).to(dev)
    for mode in ("p2p", "fused"):
        try:
            layer = ep.ExpertParallelRaggedDot(experts, shape.k, shape.n, dev, seed=2000 + rank, dispatch=mode,
                                               capacity_rows=d_tokens * top_k * world)
            for _ in range(warm):
                out = layer.forward(xd, rd_)
            torch.cuda.synchronize()
            ok = torch.ones(1, device=dev)
        except Exception as e:
            if rank == 0:
                sys.stderr.write(f"bench: decode case, mode {mode} unavailable: {e!r}\n")
            ok = torch.zeros(1, device=dev)
        dist.all_reduce(ok, op=dist.ReduceOp.MIN)
        if float(ok) == 0:
            continue
        seg = out[1]
        dist.barrier()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(args.steps):
            layer.forward(xd, rd_)
        e1.record()
        torch.cuda.synchronize()
        dist.barrier()
        n_local = experts // world
        touched = int((seg.view(world, n_local).sum(0) > 0).sum())  # local experts with at least one row
        t = torch.tensor([e0.elapsed_time(e1) / args.steps, float(touched)], dtype=torch.float64, device=dev)
        tmax = t.clone()
        dist.all_reduce(tmax, op=dist.ReduceOp.MAX)
        dist.all_reduce(t, op=dist.ReduceOp.SUM)
        decode[mode] = {"ms_per_step": float(tmax[0]),
                        "weight_GBps_all_gpus": float(t[1]) * shape.k * shape.n * 2 / (float(tmax[0]) * 1e-3) / 1e9,
                        "experts_touched": int(t[1])}
        del layer
        torch.cuda.empty_cache()
    # End to end at N GPUs: every step copies this rank's tokens, routing and the cotangent of the
    # rows it receives from pinned host memory, runs forward + backward of the fastest mode through
    # the public host-buffer calls and reads y, dx and dW back to the host.
    e2e = None
    if results:
        best_t = torch.tensor([results.get(m, [1e30])[0] for m in EP_MODES], dtype=torch.float64, device=dev)
        dist.broadcast(best_t, src=0)
        mode = EP_MODES[int(torch.argmin(best_t))]
        layer = ep.ExpertParallelRaggedDot(experts, shape.k, shape.n, dev, seed=2000 + rank, dispatch=mode)
        hx = x_tokens.cpu().pin_memory()
        hr = routing.to(torch.int32).cpu().pin_memory()
        hrows = torch.zeros(1, dtype=torch.int32).pin_memory()
        cap_rows = tokens * top_k * (world if mode != "nccl" else 1)
        out = layer.forward(x_tokens, routing)  # untimed: how many rows does this rank receive?
        torch.cuda.synchronize()
        rows_valid = int(out[0].shape[0]) if mode == "nccl" else int(out[3].cpu())
        del out
        hy = torch.empty((rows_valid, shape.n), dtype=torch.bfloat16).pin_memory()
        hdy = workloads.normal_tensor((rows_valid, shape.n), 1.0, 4000 + rank, "cpu").pin_memory()
        hdx = torch.empty((tokens, shape.k), dtype=torch.bfloat16).pin_memory()

        def step():  # copy-in of the next step runs under this step's exchange, GEMMs and copy-out
            layer.forward_host(hx, hr, hy, rows_host=hrows)
            layer.backward_host(hdy, rows_valid, hdx)

        for _ in range(2):
            step()
        torch.cuda.synchronize()
        dist.barrier()
        e2e_steps = max(3, min(args.steps, 10))
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(e2e_steps):
            step()
        layer.wait_host_outputs()
        e1.record()
        torch.cuda.synchronize()
        dist.barrier()
        assert int(hrows[0]) == rows_valid
        t = torch.tensor([e0.elapsed_time(e1) / e2e_steps], dtype=torch.float64, device=dev)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        nb = torch.tensor([hx.numel() * 2 + hr.numel() * 4 + hdy.numel() * 2,
                           hy.numel() * 2 + hdx.numel() * 2 + 4], dtype=torch.float64, device=dev)
        dist.all_reduce(nb)
        e2e_ms = float(t[0])
        e2e = {"value": 3 * 2.0 * tokens * top_k * world * shape.k * shape.n / (e2e_ms * 1e-3) / 1e12, "unit": UNIT,
               "ms_per_step": e2e_ms, "steps": e2e_steps, "dispatch": mode,
               "h2d_bytes_per_step": float(nb[0]), "d2h_bytes_per_step": float(nb[1]),
               "api": "ExpertParallelRaggedDot.forward_host + backward_host per rank, pinned host buffers: tokens, "
                      "routing and the cotangent of the rows the rank receives go in, y (the rows received; their "
                      "number is fixed by the inputs and was read once before timing) and dx come out; the weight "
                      "gradient stays on the device beside the weights it belongs to",
               "host_numa": numa_note + " (rank 0)"}
        del layer
        torch.cuda.empty_cache()
    if rank == 0 and results:
        best = min(results, key=lambda m: results[m][0])
        ms = results[best][0]
        rows_global = tokens * top_k * world
        flops = 3 * 2.0 * rows_global * shape.k * shape.n
        gemm_flops_gpu = 2.0 * tokens * top_k * shape.k * shape.n
        row_bytes_out = tokens * top_k * shape.k * 2 * (world - 1) / world
        modes = {}
        for m_, (t_ms, g_ms, x_ms, p_ms, own_ms, dl_ms, dr_ms, ret_ms) in results.items():
            fwd = ({"sort_plan_gather": p_ms, "all_to_all": x_ms, "local_ragged_dot": g_ms} if m_ == "nccl" else
                   {"count_allgather_plan": p_ms, "peer_store_dispatch_and_barrier": x_ms,
                    "local_ragged_dot": g_ms} if m_ == "p2p" else
                   {"count_allgather_plan_assign": p_ms, "own_rows_copied_from_plan_end": own_ms,
                    "fused_send_and_ragged_dot_from_plan_end": g_ms})
            modes[m_] = {
                "ms_per_step": t_ms, "tflops": flops / (t_ms * 1e-3) / 1e12,
                "forward_breakdown_ms": fwd,
                "backward_breakdown_ms": {"dlhs_gemm_on_the_owner": dl_ms, "drhs_tgmm_per_local_expert": dr_ms,
                                          "return_exchange_and_topk_combine": ret_ms},
                # fused: the exchange has no span of its own; rate over the whole send + GEMM kernel
                ("exchange_GBps_per_gpu_over_the_fused_kernel" if m_ == "fused" else "exchange_GBps_per_gpu"):
                    row_bytes_out / ((g_ms if m_ == "fused" else x_ms) * 1e-3) / 1e9,
                "return_exchange_GBps_per_gpu": row_bytes_out / (ret_ms * 1e-3) / 1e9,
                "parity_check": parity.get(m_),
            }
        # Target of one step per GPU: the three GEMMs at the measured tensor peak, or the two exchanges
        # at the measured peer-copy bandwidth (770 GB/s per direction per GPU), whichever is slower.
        target_ms = max(3 * gemm_flops_gpu / (peaks["bf16_tflops"] * 1e9), 2 * row_bytes_out / 770e9 * 1e3)
        line = {
            "metric": METRIC, "value": flops / (ms * 1e-3) / 1e12, "unit": UNIT, "n_gpus": world,
            "steps": args.steps, "warmup": warm, "ms_per_step": ms, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "bf16", "data": "synthetic",
            "config": ep_config(shape, world, tokens, top_k, experts, tokens * world),
            "method": "CUDA events on the launch stream, barrier + synchronize on both sides, max over ranks",
            "dispatch": best, "collective": EP_COLLECTIVE[best],
            "clocks": clocks,
            "gpu_launches": EP_LAUNCHES[best] * args.steps,
            "parity_check": parity.get(best),
            "local_only_ms": local_only,
            "local_only_note": "the same three GEMMs per GPU over the received rows with nothing exchanged: "
                               "step efficiency on one workload = local_only_ms / ms_per_step",
            "roofline": {"bound": "tensor", "kernel": "ragged_gemm2_kernel<gmm> (flag-gated, sender CTAs in the "
                                                      "launch) + <gmm, trans_rhs> + <tgmm, strided segments>",
                         "achieved": 3 * gemm_flops_gpu / (ms * 1e-3) / 1e12, "peak": peaks["bf16_tflops"],
                         "unit": "TFLOP/s", "frac": target_ms / ms, "target_ms": target_ms, "traffic": None,
                         "note": "per GPU over the whole step; frac = max(3 GEMMs at the measured tensor peak, two "
                                 "exchanges at 770 GB/s) / measured step",
                         "peak_source": peaks["source"] + "; NVLink 770 GB/s per direction"},
            "dispatch_modes": modes,
            "decode_case": {"tokens_per_gpu": d_tokens, "top_k": top_k, "rows_per_gpu": d_tokens * top_k,
                            "note": "forward only: exchange + local ragged_dot per step; latency-bound (a few small "
                                    "kernels and one all-gather), weights read once per touched expert",
                            "modes": decode},
            "e2e": e2e,
        }
        print(json.dumps(line), flush=True)
    dist.destroy_process_group()


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=50)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--only", default=None, choices=["fwd", "dlhs", "drhs"])
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-other-workloads", action="store_true")
    ap.add_argument("--dtype", default="bf16", choices=["bf16", "f32", "e4m3"],
                    help="N=1 profiling runs only: f32 times the TF32 kernels, e4m3 the 8-bit forward "
                         "(rd_gmm_fp8; with --only fwd); use with --no-e2e --no-cpu-baseline")
    ap.add_argument("--workload", default="mixtral",
                    choices=["mixtral", "decode", "deepseek", "deepseek_quarter", "permute"],
                    help="N=1 only; the headline line is the default (mixtral); the others are for profiling")
    args = ap.parse_args()
    if args.impl == "reference":
        run_reference(args)
        return
    if not torch.cuda.is_available():
        raise SystemExit("bench.py: no CUDA device; the product has no CPU path (use --impl reference for the CPU oracle)")
    _, world, _ = dist_env()
    if world > 1 or args.gpus > 1:
        run_expert_parallel(args)
    elif args.workload == "permute":
        run_permute(args)
    else:
        run_single(args)


if __name__ == "__main__":
    main()
