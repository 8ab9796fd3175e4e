#!/usr/bin/env python
"""Benchmark of the fused-MoE layer (``fused_experts``) on B200.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--workload NAME] [--tokens M]
    python bench.py --impl reference ...      # the reference's torch CPU path (oracle port)

One "step" is one MoE layer forward over a batch of M synthetic tokens: dynamic
activation quantisation, token-to-expert sort, gather, both grouped GEMMs (SiLU-
and-mul fused), top-k combine -- the stages the reference times.  Weights and
routing are generated once from a seed (untimed).  Rank 0 prints ONE JSON line.

N > 1 (launched through torch.distributed.run): experts are sharded contiguously
over the ranks (expert parallelism), every rank brings its own M tokens (weak
scaling), tokens travel to the owning rank and back with NCCL all-to-all.
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
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

import torch  # noqa: E402

FP8 = torch.float8_e4m3fn

# name -> shape of the benchmark configurations (E experts, K top-k, H hidden, I intermediate)
WORKLOADS = {
    "small_bf16": dict(kind="bf16", E=8, K=2, H=1024, I=512, M=64),
    "mixtral_8x7b_bf16": dict(kind="bf16", E=8, K=2, H=4096, I=14336, M=8192),
    "deepseek_v3_fp8_block": dict(kind="fp8_block", E=256, K=8, H=7168, I=2048, M=4096),
    "qwen3_30b_int8_channel": dict(kind="int8_channel", E=128, K=8, H=2048, I=768, M=16384),
    "qwen3_235b_fp8_block_zipf": dict(kind="fp8_block", E=128, K=8, H=4096, I=1536, M=256,
                                      zipf=1.2),
    # the DeepSeek-V3 shape in the native-MXFP8 recipe (E8M0 scale bytes per 32 K elements)
    "deepseek_v3_mxfp8": dict(kind="mxfp8", E=256, K=8, H=7168, I=2048, M=4096),
    # ... and in the MXFP4 (w4a8) recipe: packed e2m1 weights, dynamic 1 x 128 activation groups
    "deepseek_v3_mxfp4": dict(kind="mxfp4", E=256, K=8, H=7168, I=2048, M=4096),
}
DEFAULT_WORKLOAD = "deepseek_v3_fp8_block"

# DRAM bytes per launch of the dominant kernel (dram__bytes_read.sum + dram__bytes_write.sum of
# one ncu capture), keyed by (workload, tokens); None when no capture exists for that case.
# The capture ran on 64 of the 256 experts with the same rows per expert; DRAM traffic of this
# kernel is proportional to the expert count, so the figure is that capture's times 256/64.
NCU_TRAFFIC_BYTES = {
    ("deepseek_v3_fp8_block", 4096): 8.68e9,
}

# Dense 8-bit tensor-core peaks of this pool's B200s, measured with the recipe of the bf16
# figure in MEASURED_PEAKS.json (8192^3, best of 10 = burst, back to back for 4 s = sustained;
# `python bench.py --measure-peaks` repeats the measurement and prints it).
TENSOR_PEAKS_8BIT = {
    "fp8": dict(burst=3058.5, sustained=2633.1),
    "int8": dict(burst=3225.4, sustained=2691.9),
    "source": "bench.py --measure-peaks on a B200 of this pool, 2026-11-25, torch 2.11.0+cu128; "
              "the same run gave bf16 1678.3 burst / 1398.2 sustained",
}


def measure_tensor_peaks(device):
    """Library GEMM peaks (cuBLASLt through torch): bf16, e4m3 and int8 at 8192^3."""
    n = 8192
    out = {}

    def run(name, fn):
        for _ in range(3):
            fn()
        torch.cuda.synchronize()
        best = float("inf")
        for _ in range(10):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            fn()
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1))
        t0 = time.perf_counter()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        reps = 0
        while time.perf_counter() - t0 < 4.0:
            for _ in range(20):
                fn()
            reps += 20
            torch.cuda.synchronize()
        e1.record()
        torch.cuda.synchronize()
        out[name] = dict(burst=2.0 * n ** 3 / (best * 1e-3) / 1e12,
                         sustained=2.0 * n ** 3 * reps / (e0.elapsed_time(e1) * 1e-3) / 1e12)

    a16 = torch.randn(n, n, device=device, dtype=torch.bfloat16)
    b16 = torch.randn(n, n, device=device, dtype=torch.bfloat16)
    run("bf16", lambda: torch.matmul(a16, b16))
    a8, b8 = a16.to(FP8), b16.to(FP8).t().contiguous().t()
    one = torch.ones((), device=device, dtype=torch.float32)
    try:
        run("fp8", lambda: torch._scaled_mm(a8, b8, scale_a=one, scale_b=one,
                                            out_dtype=torch.bfloat16))
    except Exception as exc:  # noqa: BLE001 - report and carry on
        out["fp8"] = dict(error=str(exc)[:200])
    ai = torch.randint(-8, 8, (n, n), device=device, dtype=torch.int8)
    bi = torch.randint(-8, 8, (n, n), device=device, dtype=torch.int8).t().contiguous().t()
    try:
        run("int8", lambda: torch._int_mm(ai, bi))
    except Exception as exc:  # noqa: BLE001
        out["int8"] = dict(error=str(exc)[:200])
    out["how"] = ("torch.matmul bf16 / torch._scaled_mm e4m3 (bf16 out) / torch._int_mm, 8192^3, "
                  "2*N^3 ops: best of 10 (burst) and back to back for 4 s (sustained)")
    out["torch"] = torch.__version__
    out["gpu"] = torch.cuda.get_device_name(device)
    return out


def load_peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(path):
        with open(path) as f:
            d = json.load(f)
        return dict(hbm_gbs=d["hbm_gbs"], bf16_tflops=d["bf16_tflops"],
                    bf16_tflops_sustained=d.get("bf16_tflops_sustained", d["bf16_tflops"]),
                    source="measured")
    return dict(hbm_gbs=6650.0, bf16_tflops=1590.0, bf16_tflops_sustained=1400.0,
                source="fallback")


def tensor_peak(kind, peaks):
    """(TFLOP/s, source) of the dense tensor-core peak a workload kind is held against: the
    measured burst figure of the matching library GEMM, else twice the measured bf16 figure."""
    if kind == "bf16":
        return peaks["bf16_tflops"], peaks["source"] + " bf16 burst (MEASURED_PEAKS.json)"
    key = "int8" if kind.startswith("int8") else "fp8"
    got = TENSOR_PEAKS_8BIT[key]["burst"]
    if got:
        return got, f"measured {key} burst ({TENSOR_PEAKS_8BIT['source']})"
    return 2.0 * peaks["bf16_tflops"], peaks["source"] + " bf16 burst x2 (no measured 8-bit peak)"


# ---------------------------------------------------------------------------
# synthetic inputs (seeded; generated on the device expert by expert)
# ---------------------------------------------------------------------------
def _quant_block_fp8(w):
    n, k = w.shape
    v = w.float().reshape(n // 128, 128, k // 128, 128)
    amax = v.abs().amax(dim=(1, 3), keepdim=True).clamp(min=1e-10)
    s = amax / 448.0
    q = (v / s).clamp(-448, 448).to(FP8).reshape(n, k)
    return q, s.reshape(n // 128, k // 128)


def _quant_mx(w):
    """1 x 32 groups, exponent byte = ceil(log2(amax/448)) + 127, e4m3 codes."""
    n, k = w.shape
    v = w.float().reshape(n, k // 32, 32)
    amax = v.abs().amax(-1).clamp_min(torch.finfo(torch.float32).tiny)
    e = (torch.ceil(torch.log2(amax / 448.0)) + 127).clamp(0, 254)
    q = (v * torch.exp2(127 - e)[..., None]).to(FP8).reshape(n, k)
    return q, e.to(torch.uint8)


def _quant_mxfp4(w):
    """1 x 32 groups, exponent byte = ceil(log2(amax/6)) + 127, e2m1 codes (nearest of
    0, .5, 1, 1.5, 2, 3, 4, 6), two codes per byte, low nibble first."""
    n, k = w.shape
    v = w.float().reshape(n, k // 32, 32)
    amax = v.abs().amax(-1).clamp_min(torch.finfo(torch.float32).tiny)
    e = (torch.ceil(torch.log2(amax / 6.0)) + 127).clamp(0, 254)
    y = (v * torch.exp2(127 - e)[..., None]).reshape(n, k)
    lut = torch.tensor([0., .5, 1., 1.5, 2., 3., 4., 6.], device=w.device)
    code = (y.abs()[..., None] - lut).abs().argmin(-1).to(torch.uint8) | ((y < 0).to(torch.uint8) << 3)
    return code[:, 0::2] | (code[:, 1::2] << 4), e.to(torch.uint8)


def _quant_channel_int8(w):
    amax = w.float().abs().amax(dim=-1, keepdim=True).clamp(min=1e-10)
    s = amax / 127.0
    return (w.float() / s).round().clamp(-128, 127).to(torch.int8), s.squeeze(-1)


def make_weights(cfg, device, experts, seed):
    """Weights of the listed (global) expert ids: ~N(0, 0.02) masters, quantised per
    the workload kind.  Each expert has its own seed, so any rank can build any shard."""
    kind, H, I = cfg["kind"], cfg["H"], cfg["I"]
    n = len(experts)
    if kind == "bf16":
        w1 = torch.empty(n, 2 * I, H, dtype=torch.bfloat16, device=device)
        w2 = torch.empty(n, H, I, dtype=torch.bfloat16, device=device)
        w1s = w2s = None
    elif kind == "fp8_block":
        w1 = torch.empty(n, 2 * I, H, dtype=FP8, device=device)
        w2 = torch.empty(n, H, I, dtype=FP8, device=device)
        w1s = torch.empty(n, 2 * I // 128, H // 128, dtype=torch.float32, device=device)
        w2s = torch.empty(n, H // 128, I // 128, dtype=torch.float32, device=device)
    elif kind == "mxfp8":
        w1 = torch.empty(n, 2 * I, H, dtype=FP8, device=device)
        w2 = torch.empty(n, H, I, dtype=FP8, device=device)
        w1s = torch.empty(n, 2 * I, H // 32, dtype=torch.uint8, device=device)
        w2s = torch.empty(n, H, I // 32, dtype=torch.uint8, device=device)
    elif kind == "mxfp4":
        w1 = torch.empty(n, 2 * I, H // 2, dtype=torch.uint8, device=device)
        w2 = torch.empty(n, H, I // 2, dtype=torch.uint8, device=device)
        w1s = torch.empty(n, 2 * I, H // 32, dtype=torch.uint8, device=device)
        w2s = torch.empty(n, H, I // 32, dtype=torch.uint8, device=device)
    else:
        w1 = torch.empty(n, 2 * I, H, dtype=torch.int8, device=device)
        w2 = torch.empty(n, H, I, dtype=torch.int8, device=device)
        w1s = torch.empty(n, 2 * I, dtype=torch.float32, device=device)
        w2s = torch.empty(n, H, dtype=torch.float32, device=device)
    g = torch.Generator(device=device)
    for j, e in enumerate(experts):
        g.manual_seed(seed * 100003 + e)
        m1 = torch.randn(2 * I, H, generator=g, device=device) * 0.02
        m2 = torch.randn(H, I, generator=g, device=device) * 0.02
        if kind == "bf16":
            w1[j], w2[j] = m1.bfloat16(), m2.bfloat16()
        elif kind == "fp8_block":
            w1[j], w1s[j] = _quant_block_fp8(m1)
            w2[j], w2s[j] = _quant_block_fp8(m2)
        elif kind == "mxfp8":
            w1[j], w1s[j] = _quant_mx(m1)
            w2[j], w2s[j] = _quant_mx(m2)
        elif kind == "mxfp4":
            w1[j], w1s[j] = _quant_mxfp4(m1)
            w2[j], w2s[j] = _quant_mxfp4(m2)
        else:
            w1[j], w1s[j] = _quant_channel_int8(m1)
            w2[j], w2s[j] = _quant_channel_int8(m2)
    return w1, w2, w1s, w2s


def make_routing(m, num_experts, topk, seed, zipf_alpha=None):
    """Router logits ~N(0,1) -> softmax -> top-k -> renormalise (fp32 weights, int32
    ids).  With ``zipf_alpha`` the experts of a token are drawn without replacement from
    p(e) ~ (rank_e + 1)^-alpha over a seed-fixed expert permutation."""
    g = torch.Generator().manual_seed(seed)
    logits = torch.randn(m, num_experts, generator=g, dtype=torch.float32)
    scores = torch.softmax(logits, dim=-1)
    if zipf_alpha is None:
        wts, ids = torch.topk(scores, k=topk, dim=-1)
    else:
        perm = torch.randperm(num_experts, generator=g)
        p = (torch.arange(num_experts, dtype=torch.float64) + 1.0) ** (-zipf_alpha)
        prob = torch.empty(num_experts, dtype=torch.float64)
        prob[perm] = p / p.sum()
        ids = torch.multinomial(prob.expand(m, -1), topk, replacement=False, generator=g)
        wts = scores.gather(1, ids)
    wts = wts / wts.sum(dim=-1, keepdim=True)
    return wts.float().contiguous(), ids.to(torch.int32).contiguous()


def make_tokens(cfg, m, seed):
    """hidden ~N(0,1) bf16 and softmax top-k routing, on the host."""
    g = torch.Generator().manual_seed(seed)
    hidden = torch.randn(m, cfg["H"], generator=g).bfloat16()
    wts, ids = make_routing(m, cfg["E"], cfg["K"], seed + 1, cfg.get("zipf"))
    return hidden, wts, ids


def layer_kwargs(cfg, w1s, w2s):
    if cfg["kind"] == "fp8_block":
        return dict(use_fp8_w8a8=True, w1_scale=w1s, w2_scale=w2s, block_shape=[128, 128])
    if cfg["kind"] == "int8_channel":
        return dict(use_int8_w8a8=True, per_channel_quant=True, w1_scale=w1s, w2_scale=w2s)
    if cfg["kind"] == "mxfp8":
        return dict(use_mxfp8=True, w1_scale=w1s, w2_scale=w2s, block_shape=[1, 32])
    if cfg["kind"] == "mxfp4":
        return dict(use_mxfp4_w4a8=True, use_ue8m0=True, w1_scale=w1s, w2_scale=w2s,
                    block_shape=[1, 32])
    return {}


# ---------------------------------------------------------------------------
# clocks
# ---------------------------------------------------------------------------
class ClockSampler:
    """SM clock and throttle reasons sampled while the timed region runs.

    NVML is read from a thread every few milliseconds (a timed region of a few steps lasts
    tens of milliseconds, so a 100 ms `nvidia-smi -lms` loop would mostly see the idle GPU
    around it); `nvidia-smi` is the fallback when the NVML binding is missing.  Read-only.
    """
    FIELDS = ("clocks.sm,clocks.max.sm,clocks_event_reasons.hw_slowdown,"
              "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
              "clocks_event_reasons.sw_power_cap")

    def __init__(self, index):
        self.index, self.rows, self.proc = index, [], None
        self.nvml, self.handle, self.thread, self.stop_flag = None, None, None, False
        self.max_mhz, self.reasons = 0, set()

    def _nvml_loop(self):
        n = self.nvml
        masks = (("hw_slowdown", n.nvmlClocksEventReasonHwSlowdown),
                 ("hw_thermal_slowdown", n.nvmlClocksEventReasonHwThermalSlowdown),
                 ("sw_thermal_slowdown", n.nvmlClocksEventReasonSwThermalSlowdown),
                 ("sw_power_cap", n.nvmlClocksEventReasonSwPowerCap))
        while not self.stop_flag:
            try:
                self.rows.append(float(n.nvmlDeviceGetClockInfo(self.handle, n.NVML_CLOCK_SM)))
                bits = n.nvmlDeviceGetCurrentClocksEventReasons(self.handle)
                for name, mask in masks:
                    if bits & mask:
                        self.reasons.add(name)
            except Exception:
                break
            time.sleep(0.002)

    def start(self):
        try:
            import pynvml as n
            n.nvmlInit()
            # NVML enumerates physical devices: map the CUDA ordinal through its PCI bus id
            try:
                import torch
                bus = torch.cuda.get_device_properties(self.index).pci_bus_id
                dom = torch.cuda.get_device_properties(self.index).pci_domain_id
                dev = torch.cuda.get_device_properties(self.index).pci_device_id
                self.handle = n.nvmlDeviceGetHandleByPciBusId(f"{dom:08x}:{bus:02x}:{dev:02x}.0")
            except Exception:
                self.handle = n.nvmlDeviceGetHandleByIndex(self.index)
            self.max_mhz = float(n.nvmlDeviceGetMaxClockInfo(self.handle, n.NVML_CLOCK_SM))
            self.nvml = n
            self.thread = threading.Thread(target=self._nvml_loop, daemon=True)
            self.thread.start()
            return
        except Exception:
            self.nvml = None
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-i", str(self.index), "-lms", "100"], stdout=subprocess.PIPE, text=True)
            threading.Thread(target=self._read, daemon=True).start()
        except OSError:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.rows.append([x.strip() for x in line.split(",")])

    def stop(self):
        if self.nvml is not None:
            self.stop_flag = True
            self.thread.join(timeout=2)
            sm = [r for r in self.rows if isinstance(r, float)]
            return dict(sm_mhz=statistics.median(sm) if sm else None,
                        sm_min_mhz=min(sm) if sm else None, sm_max_mhz=self.max_mhz or None,
                        reasons=sorted(self.reasons), samples=len(sm), source="nvml")
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()
        sm, mx, reasons = [], 0, set()
        for r in self.rows:
            try:
                sm.append(float(r[0]))
                mx = max(mx, float(r[1]))
            except (ValueError, IndexError):
                continue
            for name, val in zip(("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown",
                                  "sw_power_cap"), r[2:6]):
                if val.lower().startswith("active"):
                    reasons.add(name)
        return dict(sm_mhz=statistics.median(sm) if sm else None, sm_max_mhz=mx or None,
                    reasons=sorted(reasons), samples=len(sm), source="nvidia-smi")


# ---------------------------------------------------------------------------
# roofline bookkeeping
# ---------------------------------------------------------------------------
def host_memory_near_gpu(local_rank):
    """Before the pinned host buffers are allocated: prefer the NUMA node the GPU hangs off, so
    that eight ranks do not all stage their copies through node 0.  Reads the node from sysfs
    (PCI address from NVML), narrows the CPU affinity to that node's CPUs when the process is
    allowed on any of them, and asks for that node's memory (set_mempolicy, MPOL_PREFERRED).
    Touches only this process; every step is optional and reported in the JSON line."""
    info = dict(gpu_node=None, cpus_bound=0, mempolicy=False)
    try:
        import pynvml
        pynvml.nvmlInit()
        bus = pynvml.nvmlDeviceGetPciInfo(pynvml.nvmlDeviceGetHandleByIndex(local_rank)).busId
        bus = bus.decode() if isinstance(bus, bytes) else bus
        bdf = bus.lower()[-12:]                    # 0000:1b:00.0
        node = int(open(f"/sys/bus/pci/devices/{bdf}/numa_node").read())
        if node < 0:
            return info
        info["gpu_node"] = node
        cpus = set()
        for part in open(f"/sys/devices/system/node/node{node}/cpulist").read().strip().split(","):
            lo, _, hi = part.partition("-")
            cpus.update(range(int(lo), int(hi or lo) + 1))
        allowed = os.sched_getaffinity(0) & cpus
        if allowed:
            os.sched_setaffinity(0, allowed)
            info["cpus_bound"] = len(allowed)
        import ctypes
        mask = ctypes.c_ulong(1 << node)
        rc = ctypes.CDLL(None, use_errno=True).syscall(238, 1, ctypes.byref(mask), 64)  # x86-64
        info["mempolicy"] = rc == 0
    except Exception as exc:                       # no NVML, no sysfs, other architecture ...
        info["error"] = type(exc).__name__
    return info


def gemm1_algorithmic(cfg, m, active_experts):
    """Algorithmic bytes and flops of one GEMM1 launch (gate/up GEMM + fused epilogue)."""
    K, H, I = cfg["K"], cfg["H"], cfg["I"]
    routes = m * K
    wb = 2 if cfg["kind"] == "bf16" else (0.5 if cfg["kind"] == "mxfp4" else 1)
    ab = 2 if cfg["kind"] in ("bf16", "mxfp4") else 1     # mxfp4: decoded 16-bit operands
    ob = 1 if cfg["kind"] in ("fp8_block", "mxfp8") else 2
    byts = active_experts * 2 * I * H * wb + routes * H * ab + routes * I * ob
    if cfg["kind"] == "fp8_block":
        byts += active_experts * (2 * I // 128) * (H // 128) * 4 + routes * (H // 128) * 4 \
            + routes * (I // 128) * 4
    if cfg["kind"] == "mxfp8":    # one scale byte per 32 elements of weights, inputs and outputs
        byts += active_experts * 2 * I * (H // 32) + routes * (H // 32) + routes * (I // 32)
    if cfg["kind"] == "mxfp4":    # what the kernels stream today: weights decoded to 16 bits
        byts = active_experts * 2 * I * H * 2 + routes * H * 2 + routes * 2 * I * 2
    return int(byts), 4.0 * routes * H * I


def layer_flops(cfg, m):
    return 6.0 * m * cfg["K"] * cfg["H"] * cfg["I"]


# ---------------------------------------------------------------------------
# the reference arm: the reference's torch path (CPU oracle port) on host cores
# ---------------------------------------------------------------------------
def cpu_reference(cfg, m, seed, budget_experts=None):
    """Time the CPU oracle on a bounded sample: the routes of the first ``E_s`` experts
    of the M-token batch (all quantisation + both GEMMs + activation for those experts),
    extrapolated linearly in the number of experts.  Returns tokens/s and a description."""
    from oracle import moe_oracle as O

    cores = os.cpu_count() or 1
    torch.set_num_threads(cores)
    E, K = cfg["E"], cfg["K"]
    per_expert_flops = layer_flops(cfg, m) / E
    # aim for ~15 s at an assumed ~25 GFLOP/s/core effective rate of the fp32 reference path
    if budget_experts is None:
        budget_experts = int(max(1, min(E, 15.0 * cores * 25e9 / max(per_expert_flops, 1.0))))
        budget_experts = max(1, min(budget_experts, 32 if cfg["kind"] != "bf16" else E))
        if cfg["kind"] in ("mxfp8", "mxfp4"):   # the oracle holds fp32 copies of the sampled experts
            budget_experts = min(budget_experts, 8)
    es = budget_experts
    hidden, wts, ids = make_tokens(cfg, m, seed)
    w1, w2, w1s, w2s = make_weights(cfg, "cpu", list(range(es)), seed)
    emap = torch.full((E,), -1, dtype=torch.int32)
    emap[:es] = torch.arange(es, dtype=torch.int32)
    tok_sample = m
    t0 = time.perf_counter()
    if cfg["kind"] == "fp8_block":
        O.moe_block_fp8(hidden, w1, w2, w1s, w2s, wts, ids, (128, 128), expert_map=emap)
    elif cfg["kind"] == "int8_channel":
        O.moe_per_channel(hidden, w1, w2, w1s, w2s, wts, ids, torch.int8, expert_map=emap)
    elif cfg["kind"] == "mxfp8":
        O.moe_mxfp8(hidden, w1, w2, w1s, w2s, wts, ids, expert_map=emap)
    elif cfg["kind"] == "mxfp4":
        # (this oracle walks the routes one by one: a token sample bounds its time)
        tok_sample = min(m, 512)
        O.moe_mxfp4(hidden[:tok_sample], w1, w2, w1s, w2s, wts[:tok_sample], ids[:tok_sample],
                    expert_map=emap)
    else:
        sel_ids = torch.where(ids < es, ids, torch.full_like(ids, -1))
        O.moe_bf16(hidden, w1, w2, wts, sel_ids)
    dt = time.perf_counter() - t0
    full = dt * E / es * (m / tok_sample)
    sample = (f"oracle port of the reference torch path on {es} of {E} experts of "
              + (f"the M={m} batch" if tok_sample == m else f"{tok_sample} tokens of the M={m} batch")
              + f" ({dt:.1f} s), scaled by {E}/{es}" + ("" if tok_sample == m else f" x {m}/{tok_sample}"))
    return m / full, cores, sample, full


def spot_check(cfg, out, hidden_h, wts_h, ids_h, device, seed, tokens=8):
    """``out`` against the CPU oracle on a few tokens; only the experts those tokens use are built
    (on the device, from the per-expert seed) and copied to the host.  Criterion: 8-bit kinds, the
    reference's own for its w8a8 layer test -- mean |actual - expected| / mean |expected| < 0.02
    (test/fused_moe/test_fused_moe.py:639-645 of the reference project); 16-bit experts, relative
    L2 error <= 1e-2.  Both figures are reported."""
    from oracle import moe_oracle as O

    m = hidden_h.shape[0]
    toks = sorted({(i * (m - 1)) // max(tokens - 1, 1) for i in range(tokens)})
    used = sorted(set(ids_h[toks].reshape(-1).tolist()))
    remap = {e: j for j, e in enumerate(used)}
    w1, w2, w1s, w2s = (None if t is None else t.cpu()
                        for t in make_weights(cfg, device, used, seed))
    loc = torch.tensor([[remap[int(e)] for e in row] for row in ids_h[toks]], dtype=torch.int32)
    h, w = hidden_h[toks], wts_h[toks]
    if cfg["kind"] == "fp8_block":
        expect = O.moe_block_fp8(h, w1, w2, w1s, w2s, w, loc, (128, 128))
    elif cfg["kind"] == "int8_channel":
        expect = O.moe_per_channel(h, w1, w2, w1s, w2s, w, loc, torch.int8)
    elif cfg["kind"] == "mxfp8":
        expect = O.moe_mxfp8(h, w1, w2, w1s, w2s, w, loc)
    elif cfg["kind"] == "mxfp4":
        expect = O.moe_mxfp4(h, w1, w2, w1s, w2s, w, loc)
    else:
        expect = O.moe_bf16(h, w1, w2, w, loc)
    torch.cuda.synchronize()
    actual = out[toks].cpu()
    err = O.rel_l2(actual, expect)
    mean_rel = float((actual.float() - expect.float()).abs().mean() / expect.float().abs().mean())
    if cfg["kind"] == "bf16":
        criterion, tol, ok = "rel_l2", 1e-2, err <= 1e-2
    else:
        criterion, tol, ok = "mean_rel", 2e-2, mean_rel < 2e-2
    return dict(rel_l2=err, mean_rel=mean_rel, criterion=criterion, tolerance=tol,
                tokens=len(toks), experts_rebuilt=len(used), ok=bool(ok))


# ---------------------------------------------------------------------------
def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default=DEFAULT_WORKLOAD, choices=sorted(WORKLOADS))
    ap.add_argument("--tokens", type=int, default=0, help="tokens per GPU (0 = workload default)")
    ap.add_argument("--experts", type=int, default=0,
                    help="shrink the expert count (profiling captures of a reduced case)")
    ap.add_argument("--seed", type=int, default=0)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--measure-peaks", action="store_true",
                    help="measure the library GEMM peaks (bf16, e4m3, int8) on cuda:0 and exit")
    ap.add_argument("--ep-direct", type=int, default=1,
                    help="N > 1: 1 = exchange over peer memory (no collective call and no host "
                         "synchronisation on the data path), 0 = NCCL all-to-all")
    ap.add_argument("--ep-return", default="routes", choices=["routes", "partials"],
                    help="N > 1, peer memory: what the owners write back -- every route's row from "
                         "the down projection's epilogue, or one partial row per token from their combine")
    ap.add_argument("--ep-replicate-below", type=int, default=4096,
                    help="N > 1: batches of at most this many tokens over all ranks take the "
                         "replicated-token path (all-gather + reduce-scatter); 0 = never")
    ap.add_argument("--ep-chunks", type=int, default=1,
                    help="N > 1: token chunks of the pipelined dispatch / return exchange (1 = serial)")
    ap.add_argument("--ep-comm-sms", type=int, default=16,
                    help="N > 1: SMs left to the exchange kernels while GEMMs run beside them "
                         "(also the CTA limit given to NCCL)")
    ap.add_argument("--no-numa", action="store_true",
                    help="N > 1: leave CPU affinity and memory policy of the ranks as they are")
    ap.add_argument("--graph", action="store_true",
                    help="replay the layer from a CUDA graph in the device-resident timing (1 GPU, or "
                         "N > 1 with the exchange over peer memory)")
    args = ap.parse_args()

    if args.measure_peaks:
        print(json.dumps(dict(tensor_peaks=measure_tensor_peaks(torch.device("cuda", 0)))),
              flush=True)
        return
    cfg = dict(WORKLOADS[args.workload])
    if args.experts:
        cfg["E"] = args.experts
    m = args.tokens or cfg["M"]
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    warmup = max(args.warmup, 3)
    config = dict(workload=f"{args.workload}_M{m}" + (f"_E{cfg['E']}" if args.experts else ""),
                  experts=cfg["E"], topk=cfg["K"],
                  hidden=cfg["H"], intermediate=cfg["I"], tokens_per_gpu=m,
                  parallelism=f"ep{world}" if world > 1 else "single",
                  l2="inputs larger than L2 (weights stream from HBM every step)")
    dtype = {"bf16": "bf16", "fp8_block": "fp8_e4m3", "int8_channel": "int8",
             "mxfp8": "mxfp8_e4m3", "mxfp4": "mxfp4_e2m1_x_e4m3"}[cfg["kind"]]

    if args.impl == "reference":
        if rank != 0:
            return
        value = None
        samples = []
        for _ in range(max(1, min(args.steps, 1))):
            value, cores, sample, full = cpu_reference(cfg, m, args.seed)
            samples.append(full)
        line = dict(metric="moe_layer_tokens_per_s", value=value, unit="tokens/s",
                    n_gpus=args.gpus, steps=1, warmup=0, ms_per_step=full * 1e3,
                    higher_is_better=True, scaling="weak", vs_baseline=None, dtype=dtype,
                    data="synthetic", config=config, impl="reference",
                    cpu_baseline=dict(value=value, unit="tokens/s", cores=cores, kind="port",
                                      sample=sample),
                    e2e=dict(value=value, unit="tokens/s", h2d_bytes_per_step=0,
                             d2h_bytes_per_step=0))
        print(json.dumps(line), flush=True)
        return

    from boltops_b200 import _cabi
    from boltops_b200.fused_moe import fused_experts, layer, ops

    _cabi.load()
    kind = {"bf16": _cabi.GEMM_BF16, "fp8_block": _cabi.GEMM_FP8_BLOCK,
            "int8_channel": _cabi.GEMM_INT8_CHANNEL, "mxfp8": _cabi.GEMM_MXFP8,
            "mxfp4": _cabi.GEMM_MXFP4}[cfg["kind"]]
    # (rows that return to peers keep the layer on row tiles)
    sizes = () if world > 1 and args.ep_direct else (cfg["H"], cfg["I"], cfg["E"] // world)
    config["gemm_schedule"] = layer.gemm_schedule(kind, m * cfg["K"] * world, cfg["E"], *sizes)
    torch.cuda.set_device(local_rank)
    device = torch.device("cuda", local_rank)
    dist = None
    if world > 1:
        import torch.distributed as dist_mod

        dist = dist_mod
        if args.ep_chunks > 1 and args.ep_comm_sms > 0:
            # the exchange kernels run beside the expert GEMMs: keep them on the SMs left to them
            os.environ.setdefault("NCCL_MAX_CTAS", str(args.ep_comm_sms))
        dist.init_process_group("nccl", device_id=device)

    numa = host_memory_near_gpu(local_rank) if world > 1 and not args.no_numa else None
    E = cfg["E"]
    per_rank = E // world
    my_experts = list(range(rank * per_rank, (rank + 1) * per_rank))
    w1, w2, w1s, w2s = make_weights(cfg, device, my_experts, args.seed)
    hidden_h, wts_h, ids_h = make_tokens(cfg, m, args.seed + 17 * rank)
    hidden_h, wts_h, ids_h = hidden_h.pin_memory(), wts_h.pin_memory(), ids_h.pin_memory()
    hidden, wts, ids = hidden_h.to(device), wts_h.to(device), ids_h.to(device)
    kwargs = layer_kwargs(cfg, w1s, w2s)
    out_host = torch.empty((m, cfg["H"]), dtype=torch.bfloat16).pin_memory()

    if world > 1:
        from boltops_b200.fused_moe.ep import ExpertParallelMoE

        ep = ExpertParallelMoE(dist.group.WORLD, E, device)
        # every rank brings the same number of tokens here, so decode-sized batches may take the
        # replicated-token path (no host round trips); the headline batch stays on the dispatch
        ep.replicate_below = args.ep_replicate_below
        ep.direct_max_tokens = m if args.ep_direct else 0
        ep.direct_return = args.ep_return
        ep.pipeline_chunks = args.ep_chunks
        ep.comm_sms = args.ep_comm_sms
        ep.topk_hint = cfg["K"]
        config["ep_exchange"] = f"peer memory, {args.ep_return} returned" if args.ep_direct \
            else "nccl all-to-all"
        if not args.ep_direct:
            config["ep_chunks"] = ep.num_chunks(m)
            config["ep_comm_sms"] = args.ep_comm_sms

        def step(h, w, i):
            return ep.forward(h, w1, w2, w, i, **kwargs)
    else:
        def step(h, w, i):
            return fused_experts(h, w1, w2, w, i, **kwargs)

    def sync_all():
        torch.cuda.synchronize()
        if dist is not None:
            dist.barrier()
            torch.cuda.synchronize()

    def timed(fn, steps):
        """K steps in one region bracketed by barrier + synchronize; an event after every step
        gives K per-step samples (max over ranks per step).  Returns (median ms per step,
        statistics): the reference reports the median of its samples and re-measures when the
        trimmed spread exceeds 3 % (test/fused_moe/test_fused_moe.py:1317-1331 of the reference);
        here the spread is reported with the number."""
        sync_all()
        evs = [torch.cuda.Event(enable_timing=True) for _ in range(steps + 1)]
        evs[0].record()
        for k in range(steps):
            fn()
            evs[k + 1].record()
        sync_all()
        per = torch.tensor([evs[k].elapsed_time(evs[k + 1]) for k in range(steps)],
                           dtype=torch.float64, device=device)
        total = torch.tensor([evs[0].elapsed_time(evs[steps]) / steps], dtype=torch.float64,
                             device=device)
        if dist is not None:
            dist.all_reduce(per, op=dist.ReduceOp.MAX)
            dist.all_reduce(total, op=dist.ReduceOp.MAX)
        vals = sorted(per.tolist())
        trim = vals[1:-1] if len(vals) >= 5 else vals
        med = statistics.median(vals)
        stats = dict(samples=len(vals), median_ms=med, mean_ms=float(total.item()),
                     min_ms=vals[0], max_ms=vals[-1],
                     trimmed_spread=(trim[-1] - trim[0]) / med if med > 0 else None)
        return med, stats

    # ---- device-resident timing ------------------------------------------------------------
    for _ in range(warmup):
        step(hidden, wts, ids)
    sync_all()
    ops.check_device_status(device)
    sampler = ClockSampler(local_rank)
    if rank == 0:
        sampler.start()
    launches0 = ops.launch_count()
    if args.graph and (world == 1 or args.ep_direct):
        # (N > 1: the peer-memory step holds no host-side state, so it replays from a graph too)
        step(hidden, wts, ids)
        launches = ops.launch_count() - launches0
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            graph_out = step(hidden, wts, ids)
        for _ in range(3):
            graph.replay()
        ms, timing = timed(graph.replay, args.steps)
        config["cuda_graph"] = True
    else:
        ms, timing = timed(lambda: step(hidden, wts, ids), args.steps)
        launches = (ops.launch_count() - launches0) // max(args.steps, 1)

    # ---- end to end through the public API with host buffers ----------------------------
    def e2e_step():
        h = hidden_h.to(device, non_blocking=True)
        w = wts_h.to(device, non_blocking=True)
        i = ids_h.to(device, non_blocking=True)
        out = step(h, w, i)
        out_host.copy_(out, non_blocking=True)
        torch.cuda.current_stream().synchronize()

    for _ in range(2):
        e2e_step()
    ms_e2e, timing_e2e = timed(e2e_step, args.steps)

    # the same traffic double-buffered: step i+1's inputs cross PCIe while step i computes and
    # step i-1's result returns (what a serving loop does); reported next to the strict number
    copy_s = torch.cuda.Stream(device=device)
    bufs = [[torch.empty_like(hidden), torch.empty_like(wts), torch.empty_like(ids)] for _ in range(2)]
    outs_h = [torch.empty_like(out_host).pin_memory() for _ in range(2)]

    def e2e_pipelined(steps):
        main = torch.cuda.current_stream()
        ready = [torch.cuda.Event() for _ in range(2)]
        done = [torch.cuda.Event() for _ in range(2)]
        freed = [torch.cuda.Event() for _ in range(2)]

        def upload(i):
            b = bufs[i % 2]
            with torch.cuda.stream(copy_s):
                copy_s.wait_event(freed[i % 2])
                b[0].copy_(hidden_h, non_blocking=True)
                b[1].copy_(wts_h, non_blocking=True)
                b[2].copy_(ids_h, non_blocking=True)
                ready[i % 2].record(copy_s)

        for e in freed:
            e.record(main)
        upload(0)
        for i in range(steps):
            if i + 1 < steps:
                upload(i + 1)
            b = bufs[i % 2]
            main.wait_event(ready[i % 2])
            out = step(b[0], b[1], b[2])
            freed[i % 2].record(main)
            done[i % 2].record(main)
            with torch.cuda.stream(copy_s):
                copy_s.wait_event(done[i % 2])
                out.record_stream(copy_s)
                outs_h[i % 2].copy_(out, non_blocking=True)
        main.wait_stream(copy_s)

    e2e_pipelined(3)
    sync_all()
    p0, p1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    p0.record()
    e2e_pipelined(args.steps)
    p1.record()
    sync_all()
    ms_e2e_pipe = p0.elapsed_time(p1) / args.steps
    if dist is not None:
        tp = torch.tensor([ms_e2e_pipe], device=device)
        dist.all_reduce(tp, op=dist.ReduceOp.MAX)
        ms_e2e_pipe = float(tp.item())
    clocks = sampler.stop() if rank == 0 else None
    ops.check_device_status(device)

    # ---- per-stage timing of the dominant kernel (rank-local, CUDA events) ---------------
    stage_ms = None
    if world == 1:
        timer = layer.StageTimer()
        layer.STAGE_TIMER = timer
        for _ in range(args.steps):
            step(hidden, wts, ids)
        torch.cuda.synchronize()
        layer.STAGE_TIMER = None
        stage_ms = timer.summary()

    ep_stats = None
    if world > 1:
        ep.profile = True
        layer.STAGE_TIMER = layer.StageTimer()
        step(hidden, wts, ids)
        ep_stats = dict(ep.last_stats)
        ep_stats["local_stage_ms"] = layer.STAGE_TIMER.summary()
        if ep._direct_failed is not None:
            ep_stats["peer_memory_unavailable"] = ep._direct_failed
        layer.STAGE_TIMER = None
        ep.profile = False
        # load balance: routes each rank's experts receive from the whole job (the Zipf workload
        # is measured as it comes, not rebalanced)
        owner = torch.div(ids.long(), cfg["E"] // world, rounding_mode="floor")
        per_rank = torch.bincount(owner.flatten(), minlength=world)[:world].to(torch.float64)
        dist.all_reduce(per_rank)
        ep_stats["routes_per_rank"] = dict(max=float(per_rank.max()), mean=float(per_rank.mean()),
                                           max_over_mean=float(per_rank.max() / per_rank.mean()))
    # ---- correctness of the multi-GPU path: rank 0 rebuilds the experts of four of its tokens
    # (any rank can build any expert from the seed) and holds its output against the CPU oracle
    ep_check = None
    check_out = step(hidden, wts, ids)          # every rank takes part in the exchange
    if rank == 0:
        ep_check = spot_check(cfg, check_out, hidden_h, wts_h, ids_h, device, args.seed)
    if rank != 0:
        if dist is not None:
            dist.destroy_process_group()
        return

    peaks = load_peaks()
    total_tokens = m * world
    value = total_tokens / (ms * 1e-3)
    tflops = layer_flops(cfg, m) * world / (ms * 1e-3) / 1e12
    line = dict(metric="moe_layer_tokens_per_s", value=value, unit="tokens/s", n_gpus=world,
                steps=args.steps, warmup=warmup, ms_per_step=ms, higher_is_better=True,
                scaling="weak", vs_baseline=None, dtype=dtype, data="synthetic", config=config,
                tflops=tflops, gpu_launches=launches, clocks=clocks, timing=timing,
                e2e=dict(value=total_tokens / (ms_e2e * 1e-3), unit="tokens/s",
                         ms_per_step=ms_e2e, timing=timing_e2e,
                         note="value: copies and layer strictly in sequence each step; "
                              "double_buffered: same bytes per step, copies overlapped with compute",
                         double_buffered_value=total_tokens / (ms_e2e_pipe * 1e-3),
                         double_buffered_ms_per_step=ms_e2e_pipe,
                         h2d_bytes_per_step=(hidden_h.numel() * 2 + wts_h.numel() * 4
                                             + ids_h.numel() * 4) * world,
                         d2h_bytes_per_step=out_host.numel() * 2 * world))
    if numa is not None:
        line["e2e"]["host_numa_rank0"] = numa
    if ep_stats is not None:
        line["ep_rank0"] = ep_stats
    if ep_check is not None:
        line["ep_check" if world > 1 else "output_check"] = ep_check
    if stage_ms is not None:
        line["stage_ms"] = stage_ms
        active = int(torch.unique(ids_h).numel())
        byts, flops = gemm1_algorithmic(cfg, m, active)
        g_ms = stage_ms.get("gemm1")
        if g_ms:
            t_hbm = byts / (peaks["hbm_gbs"] * 1e9)
            tc_peak, tc_source = tensor_peak(cfg["kind"], peaks)
            t_tc = flops / (tc_peak * 1e12)
            traffic = NCU_TRAFFIC_BYTES.get((args.workload, m))
            if t_hbm >= t_tc:
                ach = byts / (g_ms * 1e-3) / 1e9
                roof = dict(bound="hbm", achieved=ach, peak=peaks["hbm_gbs"], unit="GB/s",
                            frac=ach / peaks["hbm_gbs"], traffic=traffic)
            else:
                ach = flops / (g_ms * 1e-3) / 1e12
                roof = dict(bound="tensor", achieved=ach, peak=tc_peak, unit="TFLOP/s",
                            frac=ach / tc_peak, traffic=traffic)
            roof.update(kernel=("k_mx_gemm (gate/up GEMM, tensor-core block scaling, activation + MX "
                                "quantisation epilogue)" if cfg["kind"] == "mxfp8" else
                                ("k_stream_gemm" if config["gemm_schedule"] == "stream"
                                 else "k_grouped_gemm") + " (gate/up GEMM + SiLU-mul epilogue)"),
                        ms_per_launch=g_ms, algorithmic_bytes=byts, algorithmic_flops=flops,
                        tensor_time_ms=t_tc * 1e3, hbm_time_ms=t_hbm * 1e3,
                        peak_source=(peaks["source"] + " (MEASURED_PEAKS.json copy bandwidth)"
                                     if t_hbm >= t_tc else tc_source))
            line["roofline"] = roof
    if not args.no_cpu_baseline and world == 1:
        v, cores, sample, _ = cpu_reference(cfg, m, args.seed)
        line["cpu_baseline"] = dict(value=v, unit="tokens/s", cores=cores, kind="port",
                                    sample=sample)
    print(json.dumps(line), flush=True)
    if dist is not None:
        dist.destroy_process_group()
    if ep_check is not None and not ep_check["ok"]:
        raise SystemExit(f"layer output differs from the oracle: {ep_check}")


if __name__ == "__main__":
    main()
