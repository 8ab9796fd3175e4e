"""The work this package is used for, as a list of measurable cases.

Every layer case is one mixture-of-experts layer the way a serving engine runs it: the tokens of
one step, their routing (from the router's logits where the engine has no router of its own, else
ready-made), the expert weights resident on the GPU, one call of ``fused_experts``.  Shapes are
those of the repository's benchmark; token counts go from a single decoding sequence to a full
prefill batch.  The dense case is the block-scaled GEMM that runs beside such a layer (shared
expert).
"""
import math

import torch

from boltops_b200.fused_moe import fused_experts
from boltops_b200.fused_moe.routing import fused_topk
from boltops_b200.gemm import gemm_a8w8_blockscale

FP8 = torch.float8_e4m3fn

# E experts, K routes per token, H hidden size, I intermediate size
SMALL = dict(op="layer", E=8, K=2, H=1024, I=512)
MIXTRAL = dict(op="layer", kind="bf16", E=8, K=2, H=4096, I=14336)
DEEPSEEK = dict(op="layer", kind="fp8_block", K=8, H=7168, I=2048)
QWEN_30B = dict(op="layer", kind="int8_channel", E=128, K=8, H=2048, I=768)
QWEN_235B = dict(op="layer", kind="fp8_block", E=128, K=8, H=4096, I=1536)


def listed():
    return [
        # a test-sized layer on one small batch: nothing but launches and host work
        dict(SMALL, name="small_bf16", kind="bf16", M=64, router=True),
        # 16-bit experts, a few decoding sequences: streams all expert weights once
        dict(MIXTRAL, name="bf16_decode", M=23, router=True),
        # 16-bit experts, full prefill batch: dense tensor-core work
        dict(MIXTRAL, name="bf16_prefill", M=8192, router=False),
        # 8-bit block-scaled experts, one decoding sequence (batch-1 latency)
        dict(DEEPSEEK, name="fp8_decode_one", E=256, M=1, router=True),
        # the same layer, a decode batch that touches nearly every expert
        dict(DEEPSEEK, name="fp8_decode_batch", E=256, M=96, router=True),
        # the same layer, a prefill batch (the headline shape of the benchmark)
        dict(DEEPSEEK, name="fp8_prefill", E=256, M=4096, router=False),
        # one rank of eight with replicated tokens: 32 of 256 experts live here, the rest masked
        dict(DEEPSEEK, name="fp8_expert_parallel_rank", E=256, shards=8, M=16384, router=False),
        # a few hot experts (Zipf-distributed routing), decode batch
        dict(QWEN_235B, name="fp8_decode_skewed", M=256, router=False, zipf=1.2),
        # 8-bit integer experts with per-channel scales, long prefill, many small experts
        dict(QWEN_30B, name="int8_prefill", M=16384, router=True),
        # microscaled experts, a quarter of the 256 on this GPU: ragged prefill chunks
        dict(DEEPSEEK, name="mxfp8_prefill", kind="mxfp8", E=64, M=1000, router=False),
        dict(DEEPSEEK, name="mxfp4_prefill", kind="mxfp4", E=64, M=1500, router=False),
        # shared expert beside the layer: dense block-scaled GEMM on a ragged batch
        dict(op="dense", name="fp8_dense", M=777, N=4096, H=7168),
    ]


def _between(rng, low, high):
    """A whole number spread evenly over the logarithm of [low, high]."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    """One more case: a family, then a token count anywhere in the family's range."""
    family = rng.choice(("small", "mixtral", "deepseek", "deepseek", "parallel", "skewed", "int8",
                         "int8", "mxfp8", "mxfp4", "dense"))
    if family == "small":
        return dict(SMALL, kind=rng.choice(("bf16", "bf16", "f16")), M=_between(rng, 1, 512),
                    router=rng.random() < 0.5, clamp=rng.random() < 0.25)
    if family == "mixtral":
        return dict(MIXTRAL, M=_between(rng, 1, 8192), router=rng.random() < 0.5)
    if family == "deepseek":
        return dict(DEEPSEEK, E=rng.choice((32, 64, 128, 256)), M=_between(rng, 1, 8192),
                    router=rng.random() < 0.5)
    if family == "parallel":
        return dict(DEEPSEEK, E=256, shards=rng.choice((4, 8)), M=_between(rng, 8, 16384),
                    router=False)
    if family == "skewed":
        return dict(QWEN_235B, M=_between(rng, 1, 256), router=False, zipf=1.2)
    if family == "int8":
        return dict(QWEN_30B, M=_between(rng, 16, 16384), router=rng.random() < 0.5)
    if family == "dense":
        n, k = rng.choice(((4096, 7168), (7168, 2048)))
        return dict(op="dense", M=_between(rng, 1, 8192), N=n, H=k)
    return dict(DEEPSEEK, kind=family, E=64, M=_between(rng, 1, 2048), router=False)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _quant_block(w):
    """[..., N, K] -> e4m3 codes and one fp32 scale per 128 x 128 block."""
    *lead, n, k = w.shape
    v = w.view(*lead, n // 128, 128, k // 128, 128)
    s = v.abs().amax(-1).amax(-2).float().clamp_min(1e-10) / 448.0
    q = (v / s[..., :, None, :, None].to(w.dtype)).to(FP8).view(*lead, n, k)
    return q, s


def _quant_channel(w):
    """[..., N, K] -> int8 codes and one fp32 scale per row."""
    s = w.abs().amax(-1).float().clamp_min(1e-10) / 127.0
    return (w / s[..., None].to(w.dtype)).round().clamp_(-127, 127).to(torch.int8), s


def _mx_exponent(v, largest):
    """E8M0 byte of every group: 2^(byte - 127) >= amax / largest."""
    amax = v.abs().amax(-1).float().clamp_min(torch.finfo(torch.float32).tiny)
    return (torch.ceil(torch.log2(amax / largest)) + 127).clamp(0, 254)


def _quant_mxfp8(w):
    v = w.view(*w.shape[:-1], w.shape[-1] // 32, 32)
    e = _mx_exponent(v, 448.0)
    q = (v * torch.exp2(127 - e)[..., None].to(w.dtype)).to(FP8).view(w.shape)
    return q, e.to(torch.uint8)


def _quant_mxfp4(w):
    """e2m1 codes (0, .5, 1, 1.5, 2, 3, 4, 6), two per byte, low nibble first."""
    v = w.view(*w.shape[:-1], w.shape[-1] // 32, 32)
    e = _mx_exponent(v, 6.0)
    y = (v * torch.exp2(127 - e)[..., None].to(w.dtype)).view(w.shape)
    a = y.abs()
    code = torch.zeros(w.shape, dtype=torch.uint8, device=w.device)
    for t in (0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0):
        code += a > t
    code += (y < 0).to(torch.uint8) * 8
    return code[..., 0::2] + code[..., 1::2] * 16, e.to(torch.uint8)


def _weights(kind, experts, n, k, gen):
    """Expert weights ~N(0, 0.02) in the storage of `kind`: (weight, scale or None)."""
    quant = {"fp8_block": _quant_block, "int8_channel": _quant_channel, "mxfp8": _quant_mxfp8,
             "mxfp4": _quant_mxfp4}.get(kind)
    dtype = torch.float16 if kind == "f16" else torch.bfloat16
    w = s = None
    step = max(1, min(experts, (1 << 28) // (n * k)))
    for e in range(0, experts, step):
        c = min(step, experts - e)
        part = torch.randn(c, n, k, generator=gen, device="cuda", dtype=dtype).mul_(0.02)
        q, qs = (part, None) if quant is None else quant(part)
        if w is None:
            w = torch.empty(experts, *q.shape[1:], dtype=q.dtype, device="cuda")
            s = None if qs is None else torch.empty(experts, *qs.shape[1:], dtype=qs.dtype,
                                                    device="cuda")
        w[e:e + c] = q
        if s is not None:
            s[e:e + c] = qs
    return w, s


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    m, h = case["M"], case["H"]
    if case["op"] == "dense":
        w, ws = _weights("fp8_block", 1, case["N"], h, gen)
        x = torch.randn(m, h // 128, 128, generator=gen, device="cuda")
        xs = x.abs().amax(-1) / 448.0
        return dict(case=case, x=(x / xs[..., None]).to(FP8).view(m, h), xs=xs, w=w[0], ws=ws[0])
    kind, experts, inter = case["kind"], case["E"], case["I"]
    local = experts // case.get("shards", 1)
    w1, s1 = _weights(kind, local, 2 * inter, h, gen)
    w2, s2 = _weights(kind, local, h, inter, gen)
    dtype = torch.float16 if kind == "f16" else torch.bfloat16
    x = torch.randn(m, h, generator=gen, device="cuda", dtype=dtype)
    logits = torch.randn(m, experts, generator=gen, device="cuda")
    kw = {}
    if kind == "fp8_block":
        kw = dict(use_fp8_w8a8=True, block_shape=[128, 128])
    elif kind == "int8_channel":
        kw = dict(use_int8_w8a8=True, per_channel_quant=True)
    elif kind == "mxfp8":
        kw = dict(use_mxfp8=True, block_shape=[1, 32])
    elif kind == "mxfp4":
        kw = dict(use_mxfp4_w4a8=True, use_ue8m0=True, block_shape=[1, 32])
    if s1 is not None:
        kw.update(w1_scale=s1, w2_scale=s2)
    if case.get("clamp"):   # biases and the clamped gate with a slope
        kw.update(b1=torch.randn(local, 2 * inter, generator=gen, device="cuda", dtype=dtype),
                  b2=torch.randn(local, h, generator=gen, device="cuda", dtype=dtype),
                  gemm1_alpha=1.702, gemm1_limit=7.0)
    if local != experts:    # this rank holds a contiguous run of experts
        first = (seed % case["shards"]) * local
        ids = torch.arange(experts, device="cuda", dtype=torch.int32) - first
        kw.update(expert_map=torch.where((ids >= 0) & (ids < local), ids, -1),
                  global_num_experts=experts)
    state = dict(case=case, x=x, w1=w1, w2=w2, kw=kw)
    if case["router"]:
        state["logits"] = logits
        return state
    scores = torch.softmax(logits, -1)
    order = scores
    if case.get("zipf"):    # experts of a token without replacement, p(e) ~ (rank + 1)^-zipf
        rank = torch.rand(experts, generator=gen, device="cuda").argsort().argsort() + 1
        noise = torch.rand(m, experts, generator=gen, device="cuda").clamp_(1e-7, 1 - 1e-7)
        order = -case["zipf"] * torch.log(rank.float()) - torch.log(-torch.log(noise))
    ids = order.topk(case["K"], -1).indices
    weights = scores.gather(1, ids)
    state.update(ids=ids.to(torch.int32), weights=weights / weights.sum(-1, keepdim=True))
    return state


def run(state):
    case = state["case"]
    if case["op"] == "dense":
        return gemm_a8w8_blockscale(state["x"], state["w"], state["xs"], state["ws"])
    if case["router"]:
        weights, ids = fused_topk(state["x"], state["logits"], case["K"], True)
    else:
        weights, ids = state["weights"], state["ids"]
    out = fused_experts(state["x"], state["w1"], state["w2"], weights, ids, **state["kw"])
    return (out, weights, ids) if case["router"] else out


# ---------------------------------------------------------------------------
# what a pass cannot do without, and how far two right answers may be apart
# ---------------------------------------------------------------------------
def work(case):
    m, h = case["M"], case["H"]
    if case["op"] == "dense":
        n = case["N"]
        return dict(flops=2.0 * m * n * h,
                    bytes=m * h + m * h / 32 + n * h + n * h / 4096 + 2.0 * m * n)
    experts, k, inter = case["E"], case["K"], case["I"]
    share = 1.0 / case.get("shards", 1)
    # expected number of experts that a batch touches
    if case.get("zipf"):
        p = [(e + 1.0) ** -case["zipf"] for e in range(experts)]
        touched = sum(1 - (1 - min(1.0, k * x / sum(p))) ** m for x in p)
    else:
        touched = experts * (1 - (1 - k / experts) ** m) * share
    per_weight = {"bf16": 2.0, "f16": 2.0, "fp8_block": 1 + 4 / 16384, "int8_channel": 1.0,
                  "mxfp8": 1 + 1 / 32, "mxfp4": 0.5 + 1 / 32}[case["kind"]]
    weights = touched * 3 * inter * h * per_weight
    routing = m * (4.0 * experts + 8 * k if case["router"] else 8.0 * k)
    return dict(flops=6.0 * m * k * share * inter * h, bytes=weights + 4.0 * m * h + routing)


def tolerance(case):
    """Measured: the same layer with its reductions in another order (hidden and intermediate
    columns permuted) is off by 9e-4 with bf16 experts, 1.7e-4 with biases and f16, 4e-4 with
    block-scaled, 3.3e-4 with microscaled ones (a sum that rounds the other way moves an
    activation by one bf16 or e4m3 step; single values by up to 0.04), 3e-5 in the dense GEMM.
    Per-channel int8 sums are exact, but its activation passes through bf16 like the others."""
    if case["op"] == "dense":
        return {"rel": 2e-4, "max": 0.03}
    if case["kind"] in ("bf16", "f16"):
        return {"rel": 4e-3, "max": 0.08}
    return {"rel": 2e-3, "max": 0.16}


# ---------------------------------------------------------------------------
# the same answers in 64 bits
# ---------------------------------------------------------------------------
def _exact_weight(kind, w, s):
    """One expert's weight [N, K] as the values its codes and scales stand for."""
    if kind in ("bf16", "f16"):
        return w.double()
    if kind == "fp8_block":
        return w.double() * s.double().repeat_interleave(128, 0).repeat_interleave(128, 1)
    if kind == "int8_channel":
        return w.double() * s.double()[:, None]
    if kind == "mxfp4":
        table = torch.tensor((0, .5, 1, 1.5, 2, 3, 4, 6), dtype=torch.float64, device=w.device)
        code = torch.stack((w & 15, w >> 4), -1).flatten(-2).long()
        w = table[code & 7] * torch.where(code & 8 != 0, -1.0, 1.0)
    return w.double() * torch.exp2(s.double() - 127).repeat_interleave(32, 1)


def _exact_rows(kind, v):
    """Activations [m, K] after the recipe's quantiser (which is part of what the layer computes)."""
    if kind in ("bf16", "f16"):
        return v
    group = {"fp8_block": 128, "int8_channel": v.shape[1], "mxfp8": 32, "mxfp4": 128}[kind]
    y = v.view(v.shape[0], -1, group)
    amax = y.abs().amax(-1, keepdim=True).clamp_min(1e-10)
    if kind == "int8_channel":
        s = amax / 127.0
        return ((y / s).round() * s).view(v.shape)
    s = amax / 448.0
    if kind.startswith("mx"):
        s = torch.exp2(torch.ceil(torch.log2(s)))
    return ((y / s).float().to(FP8).double() * s).view(v.shape)


def exact(case, seed):
    state = prepare(case, seed)
    x = state["x"]
    if case["op"] == "dense":
        xd = (x.double().view(case["M"], -1, 128) * state["xs"].double()[..., None]).flatten(1)
        return xd @ _exact_weight("fp8_block", state["w"], state["ws"]).t()
    kind, kw = case["kind"], state["kw"]
    if case["router"]:
        scores, ids = torch.softmax(state["logits"].double(), -1).topk(case["K"], -1)
        weights = scores / scores.sum(-1, keepdim=True)
    else:
        weights, ids = state["weights"].double(), state["ids"].long()
    if "expert_map" in kw:
        ids = kw["expert_map"].long()[ids]
    rows = _exact_rows(kind, x.double())
    out = torch.zeros_like(rows)
    for e in range(state["w1"].shape[0]):
        token, slot = (ids == e).nonzero(as_tuple=True)
        if not token.numel():
            continue
        s1, s2 = (kw[n][e] if n in kw else None for n in ("w1_scale", "w2_scale"))
        g = rows[token] @ _exact_weight(kind, state["w1"][e], s1).t()
        if case.get("clamp"):
            gate, up = (g + kw["b1"][e].double()).chunk(2, -1)
            gate, up = gate.clamp(max=7.0), up.clamp(-7.0, 7.0)
            act = gate * torch.sigmoid(1.702 * gate) * (up + 1)
        else:
            gate, up = g.chunk(2, -1)
            act = gate * torch.sigmoid(gate) * up
        y = _exact_rows(kind, act) @ _exact_weight(kind, state["w2"][e], s2).t()
        if case.get("clamp"):
            y = y + kw["b2"][e].double()
        out.index_add_(0, token, y * weights[token, slot][:, None])
    return (out, weights, None) if case["router"] else out
