"""Native-MXFP8 experts (`use_mxfp8=True`): e4m3 weights and activations with one E8M0
exponent byte per 32 consecutive K elements.

Reference semantics (boltops/fused_moe/triton/fused_moe.py:978-996,1079-1197 and the CPU
statement in test/fused_moe/test_fused_moe.py:1904-1931 of the reference project): activations
are quantised inside the layer per 1 x 32 group with scale 2^ceil(log2(amax/448)); GEMM1 is
rounded to the input dtype; the split gated activation and the second quantisation run in fp32
on that; GEMM2 and the router weights stay in fp32 until the sum over a token's routes; one cast
at the end.

How it runs here.  When both reduction lengths (hidden and intermediate size) are whole
128-wide K blocks, the two GEMMs use the tensor cores' block-scaled e4m3 instruction
(`BOLT_GEMM_MXFP8`): codes stay 8-bit, the exponent bytes are re-tiled once per call for the
activations (`bolt_mx_sf_layout`) and once per weight tensor (cached).  Other shapes rely on an
identity: an e4m3 value times a power of two is exactly representable in bf16 / fp16 and
products of two such values are exact in fp32, so the MX contraction equals a 16-bit GEMM over
the DEQUANTISED operands with fp32 accumulation; activations are then dequantised in the
quantiser kernel itself and the checkpoint weights decoded once (`bolt_mx_dequant_rows`,
cached), at 16-bit memory traffic.
"""
from __future__ import annotations

import weakref
from typing import Optional

import torch

from .. import _cabi
from . import ops


class _Stage:
    """Same per-stage CUDA-event bookkeeping as the main layer (off unless a timer is set)."""

    def __init__(self, name):
        self.name = name

    def __enter__(self):
        from . import layer
        self.t = layer.STAGE_TIMER
        self.start = self.t.begin() if self.t is not None else None

    def __exit__(self, *exc):
        if self.t is not None:
            self.t.end(self.name, self.start)
        return False

_decoded = {}     # (data_ptr, scale data_ptr, shape, dtype) -> (weakrefs of the sources, decoded tensor)


def _decode_weights(w: torch.Tensor, scale: torch.Tensor, dtype: torch.dtype) -> torch.Tensor:
    """Checkpoint weights [E, N, K] e4m3 + E8M0 bytes [E, N, K/32] -> [E, N, K] in `dtype`.
    Decoded once per (weight, scale) pair and kept while both source tensors are alive and
    unmodified (their version counters are part of the key)."""
    key = (w.data_ptr(), scale.data_ptr(), tuple(w.shape), dtype, w._version, scale._version)
    hit = _decoded.get(key)
    if hit is not None and hit[0]() is w and hit[1]() is scale:
        return hit[2]
    for k in [k for k, v in _decoded.items() if v[0]() is None or v[1]() is None]:
        del _decoded[k]
    out = ops.mx_dequant_rows(w.contiguous(), scale.contiguous(), dtype)
    _decoded[key] = (weakref.ref(w), weakref.ref(scale), out)
    return out


def _tile_weight_scales(w: torch.Tensor, scale: torch.Tensor, gated: bool = False) -> torch.Tensor:
    """E8M0 bytes [E, N, K/32] -> the 512-byte tiles the block-scaled GEMM kind reads
    ([E * ceil(N/128), K/128, 512]); done once per scale tensor, like the decoding above.
    gated: rows in the order the gated kernel loads the weight rows of a tile
    ([gate n0.., up n0.., gate n0+64.., up n0+64..], 64 rows each, n0 = 128 * column tile)."""
    key = ("sf", scale.data_ptr(), tuple(scale.shape), scale._version, gated)
    hit = _decoded.get(key)
    if hit is not None and hit[0]() is scale:
        return hit[2]
    for k in [k for k, v in _decoded.items() if v[0]() is None or v[1]() is None]:
        del _decoded[k]
    e, n, sf_cols = scale.shape
    if gated:
        half = n // 2
        assert half % 128 == 0 and e * n < (1 << 24)
        j = torch.arange(256, device=scale.device)
        # tile row j -> weight row: 64-row pieces gate, up, gate + 64, up + 64
        piece = j // 64
        within = (piece % 2) * half + (piece // 2) * 64 + j % 64
        rows = (torch.arange(half // 128, device=scale.device)[:, None] * 128 + within[None, :])
        idx = (torch.arange(e, device=scale.device)[:, None, None] * n + rows[None]).to(torch.int32)
        out = ops.mx_sf_layout(scale.reshape(e * n, sf_cols), idx.numel(), idx.reshape(-1).contiguous())
        _decoded[key] = (weakref.ref(scale), weakref.ref(scale), out)
        return out
    n_pad = (n + 127) // 128 * 128
    src = scale
    if n_pad != n:
        src = torch.zeros((e, n_pad, sf_cols), dtype=torch.uint8, device=scale.device)
        src[:, :n] = scale
    out = ops.mx_sf_layout(src.reshape(e * n_pad, sf_cols), e * n_pad)
    _decoded[key] = (weakref.ref(scale), weakref.ref(scale), out)
    return out


def validate(hidden_states, w1, w2, w1_scale, w2_scale, a1_scale, a2_scale, b1, b2,
             apply_router_weight_on_input, output_dtype, block_shape, activation, is_gated,
             inplace, no_combine) -> None:
    """The reference's argument checks for the native path, same order, types and messages."""
    if hidden_states.dtype not in (torch.bfloat16, torch.float16):
        raise ValueError("native MXFP8 requires BF16/FP16 hidden_states")
    if a1_scale is not None or a2_scale is not None:
        raise ValueError("native MXFP8 quantizes activations internally; "
                         "a1_scale/a2_scale must be None")
    if b1 is not None or b2 is not None or apply_router_weight_on_input:
        raise ValueError("native MXFP8 does not support bias or input routing weights")
    if output_dtype is not None and output_dtype != hidden_states.dtype:
        raise ValueError("native MXFP8 output_dtype must match hidden_states.dtype")
    if w1.dtype != torch.float8_e4m3fn or w2.dtype != torch.float8_e4m3fn:
        raise ValueError("MXFP8 weights must be E4M3; FNUZ is not supported")
    if block_shape is not None and tuple(block_shape) != (1, 32):
        raise ValueError("native MXFP8 requires weight block_shape=[1,32]")
    for scale in (w1_scale, w2_scale):
        if scale is None or scale.dtype != torch.uint8:
            raise ValueError("native MXFP8 requires uint8 E8M0 weight scales")
    if not is_gated or activation not in ("silu", "swigluoai"):
        raise ValueError("MXFP8 requires gated ('silu', 'swigluoai')")
    if no_combine:
        assert not inplace, "no_combine + inplace is not supported"


def fused_experts_mxfp8(hidden_states, w1, w2, topk_weights, topk_ids, *, w1_scale, w2_scale,
                        activation: str, inplace: bool, no_combine: bool,
                        global_num_experts: int, expert_map: Optional[torch.Tensor],
                        routed_scaling_factor: float, gemm1_alpha, gemm1_beta, gemm1_limit,
                        chunk: int) -> torch.Tensor:
    if not hidden_states.is_cuda:
        raise ValueError("boltops_b200 kernels need CUDA tensors (there is no CPU path)")
    assert hidden_states.shape[1] == w1.shape[2], "Hidden size mismatch"
    assert topk_weights.shape == topk_ids.shape, "topk shape mismatch"
    assert hidden_states.is_contiguous(), "Hidden_states must be contiguous"
    dtype = hidden_states.dtype
    dev = hidden_states.device
    num_tokens, hidden = hidden_states.shape
    e_local, n1, _ = w1.shape
    inter = n1 // 2
    model_dim = w2.shape[1]
    topk = topk_ids.shape[1]
    assert hidden % 32 == 0 and inter % 32 == 0, "MXFP8 needs K dimensions divisible by 32"
    assert tuple(w1_scale.shape) == (e_local, n1, hidden // 32), "w1_scale shape"
    assert tuple(w2_scale.shape) == (e_local, model_dim, inter // 32), "w2_scale shape"
    if expert_map is None:
        global_num_experts = e_local          # appended shared experts included, as the reference
    elif global_num_experts == -1:
        global_num_experts = expert_map.numel()
    oai = activation == "swigluoai"
    alpha = (1.702 if oai else 1.0) if gemm1_alpha is None else gemm1_alpha
    beta = (1.0 if oai else 0.0) if gemm1_beta is None else gemm1_beta
    # Both reduction lengths in whole 128-wide K blocks: the tensor core applies the E8M0 scales
    # itself (BOLT_GEMM_MXFP8) and the weights stay in 8 bits.  Otherwise the operands are
    # dequantised (exactly) and the 16-bit kind computes the same contraction.
    native = hidden % 128 == 0 and inter % 128 == 0
    from .layer import _use_gather
    if native:
        kind = _cabi.GEMM_MXFP8
        w1 = w1 if w1.is_contiguous() else w1.contiguous()
        w2 = w2 if w2.is_contiguous() else w2.contiguous()
        sfb1 = _tile_weight_scales(w1, w1_scale, gated=True)
        sfb2 = _tile_weight_scales(w2, w2_scale)
    else:
        kind = _cabi.GEMM_BF16 if dtype == torch.bfloat16 else _cabi.GEMM_F16
        w1_d = _decode_weights(w1, w1_scale, dtype)
        w2_d = _decode_weights(w2, w2_scale, dtype)
    expert_mask = (expert_map >= 0).to(torch.int32) if expert_map is not None else None
    if topk_ids.dtype != torch.int32:
        topk_ids = topk_ids.to(torch.int32)
    topk_weights = topk_weights.to(torch.float32)

    if no_combine:
        out = torch.empty((num_tokens, topk, model_dim), device=dev, dtype=dtype)
    elif inplace:
        out = hidden_states
    else:
        out = torch.empty((num_tokens, model_dim), device=dev, dtype=dtype)
    for begin in range(0, num_tokens, chunk):
        end = min(begin + chunk, num_tokens)
        m = end - begin
        ids = topk_ids[begin:end].contiguous()
        wts = topk_weights[begin:end].contiguous()
        route_pos = torch.empty((m, topk), device=dev, dtype=torch.int32)
        with _Stage("sort"):
            sorted_ids, sorted_w, expert_ids, num_valid, _, _ = ops.moe_sorting_ck(
                ids, wts, global_num_experts, None, None, ops.SORT_UNIT, expert_mask,
                alloc_moe_buf=False, route_pos=route_pos)
        if expert_map is not None:
            expert_ids = ops.relabel_tiles(expert_ids, expert_map)
        cap = sorted_ids.shape[0]
        common = dict(kind=kind, sorted_expert_ids=expert_ids, num_valid=num_valid,
                      sorted_ids=sorted_ids, sorted_weights=sorted_w, num_tokens=m, topk=topk)
        if native:
            # A1: codes + exponent bytes once per token; codes gathered into sorted rows, or by GEMM1
            # itself while those rows would be mostly padding (layer._use_gather); bytes gathered
            # straight into the tiled layout
            in_gemm = _use_gather(m * topk, global_num_experts)
            with _Stage("quant_a1"):
                x_q, x_s, _ = ops.mx_quant_rows(hidden_states[begin:end])
            with _Stage("gather"):
                a1 = x_q if in_gemm else ops.gather_rows(x_q, sorted_ids, num_valid, cap)[0]
                sfa = ops.mx_sf_layout(x_s, cap, sorted_ids, num_valid)
            # GEMM1 with the rounding to the input dtype, the split gated activation (fp32) and
            # the second quantisation in its epilogue: 32 outputs of a thread are one MX group
            act = torch.empty((cap, inter), device=dev, dtype=torch.float8_e4m3fn)
            act_s = torch.empty((cap, inter // 32), device=dev, dtype=torch.uint8)
            with _Stage("gemm1"):
                ops.grouped_gemm(epilogue=_cabi.EPI_SILU_MUL_QUANT, a=a1, a_gather=in_gemm, b=w1, c=act,
                                 a_scale=sfa, b_scale=sfb1, c_scale=act_s,
                                 c_scale_ld=inter // 32, mid_dtype=dtype, act_alpha=alpha,
                                 act_beta=beta, act_limit=gemm1_limit, **common)
            with _Stage("scales_a2"):
                gemm2 = dict(a=act, b=w2, a_scale=ops.mx_sf_layout(act_s, cap), b_scale=sfb2)
        else:
            _, _, x_d = ops.mx_quant_rows(hidden_states[begin:end], want_codes=False,
                                          deq_dtype=dtype)
            a_sorted, _ = ops.gather_rows(x_d, sorted_ids, num_valid, cap)
            g1 = torch.empty((cap, n1), device=dev, dtype=dtype)
            ops.grouped_gemm(epilogue=_cabi.EPI_STORE, a=a_sorted, b=w1_d, c=g1, **common)
            _, _, act = ops.mx_quant_rows(g1, gated=True, alpha=alpha, beta=beta,
                                          limit=gemm1_limit, want_codes=False, deq_dtype=dtype)
            gemm2 = dict(a=act, b=w2_d)
        # GEMM2 in fp32 with the router weight, then the fp32 sum over the routes
        if no_combine:
            c3 = torch.zeros((m * topk, model_dim), device=dev, dtype=torch.float32) \
                if expert_map is not None else \
                torch.empty((m * topk, model_dim), device=dev, dtype=torch.float32)
            ops.grouped_gemm(epilogue=_cabi.EPI_STORE, c=c3, scatter=True,
                             mul_routed_weight=False, **gemm2, **common)
            out[begin:end].copy_(c3.view(m, topk, model_dim))
        else:
            c_sorted = torch.empty((cap, model_dim), device=dev, dtype=torch.float32)
            with _Stage("gemm2"):
                ops.grouped_gemm(epilogue=_cabi.EPI_STORE, c=c_sorted, scatter=False,
                                 mul_routed_weight=True, **gemm2, **common)
            with _Stage("combine"):
                ops.gather_sum(c_sorted, route_pos, out[begin:end], routed_scaling_factor)
    return out
