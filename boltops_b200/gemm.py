"""Dense block-scaled GEMM on the grouped-GEMM kernel (one "expert").

Same call surface as the reference's ``gemm_a8w8_blockscale``
(boltops/gemm/gemm_a8w8_blockscale.py:10-70 in the reference project) and
``w8a8_triton_block_scaled_mm`` for the recipe the fused-MoE path uses: e4m3 or int8
operands, A scales per row and 128 K elements, B scales per 128x128 block.  It is the
op a DeepSeek-style layer calls next to ``fused_experts`` (shared experts, dense layers).
"""
from __future__ import annotations

from typing import Optional, Sequence

import torch

from . import _cabi
from .fused_moe import ops


def gemm_a8w8_blockscale(x: torch.Tensor, w: torch.Tensor, x_scale: torch.Tensor,
                         w_scale: torch.Tensor, dtype: Optional[torch.dtype] = torch.bfloat16,
                         out: Optional[torch.Tensor] = None, config=None, backend=None):
    """``y[m, n] = sum_kb (x[m, kb] . w[n, kb]) * x_scale[m, kb] * w_scale[n//128, kb]``.

    x [M, K] and w [N, K] e4m3 or int8 (same dtype), x_scale [M, K/128], w_scale
    [N/128, K/128] floating point; K and N multiples of 128.  w and w_scale lie on x's device;
    x_scale and ``out`` may lie elsewhere and are copied.  ``config`` / ``backend`` are accepted
    for signature compatibility and ignored (one kernel, one schedule)."""
    if dtype is None:
        dtype = torch.bfloat16
    if not x.is_cuda:
        raise ValueError("boltops_b200 kernels need CUDA tensors (there is no CPU path)")
    if x.dtype != w.dtype or x.dtype not in (torch.float8_e4m3fn, torch.int8):
        raise TypeError("x and w must both be float8_e4m3fn or int8")
    m, k = x.shape
    n = w.shape[0]
    if w.shape[1] != k or k % 128 or n % 128:
        raise NotImplementedError("K and N must be multiples of 128 (1x128 / 128x128 scale recipe)")
    if tuple(x_scale.shape) != (m, k // 128) or tuple(w_scale.shape) != (n // 128, k // 128):
        raise ValueError("scale shapes do not match the 1x128 / 128x128 recipe")
    kind = _cabi.GEMM_FP8_BLOCK if x.dtype == torch.float8_e4m3fn else _cabi.GEMM_INT8_BLOCK
    dev = x.device
    # the kernels take addresses: none of another device may reach them
    for name, t in (("w", w), ("w_scale", w_scale)):
        if t.device != dev:
            raise ValueError(f"{name} is on {t.device}, x on {dev}")
    if out is not None:
        assert out.shape == (m, n) and out.dtype == dtype and out.is_contiguous()
    elsewhere = out is not None and out.device != dev     # the result is copied there
    c = out if out is not None and not elsewhere else torch.empty((m, n), dtype=dtype, device=dev)
    if m == 0:
        return out if elsewhere else c
    # Two launches: the scales to group-major order (with the one "expert"'s tile labels), the GEMM.
    # Rows that only pad the last row tile exist nowhere: the tensor map reads them as zeros and
    # nothing is stored for them.
    x, w = x.contiguous(), w.contiguous()
    if x.data_ptr() % 16:
        x = x.clone()       # the tensor map needs a 16-byte aligned base
    x_scale = x_scale.to(device=dev, dtype=torch.float32).contiguous()
    w_scale = w_scale.float().contiguous()
    cap = ops.ceil_to(m, 128)
    groups, tiles = k // 128, cap // 128
    ws = torch.empty(groups * cap + tiles + 1, dtype=torch.float32, device=dev)
    scale_t = ws.data_ptr()
    tile_ids = scale_t + 4 * groups * cap
    num_rows = tile_ids + 4 * tiles
    args = _cabi.GemmArgs()
    args.kind, args.epilogue = kind, _cabi.EPI_STORE
    args.capacity, args.n, args.k, args.num_experts = cap, n, k, 1
    args.a, args.b, args.c = x.data_ptr(), w.data_ptr(), c.data_ptr()
    args.dense_rows = m
    args.a_scale, args.a_scale_ld, args.b_scale = scale_t, cap, w_scale.data_ptr()
    args.c_dtype = args.mid_dtype = _cabi.dtype_code(dtype)
    args.c_ld, args.topk = n, 1
    args.sorted_expert_ids, args.num_valid_ids = tile_ids, num_rows
    args.status = ops.device_status(dev).data_ptr()
    args.sm_count = ops.gemm_sm_count(dev)
    lib = _cabi.load()
    stream = _cabi.stream_of(x)
    with _cabi.on_device(dev):
        _cabi.check(lib.bolt_dense_prep(x_scale.data_ptr(), m, groups, scale_t, cap, tile_ids,
                                        num_rows, stream))
        _cabi.check(lib.bolt_grouped_gemm(args, stream))
    ops._count(2)
    if elsewhere:
        return out.copy_(c)
    return c


def w8a8_block_scaled_mm(A: torch.Tensor, B: torch.Tensor, As: torch.Tensor, Bs: torch.Tensor,
                         block_size: Sequence[int], output_dtype: torch.dtype = torch.float16):
    """vLLM/SGLang-style name of the same operation (B is [N, K], ``block_size`` [128, 128])."""
    if list(block_size) != [128, 128]:
        raise NotImplementedError("only block_size [128, 128] is built in boltops_b200")
    return gemm_a8w8_blockscale(A, B, As, Bs, dtype=output_dtype)


w8a8_triton_block_scaled_mm = w8a8_block_scaled_mm
w8a8_block_int8_matmul = w8a8_block_scaled_mm
