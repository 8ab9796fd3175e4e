"""The weight-streaming schedule of the grouped GEMM (experts with few rows) against the row-tile
schedule, which runs the same tensor-core arithmetic in the same order: equal bit for bit."""
import pytest
import torch

from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu

FP8 = torch.float8_e4m3fn


def _rows(counts, topk=2):
    """Routing in which expert e gets exactly counts[e] tokens (its slot-0 routes); the slot-1 routes
    go nowhere (-1)."""
    ids = torch.cat([torch.full((c,), e, dtype=torch.int32) for e, c in enumerate(counts)])
    ids = ids[torch.randperm(len(ids), generator=torch.Generator().manual_seed(5))]
    return torch.stack([ids, torch.full_like(ids, -1)], 1).contiguous()


# rows per expert around the column counts of the instruction (16, 32, 64, 128), the passes of a
# row tile and the tile itself; none at all; a tile and a remainder
COUNTS = {
    "edges": [1, 15, 16, 17, 31, 32, 33, 0],
    "wide": [63, 64, 65, 127, 128, 129, 0, 3],
    "one": [0, 0, 1, 0, 0, 0, 0, 0],
    "twice": [0, 0, 0, 0, 0, 40, 2, 1],   # both slots of every token: more rows than half an item holds
}


@pytest.mark.parametrize("counts", sorted(COUNTS))
@pytest.mark.parametrize("kind,hidden,inter", [
    ("bf16", 512, 256), ("f16", 192, 320),          # 320: a last column tile that is part empty
    ("fp8_block", 640, 384), ("int8_block", 256, 128),
    ("fp8_channel", 384, 256), ("int8_channel", 128, 384),
])
@pytest.mark.parametrize("extra", ["plain", "bias", "clamp", "no_combine", "f32", "map"])
def test_stream_equals_row_tiles(monkeypatch, kind, hidden, inter, counts, extra):
    from boltops_b200.fused_moe import fused_experts, ops
    ids = _rows(COUNTS[counts])
    if counts == "twice":
        ids[:, 1] = ids[:, 0]
    m, e = ids.shape[0], 8
    g = torch.Generator().manual_seed(11)
    dt = torch.float16 if kind == "f16" else torch.bfloat16
    x = torch.randn(m, hidden, generator=g).to(dt)
    m1 = torch.randn(e, 2 * inter, hidden, generator=g) * 0.05
    m2 = torch.randn(e, hidden, inter, generator=g) * 0.05
    kw = {}
    if kind in ("bf16", "f16"):
        w1, w2 = m1.to(dt), m2.to(dt)
    elif kind.endswith("block"):
        fp8 = kind.startswith("fp8")
        w1, s1 = O.quantize_weight_block_fp8(m1)
        w2, s2 = O.quantize_weight_block_fp8(m2)
        if not fp8:     # the same scales with integer codes
            w1, w2 = ((w.float() * (127.0 / 448.0)).round().to(torch.int8) for w in (w1, w2))
        kw = dict(block_shape=[128, 128], w1_scale=s1.cuda(), w2_scale=s2.cuda())
        kw["use_fp8_w8a8" if fp8 else "use_int8_w8a8"] = True
    else:
        w1, s1 = O.quantize_weight_channel_int8(m1)
        w2, s2 = O.quantize_weight_channel_int8(m2)
        kw = dict(per_channel_quant=True, w1_scale=s1.cuda(), w2_scale=s2.cuda())
        if kind == "fp8_channel":
            w1, w2 = w1.float().to(FP8), w2.float().to(FP8)
            kw["use_fp8_w8a8"] = True
        else:
            kw["use_int8_w8a8"] = True
    if extra in ("bias", "clamp"):
        kw.update(b1=torch.randn(e, 2 * inter, generator=g).to(dt).cuda(),
                  b2=torch.randn(e, hidden, generator=g).to(dt).cuda())
    if extra == "clamp":
        kw.update(gemm1_alpha=1.702, gemm1_limit=7.0)
    if extra == "no_combine":
        kw.update(no_combine=True)
    if extra == "f32":
        if kind in ("bf16", "f16"):
            pytest.skip("16-bit rows between the GEMMs")
        kw.update(output_dtype=torch.float32)
    w1, w2 = w1.cuda(), w2.cuda()
    if extra == "map":      # the upper half of the experts lives here
        kw.update(expert_map=torch.tensor([-1] * 4 + list(range(4)), dtype=torch.int32).cuda(),
                  global_num_experts=e)
        w1, w2 = w1[4:].contiguous(), w2[4:].contiguous()
        for name in ("w1_scale", "w2_scale"):
            if name in kw:
                kw[name] = kw[name][4:].contiguous()
    wts = torch.rand(m, 2, generator=g)
    outs = {}
    for sched in ("tiles", "stream"):
        monkeypatch.setenv("BOLTOPS_B200_GEMM_SCHEDULE", sched)
        out = fused_experts(x.cuda(), w1, w2, wts.cuda(), ids.cuda(), **kw)
        if extra == "no_combine":
            out = out[:, 0]     # the slot of a route that goes nowhere is not written
        torch.cuda.synchronize()
        ops.check_device_status(out.device)
        outs[sched] = out.cpu()
    assert torch.isfinite(outs["tiles"]).all()
    assert torch.equal(outs["stream"], outs["tiles"])


def test_stream_refuses_what_it_has_no_form_for():
    from boltops_b200 import _cabi
    from boltops_b200.fused_moe import ops
    x = torch.zeros(128, 72, dtype=torch.bfloat16, device="cuda")   # 144 bytes: no whole K block
    c = torch.zeros(128, 64, dtype=torch.bfloat16, device="cuda")
    one = torch.zeros(1, dtype=torch.int32, device="cuda")
    with pytest.raises(_cabi.BoltError, match="streaming schedule"):
        ops.grouped_gemm(kind=_cabi.GEMM_BF16, epilogue=_cabi.EPI_STORE, a=x,
                         b=torch.zeros(1, 64, 72, dtype=torch.bfloat16, device="cuda"), c=c,
                         sorted_expert_ids=one, num_valid=one, sorted_ids=one.repeat(128),
                         num_tokens=1, stream=True)


def _quantised(kind, e, hidden, inter, g):
    """Weights and keyword arguments of a layer of one kind."""
    m1 = torch.randn(e, 2 * inter, hidden, generator=g) * 0.05
    m2 = torch.randn(e, hidden, inter, generator=g) * 0.05
    if kind == "bf16":
        return m1.bfloat16().cuda(), m2.bfloat16().cuda(), {}
    if kind == "fp8_block":
        quant, kw = O.quantize_weight_block_fp8, dict(use_fp8_w8a8=True, block_shape=[128, 128])
    else:
        quant, kw = O.quantize_weight_channel_int8, dict(use_int8_w8a8=True, per_channel_quant=True)
    (w1, s1), (w2, s2) = quant(m1), quant(m2)
    return w1.cuda(), w2.cuda(), dict(kw, w1_scale=s1.cuda(), w2_scale=s2.cuda())


@pytest.mark.parametrize("kind", ["bf16", "fp8_block", "int8_channel"])
@pytest.mark.parametrize("extra", ["input_weight", "ue8m0", "not_finite"])
def test_stream_options_equal_row_tiles(monkeypatch, kind, extra):
    """Router weight on the input (before the gate), power-of-two scales, and rows of NaN and
    infinity, which stay in their own rows."""
    from boltops_b200.fused_moe import fused_experts, ops
    if extra == "ue8m0" and kind != "fp8_block":
        pytest.skip("power-of-two scales belong to the block-scaled kind")
    hidden, inter, e = 512, 256, 8
    g = torch.Generator().manual_seed(21)
    ids = _rows(COUNTS["edges"])
    m = ids.shape[0]
    x = torch.randn(m, hidden, generator=g).bfloat16()
    w1, w2, kw = _quantised(kind, e, hidden, inter, g)
    wts = torch.rand(m, 2, generator=g)
    bad = torch.zeros(m, dtype=torch.bool)
    if extra == "input_weight":
        kw["apply_router_weight_on_input"] = True
    elif extra == "ue8m0":
        kw["use_ue8m0"] = True
    else:
        bad[::7] = True
        x[::14, 3] = float("nan")
        x[7::14, 5] = float("inf")
    outs = []
    for sched in ("tiles", "stream"):
        monkeypatch.setenv("BOLTOPS_B200_GEMM_SCHEDULE", sched)
        out = fused_experts(x.cuda(), w1, w2, wts.cuda(), ids.cuda(), **kw)
        ops.check_device_status(out.device)
        outs.append(out.cpu())
    assert torch.isfinite(outs[0][~bad]).all() and torch.equal(outs[0][~bad], outs[1][~bad])
    assert torch.equal(outs[0].isnan(), outs[1].isnan())
    assert torch.equal(outs[0].nan_to_num(), outs[1].nan_to_num())


@pytest.mark.parametrize("counts", ["edges", "wide"])
@pytest.mark.parametrize("pitch", [0, 3])               # 3: rows of the result on no 16-byte grid
@pytest.mark.parametrize("token_scales", [False, True])
@pytest.mark.parametrize("c_dtype", [torch.bfloat16, torch.float32])
def test_stream_scales_by_token_and_any_row_pitch(monkeypatch, c_dtype, token_scales, pitch, counts):
    """Row scales of the per-channel kinds in token order or in sorted order, under both schedules,
    and results stored column by column: equal bit for bit, nothing written between the rows."""
    from boltops_b200 import _cabi
    from boltops_b200.fused_moe import ops
    lib = _cabi.load()

    class Lib:
        def __getattr__(self, name):
            return getattr(lib, name)

        def bolt_grouped_gemm(self, args, stream):
            args._obj.a_scale_token_order = int(token_scales)
            return lib.bolt_grouped_gemm(args, stream)

    ids = _rows(COUNTS[counts])
    m, e, n, k = ids.shape[0], 8, 328, 256
    g = torch.Generator().manual_seed(3)
    wts = torch.rand(m, 2, generator=g).cuda()
    sorted_ids, sorted_w, expert_ids, num_valid = ops.moe_sorting_ck(
        ids.cuda(), wts, e, None, None, 128, None, alloc_moe_buf=False)[:4]
    cap = sorted_ids.shape[0]
    x = torch.randint(-127, 128, (m, k), generator=g, dtype=torch.int8).cuda()
    w = torch.randint(-127, 128, (e, n, k), generator=g, dtype=torch.int8).cuda()
    by_token, b_s = torch.rand(m, generator=g).cuda(), torch.rand(e, n, generator=g).cuda()
    _, by_row = ops.gather_rows(x, sorted_ids, num_valid, cap, by_token[:, None])
    live = (sorted_ids & 0xFFFFFF) < m
    live[int(num_valid):] = False
    outs = []
    with monkeypatch.context() as patch:
        patch.setattr(_cabi, "load", lambda: Lib())
        for stream in (False, True):
            buf = torch.full((cap, n + pitch), -7.0, dtype=c_dtype, device="cuda")
            ops.grouped_gemm(kind=_cabi.GEMM_INT8_CHANNEL, epilogue=_cabi.EPI_STORE, a=x, b=w,
                             c=buf[:, :n], sorted_expert_ids=expert_ids, num_valid=num_valid,
                             a_scale=by_token if token_scales else by_row.reshape(-1), a_scale_ld=cap,
                             b_scale=b_s, num_tokens=m, topk=2, mul_routed_weight=True,
                             sorted_ids=sorted_ids, sorted_weights=sorted_w, a_gather=True, stream=stream)
            assert (buf[:, n:] == -7.0).all()
            outs.append(buf[live, :n].cpu())
    ops.check_device_status(x.device)
    token = (sorted_ids[live] & 0xFFFFFF).long().cpu()
    expert = expert_ids.repeat_interleave(128)[:cap][live].long().cpu()
    want = torch.einsum("rk,rnk->rn", x.cpu().double()[token], w.cpu().double()[expert])
    want = want * by_token.cpu().double()[token][:, None] * b_s.cpu().double()[expert]
    want = want * sorted_w[live].cpu().double()[:, None]
    # The integer sums are exact; three products in 32 bits (2^-24 each) and, for bf16 with its eight
    # significant bits, a rounding by half a unit in the last place (2^-8 of the value at most)
    rel = 4 * 2.0 ** -24 + (2.0 ** -8 if c_dtype == torch.bfloat16 else 0.0)
    assert ((outs[0].double() - want).abs() <= rel * want.abs() + 1e-30).all()
    assert torch.equal(outs[0], outs[1])
