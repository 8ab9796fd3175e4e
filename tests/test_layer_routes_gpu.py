"""Routes through the layer that depend on sizes, against the routes they replace."""
import pytest
import torch

from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [257, 300])        # just above 64 routes per expert / more than a tile
@pytest.mark.parametrize("hidden", [512, 2064])  # 2064: a reduction tail of 16 bytes
@pytest.mark.parametrize("bias", [False, True])
def test_per_channel_rows_gathered_by_the_gemm(monkeypatch, m, hidden, bias):
    """From 64 routes per expert on GEMM 1 of the per-channel kinds reads codes and scales in token
    order; the kernel-by-kernel orchestration still places sorted rows.  Equal bit for bit."""
    from boltops_b200.fused_moe import fused_experts, layer
    e, topk, inter = 8, 2, 256
    g = torch.Generator().manual_seed(3)
    x = torch.randn(m, hidden, generator=g).bfloat16().cuda()
    w1, s1 = O.quantize_weight_channel_int8(torch.randn(e, 2 * inter, hidden, generator=g) * 0.05)
    w2, s2 = O.quantize_weight_channel_int8(torch.randn(e, hidden, inter, generator=g) * 0.05)
    wts, ids = O.make_routing(m, e, topk, 9)
    ids[3, 1] = -1
    kw = dict(use_int8_w8a8=True, per_channel_quant=True, w1_scale=s1.cuda(), w2_scale=s2.cuda())
    if bias:
        kw.update(b1=torch.randn(e, 2 * inter, generator=g).bfloat16().cuda(),
                  b2=torch.randn(e, hidden, generator=g).bfloat16().cuda())
    args = (x, w1.cuda(), w2.cuda(), wts.cuda(), ids.cuda())
    one = fused_experts(*args, **kw)
    monkeypatch.setattr(layer, "_ONE_CALL", False)
    steps = fused_experts(*args, **kw)
    assert torch.equal(one.cpu(), steps.cpu())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("m", [1, 31, 127, 128, 129, 300])
@pytest.mark.parametrize("n,k", [(128, 128), (384, 4224)])    # 4224: 33 scale groups
def test_dense_rows_end_inside_a_tile(dtype, m, n, k):
    """The dense GEMM reads no row past the last and writes none: the result of M rows equals the
    first M rows of the result of a whole number of tiles, bit for bit, and lies in a guarded buffer."""
    from boltops_b200.gemm import gemm_a8w8_blockscale
    g = torch.Generator().manual_seed(m)
    full = (m + 127) // 128 * 128
    x = (torch.randn(full, k, generator=g) * 50).clamp(-448, 448).to(torch.float8_e4m3fn).cuda()
    w = (torch.randn(n, k, generator=g) * 50).clamp(-448, 448).to(torch.float8_e4m3fn).cuda()
    xs = (torch.rand(full, k // 128, generator=g) + 0.5).cuda()
    ws = (torch.rand(n // 128, k // 128, generator=g) + 0.5).cuda()
    whole = gemm_a8w8_blockscale(x, w, xs, ws, dtype=dtype)
    buf = torch.full((full + 64, n), -7.0, dtype=dtype, device="cuda")
    out = gemm_a8w8_blockscale(x[:m], w, xs[:m], ws, dtype=dtype, out=buf[:m])
    assert torch.equal(out.cpu(), whole[:m].cpu())
    assert (buf[m:] == -7.0).all()
    some = gemm_a8w8_blockscale(x[:m], w, xs[:m].double(), ws, dtype=dtype)   # any floating scale type
    assert torch.equal(some.cpu(), out.cpu())


def test_dense_operands_off_the_device_or_the_16_byte_grid():
    """Row scales and the result may lie in host memory, x and the result at any address."""
    from boltops_b200.gemm import gemm_a8w8_blockscale
    m, n, k = 130, 128, 256
    g = torch.Generator().manual_seed(2)
    x = torch.randint(-127, 128, (m, k), generator=g, dtype=torch.int8)
    w = torch.randint(-127, 128, (n, k), generator=g, dtype=torch.int8).cuda()
    xs, ws = torch.rand(m, k // 128, generator=g), torch.rand(n // 128, k // 128, generator=g).cuda()
    want = gemm_a8w8_blockscale(x.cuda(), w, xs.cuda(), ws)
    assert torch.equal(gemm_a8w8_blockscale(x.cuda(), w, xs, ws), want)
    host = torch.zeros(m, n, dtype=torch.bfloat16)
    assert gemm_a8w8_blockscale(x.cuda(), w, xs.cuda(), ws, out=host) is host
    assert torch.equal(host, want.cpu())
    odd = torch.zeros(m * k + 1, dtype=torch.int8, device="cuda")[1:].view(m, k)
    odd.copy_(x)
    assert torch.equal(gemm_a8w8_blockscale(odd, w, xs.cuda(), ws), want)
    for dtype in (torch.bfloat16, torch.float32):
        buf = torch.zeros(m * n + 1, dtype=dtype, device="cuda")
        out = buf[1:].view(m, n)
        gemm_a8w8_blockscale(x.cuda(), w, xs.cuda(), ws, dtype=dtype, out=out)
        assert torch.equal(out, gemm_a8w8_blockscale(x.cuda(), w, xs.cuda(), ws, dtype=dtype))
    for moved in (dict(w=w.cpu()), dict(w_scale=ws.cpu())):
        with pytest.raises(ValueError, match="x on cuda"):
            gemm_a8w8_blockscale(x.cuda(), moved.get("w", w), xs.cuda(), moved.get("w_scale", ws))


@pytest.mark.parametrize("kind", ["mxfp8", "mxfp4"])
@pytest.mark.parametrize("m", [1, 33, 300])          # tiles of one row, of a few, full and a remainder
@pytest.mark.parametrize("mapped", [False, True])
def test_mx_rows_gathered_by_the_gemm(monkeypatch, kind, m, mapped):
    """GEMM 1 of the MX kinds reading its codes in token order or from sorted rows: the same bytes."""
    from boltops_b200.fused_moe import fused_experts, layer, ops
    e, topk, hidden, inter = 8, 2, 384, 256
    g = torch.Generator().manual_seed(m)
    x = torch.randn(m, hidden, generator=g).bfloat16().cuda()
    wts, ids = O.make_routing(m, e, topk, 9)
    if mapped:
        ids[0, 1] = -1

    def weight(n, k):
        scale = torch.randint(118, 124, (e, n, k // 32), dtype=torch.uint8, generator=g).cuda()
        if kind == "mxfp8":
            return (torch.randn(e, n, k, generator=g) * 2).to(torch.float8_e4m3fn).cuda(), scale
        return torch.randint(0, 256, (e, n, k // 2), dtype=torch.uint8, generator=g).cuda(), scale

    (w1, s1), (w2, s2) = weight(2 * inter, hidden), weight(hidden, inter)
    kw = dict(use_mxfp8=True) if kind == "mxfp8" else dict(use_mxfp4_w4a8=True, use_ue8m0=True)
    if mapped:      # the upper half of the experts lives here
        w1, s1, w2, s2 = (t[4:].contiguous() for t in (w1, s1, w2, s2))
        kw.update(expert_map=torch.tensor([-1] * 4 + list(range(4)), dtype=torch.int32).cuda(),
                  global_num_experts=e)

    def run():
        return fused_experts(x, w1, w2, wts.cuda(), ids.int().cuda(), w1_scale=s1, w2_scale=s2,
                             block_shape=[1, 32], **kw).cpu()

    run()       # (the weights' scales are laid out on first use)
    outs, launches = [], []
    for gather in (False, True):
        monkeypatch.setattr(layer, "_GATHER", gather)
        before = ops.launch_count()
        outs.append(run())
        launches.append(ops.launch_count() - before)
        ops.check_device_status(x.device)
    assert launches[1] == launches[0] - 1           # no sorted copy
    assert torch.isfinite(outs[0]).all() and (m == 1 or outs[0].abs().max() > 0)
    assert torch.equal(outs[0], outs[1])
