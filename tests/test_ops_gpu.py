"""Small MoE operators against plain PyTorch fp32 references."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('T,E,K', [(37, 16, 2), (300, 256, 8), (64, 2048, 32)])
def test_router_topk_softmax(T, E, K):
    import deepep_b200
    logits = torch.randn((T, E), device='cuda', generator=torch.Generator(device='cuda').manual_seed(0))
    idx, w = deepep_b200._C.router_topk(logits, K)
    vals, ref_idx = torch.topk(logits, K, dim=1, sorted=True)
    assert torch.equal(idx, ref_idx)
    assert torch.allclose(w, torch.softmax(vals, dim=1), atol=1e-6, rtol=1e-5)


@pytest.mark.parametrize('pow2,col_major', [(False, False), (True, False), (False, True)])
def test_quant_dequant_1x128(pow2, col_major):
    import deepep_b200
    from deepep_b200.utils.math import per_token_cast_back, per_token_cast_to_fp8
    x = torch.randn((333, 1024), device='cuda', generator=torch.Generator(device='cuda').manual_seed(1)).bfloat16()
    q, sf = deepep_b200._C.quant_1x128(x, pow2, col_major)
    rq, rsf = per_token_cast_to_fp8(x, round_scale=pow2)
    assert torch.equal(q.view(torch.uint8), rq.view(torch.uint8)) and torch.equal(sf, rsf)
    if col_major:
        assert sf.stride(0) == 1
    back = deepep_b200._C.dequant_1x128(q, sf.contiguous())
    assert torch.equal(back, per_token_cast_back(rq, rsf))


def test_swiglu_forward_backward_and_fused_cast():
    import deepep_b200
    from deepep_b200.utils.math import per_token_cast_to_fp8
    C = deepep_b200._C
    g = torch.Generator(device='cuda').manual_seed(2)
    M, I = 200, 512
    x = torch.randn((M, 2 * I), device='cuda', generator=g).bfloat16()
    rw = torch.rand(M, device='cuda', generator=g)
    out, _ = C.swiglu(x, rw)
    xf = x.float().requires_grad_(True)
    ref = torch.nn.functional.silu(xf[:, :I]) * xf[:, I:] * rw[:, None]
    assert torch.allclose(out.float(), ref.detach(), rtol=2e-2, atol=2e-2)
    q, sf = C.swiglu(x, rw, None, True)
    rq, rsf = per_token_cast_to_fp8(out)
    assert torch.equal(q.view(torch.uint8), rq.view(torch.uint8)) and torch.equal(sf, rsf)
    dout = torch.randn((M, I), device='cuda', generator=g).bfloat16()
    ref.backward(dout.float())
    dx = C.swiglu_backward(x, dout, rw)
    assert torch.allclose(dx.float(), xf.grad, rtol=3e-2, atol=3e-2)
    t = C.transpose_bf16(x)
    assert torch.equal(t, x.t().contiguous())


def test_ops_package_wrappers():
    """deepep_b200.ops: the typed entry points and their fp32 references agree."""
    from deepep_b200 import ops
    g = torch.Generator(device='cuda').manual_seed(3)
    a = torch.randn((300, 512), device='cuda', generator=g).bfloat16()
    b = (torch.randn((256, 512), device='cuda', generator=g) * 0.05).bfloat16()
    ref = ops.ref_gemm(a, b)
    assert ((ops.gemm(a, b).float() - ref).norm() / ref.norm()).item() < 1e-2
    # grouped, fp8 with block scales
    G, N, K = 3, 256, 512
    ends = torch.tensor([100, 300, 520], dtype=torch.int32, device='cuda')      # starts 0, 128, 384
    M = 640
    x = torch.randn((M, K), device='cuda', generator=g).bfloat16()
    w = (torch.randn((G, N, K), device='cuda', generator=g) * 0.05).bfloat16()
    out = ops.grouped_gemm(x, w, ends, 128)
    ref = ops.ref_grouped_gemm(x, w, ends, 128)
    for s0, e0 in ((0, 100), (128, 300), (384, 520)):
        assert ((out[s0:e0].float() - ref[s0:e0]).norm() / ref[s0:e0].norm()).item() < 1e-2
    xq, sfa = ops.quant_1x128(x)
    got8 = ops.gemm(xq, b.to(torch.float8_e4m3fn), sfa, torch.ones((2, 4), device='cuda'))
    ref8 = ops.ref_gemm(xq, b.to(torch.float8_e4m3fn), sfa, torch.ones((2, 4), device='cuda'))
    assert ((got8.float() - ref8).norm() / ref8.norm()).item() < 1e-2
    idx, wts = ops.router_topk(torch.randn((50, 64), device='cuda', generator=g), 4)
    assert idx.shape == (50, 4) and torch.allclose(wts.sum(dim=1), torch.ones(50, device='cuda'), atol=1e-5)
    y, _ = ops.swiglu(x)
    assert torch.allclose(y.float(), ops.ref_swiglu(x), rtol=2e-2, atol=2e-2)
    assert torch.equal(ops.transpose(x), x.t().contiguous())
    assert torch.equal(ops.dequant_1x128(xq, sfa), (xq.float() * sfa.repeat_interleave(128, dim=1)).bfloat16())


@pytest.mark.parametrize('rows,cols', [(64, 64), (200, 328), (130, 72), (1, 7), (512, 4096)])
def test_transpose_interior_edge_and_unaligned(rows, cols):
    """Interior tiles of aligned tensors take the 16-byte path, edge tiles and unaligned views the element-wise one."""
    import deepep_b200
    C = deepep_b200._C
    g = torch.Generator(device='cuda').manual_seed(rows * 1000 + cols)
    x = torch.randn((rows, cols), device='cuda', generator=g).bfloat16()
    assert torch.equal(C.transpose_bf16(x), x.t().contiguous())
    if cols > 8:     # a view whose rows start 2 bytes off a 16-byte boundary
        v = x[:, 1:]
        assert torch.equal(C.transpose_bf16(v), v.t().contiguous())


# rows of half a piece, of two pieces (the last one half), of four and eight: many rows in a warp; more than a warp, not whole warps
@pytest.mark.parametrize('I', [8, 24, 64, 128, 384, 640])
def test_streaming_ops_skip_or_zero_alignment_gaps(I):
    """Rows of the expanded layout behind their expert's end: the forward kernel leaves them alone, the backward kernels
    write zeros there, whatever the inputs hold in them."""
    import deepep_b200
    C = deepep_b200._C
    g = torch.Generator(device='cuda').manual_seed(5)
    align, ends_list = 16, [5, 16, 16, 49]          # a ragged group, a full one, an empty one, one that ends behind a full tile
    ends = torch.tensor(ends_list, dtype=torch.int32, device='cuda')
    M = 80                                           # rows past the last group's aligned end as well
    valid = torch.zeros(M, dtype=torch.bool, device='cuda')
    start = 0
    for e in ends_list:
        valid[start:e] = True
        start = -(-e // align) * align
    x = torch.randn((M, 2 * I), device='cuda', generator=g).bfloat16()
    dout = torch.randn((M, I), device='cuda', generator=g).bfloat16()
    rw = torch.rand(M, device='cuda', generator=g)
    full, _ = C.swiglu(x, rw)
    dx0, act0, dw0 = C.swiglu_backward(x, dout, rw, True)
    bad = x.clone()
    bad[~valid] = float('nan')
    out, _ = C.swiglu(bad, rw, group_end=ends, group_alignment=align)
    assert torch.equal(out[valid], full[valid])
    dx, act, dw = C.swiglu_backward(bad, dout, rw, True, group_end=ends, group_alignment=align)
    assert torch.equal(dx[valid], dx0[valid]) and torch.equal(act[valid], act0[valid]) and torch.equal(dw[valid], dw0[valid])
    assert (dx[~valid] == 0).all() and (act[~valid] == 0).all() and (dw[~valid] == 0).all()
    if I % 128 == 0:
        q, sf = C.quant_1x128(dout)
        q.view(torch.uint8)[~valid] = 0x7f          # NaN
        back = C.dequant_1x128(q, sf, group_end=ends, group_alignment=align)
        assert torch.equal(back[valid], C.dequant_1x128(*C.quant_1x128(dout))[valid]) and (back[~valid] == 0).all()


@pytest.mark.parametrize('offset', [1, 8, 16])
def test_inputs_that_start_anywhere(offset):
    """Contiguous views into flat buffers, as parameter buckets and received messages are: they start on no 16-byte boundary."""
    from deepep_b200 import ops
    from deepep_b200.models.moe import FusedMoE, MoEConfig, quantize_weight_128x128
    from deepep_b200.parallel.local_cluster import SingleProcessGroup
    import deepep_b200
    g = torch.Generator(device='cuda').manual_seed(offset)

    def view(t):
        flat = torch.empty(t.numel() + offset, dtype=t.dtype, device='cuda')
        flat[offset:].view(t.shape).copy_(t)
        return flat[offset:].view(t.shape)

    q, sf = ops.quant_1x128(torch.randn((5, 384), device='cuda', generator=g).bfloat16())
    assert torch.equal(ops.dequant_1x128(view(q), sf), ops.dequant_1x128(q, sf))
    w = torch.randn((2, 256, 128), device='cuda', generator=g).bfloat16()
    for a, b in zip(quantize_weight_128x128(view(w)), quantize_weight_128x128(w)):
        assert torch.equal(a.float(), b.float())
    buf = deepep_b200.ElasticBuffer(SingleProcessGroup(), num_max_tokens_per_rank=32, hidden=256, num_topk=2, num_gpu_timeout_secs=5)
    layer = FusedMoE(buf, MoEConfig(hidden=256, intermediate=128, num_experts=4, num_topk=2))
    x = torch.randn((32, 256), device='cuda', generator=g).bfloat16()
    y = layer(x)
    layer.router.data = view(layer.router.data)
    assert torch.equal(layer(x), y)
    torch.cuda.synchronize()
    buf.destroy()


@pytest.mark.parametrize('M,I', [(1, 8), (37, 8), (333, 128), (100, 384), (7, 16384)])
def test_streaming_ops_on_narrow_and_long_rows(M, I):
    """Rows that share a warp, and rows that a block of twice the threads walks; row counts that leave lanes without work."""
    from deepep_b200 import ops
    from deepep_b200.utils.math import per_token_cast_back, per_token_cast_to_fp8
    import deepep_b200
    g = torch.Generator(device='cuda').manual_seed(M + I)
    x = torch.randn((M, 2 * I), device='cuda', generator=g).bfloat16()
    rw = torch.rand((M,), device='cuda', generator=g)
    dout = torch.randn((M, I), device='cuda', generator=g).bfloat16()
    xf, wf = x.double().requires_grad_(True), rw.double().requires_grad_(True)
    ref = torch.nn.functional.silu(xf[:, :I]) * xf[:, I:] * wf[:, None]
    ref.backward(dout.double())
    half = max(1, M // 2)
    out, _ = ops.swiglu(x, rw)
    part, _ = ops.swiglu(x, rw, num_valid_rows=torch.tensor([half], dtype=torch.int32, device='cuda'))
    assert torch.equal(part[:half], out[:half])
    # one bf16 rounding (2^-9 of a value) and a few fp32 ones
    assert ((out.double() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-30).all()
    dx, act, dw = deepep_b200._C.swiglu_backward(x, dout, rw, True)
    assert ((dx.double() - xf.grad).abs() <= 2 ** -7 * xf.grad.abs() + 1e-4).all()
    assert ((act.double() - ref).abs() <= 2 ** -7 * ref.abs() + 1e-30).all()
    # the activation that the gradient of the weight sees is rounded to bf16: 2^-9 of every term
    terms = (dout.double() * ref.detach() / wf[:, None].detach()).abs().sum(dim=1)
    assert ((dw.double() - wf.grad).abs() <= 2 ** -8 * terms + 1e-6).all()
    if I % 128 == 0:
        q, sf = ops.swiglu(x, rw, quant=True)
        rq, rsf = per_token_cast_to_fp8(out)
        assert torch.equal(q.view(torch.uint8), rq.view(torch.uint8)) and torch.equal(sf, rsf)
        q, sf = ops.quant_1x128(x)
        rq, rsf = per_token_cast_to_fp8(x)
        assert torch.equal(q.view(torch.uint8), rq.view(torch.uint8)) and torch.equal(sf, rsf)
        assert torch.equal(ops.dequant_1x128(q, sf), per_token_cast_back(rq, rsf))


def test_swiglu_far_from_zero():
    """Gates whose sigmoid is about 1e-38, infinities and NaN: as the formula in fp32 gives them, also beside ordinary values."""
    from deepep_b200 import ops
    gates = torch.tensor([float('-inf'), float('inf'), float('nan'), -87.0, -87.5, -88.0, -88.5, 87.5, 100.0, 3e38, 0.0, -0.0, 1e-38, 5.0, -86.5, -1.0], device='cuda').bfloat16()
    up = torch.full((16,), 2.0 ** 60, device='cuda').bfloat16()
    up[9] = 0.5
    x = torch.cat([gates, up]).view(1, 32)
    gf, uf = gates.double(), up.double()
    s = torch.sigmoid(gf)
    ref, out = gf * s * uf, ops.swiglu(x)[0][0].double()
    dx = ops.swiglu_backward(x, torch.ones((1, 16), device='cuda').bfloat16())[0].double()
    dg, du = uf * s * (1 + gf * (1 - s)), gf * s
    tiny = 2.0 ** -126                                   # the smallest normal fp32 number: fewer bits are left below it
    for got, want in ((out, ref), (dx[:16], dg), (dx[16:], du)):
        ok = want.isfinite()
        # the exponential's error grows with its argument: 88 * 2^-23 of the result, then bf16 roundings; a sigmoid below the normal range
        # has an error of up to 2^-149 itself, times the factors behind it
        assert ((got[ok] - want[ok]).abs() <= 2 ** -7 * want[ok].abs() + tiny).all()
        assert (got[want.isnan()].isnan()).all()


@pytest.mark.parametrize('pow2', [False, True])
def test_weight_quantisation_of_blocks_that_are_not_finite(pow2):
    """A NaN makes its whole 128 x 128 block NaN, an infinity leaves zeros beside a NaN, as the elementwise definition has it;
    an all-zero block and one of the smallest values keep the floor of the scale."""
    from deepep_b200.models.moe import quantize_weight_128x128
    w = (torch.randn((2, 256, 384), device='cuda', generator=torch.Generator(device='cuda').manual_seed(9)) * 0.02).bfloat16()
    w[0, 5, 7], w[0, 130, 300], w[1, 255, 0], w[1, :128, :128] = float('nan'), float('-inf'), float('-nan'), 0
    w[1, :128, 128:256] = 1e-30
    (q, sf), (rq, rsf) = quantize_weight_128x128(w, pow2), quantize_weight_128x128(w.cpu(), pow2)
    q, rq = q.float().cpu(), rq.float()
    assert torch.equal(sf.cpu().isnan(), rsf.isnan()) and torch.equal(sf.cpu().nan_to_num(0), rsf.nan_to_num(0))
    assert torch.equal(q.isnan(), rq.isnan()) and torch.equal(q.nan_to_num(0), rq.nan_to_num(0))
    assert q[0, :128, :128].isnan().all() and rsf[0, 0, 0].isnan()
