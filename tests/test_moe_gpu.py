"""Fused MoE layer forward + backward (bf16 and FP8 forward) with emulated ranks, against a dense
fp32 PyTorch reference with autograd; plus the single-rank nn.Module path."""
import os
import subprocess
import sys

import pytest
import torch

from conftest import make_routed_inputs

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp(min=1e-6)).item()


@pytest.mark.parametrize('use_fp8', [False, True, 'pow2'])
def test_moe_forward_backward_emulated(use_fp8):
    pow2 = use_fp8 == 'pow2'       # power-of-two scales: the expert GEMMs use the block-scaled tensor-core instruction
    use_fp8 = bool(use_fp8)
    from deepep_b200.models.moe import ExpertWeights, MoEConfig, moe_backward, moe_forward, reference_moe
    from deepep_b200.parallel.local_cluster import LocalCluster
    R, T, H, I, E, K = 2, 96, 256, 256, 8, 2
    EL = E // R
    # poison the allocator's free blocks: padding rows and their scales must not leak stale memory into the result
    junk = torch.full((64 << 20,), float('nan'), device='cuda')
    del junk
    cfg = MoEConfig(hidden=H, intermediate=I, num_experts=E, num_topk=K, use_fp8=use_fp8, pow2_scales=pow2, num_sms=4)
    cl = LocalCluster(R, num_max_tokens_per_rank=T, hidden=H, num_topk=K, num_gpu_timeout_secs=5)
    xs, idxs, ws = make_routed_inputs(R, T, H, E, K, seed=21, device='cuda', vary_tokens=True)
    g = torch.Generator(device='cuda').manual_seed(3)
    w13_all = (torch.randn((E, 2 * I, H), device='cuda', generator=g) * 0.05).bfloat16()
    w2_all = (torch.randn((E, H, I), device='cuda', generator=g) * 0.05).bfloat16()
    weights = [ExpertWeights(w13_all[r * EL:(r + 1) * EL], w2_all[r * EL:(r + 1) * EL], use_fp8, pow2) for r in range(R)]

    ys, ctxs = moe_forward(cl, weights, xs, idxs, ws, cfg)
    torch.cuda.synchronize()
    cl.check_status()
    # reference with autograd
    xr = [x.float().requires_grad_(True) for x in xs]
    wr = [w.float().requires_grad_(True) for w in ws]
    w13r, w2r = w13_all.float().requires_grad_(True), w2_all.float().requires_grad_(True)
    refs = reference_moe(xr, idxs, wr, w13r, w2r)
    tol = (0.1 if pow2 else 0.08) if use_fp8 else 0.03
    for r in range(R):
        assert _rel(ys[r], refs[r]) < tol

    dys = [torch.randn(y.shape, device='cuda', generator=g).bfloat16() for y in ys]
    dxs, dws, dW13s, dW2s = moe_backward(cl, weights, ctxs, dys, cfg)
    torch.cuda.synchronize()
    cl.check_status()
    torch.autograd.backward(refs, [d.float() for d in dys])
    for r in range(R):
        assert _rel(dxs[r], xr[r].grad) < tol + 0.02
        valid = idxs[r] >= 0
        assert _rel(torch.where(valid, dws[r], torch.zeros_like(dws[r])), torch.where(valid, wr[r].grad, torch.zeros_like(wr[r].grad))) < tol + 0.03
        assert _rel(dW13s[r], w13r.grad[r * EL:(r + 1) * EL]) < tol + 0.03
        assert _rel(dW2s[r], w2r.grad[r * EL:(r + 1) * EL]) < tol + 0.03
    cl.destroy()


def test_moe_module_single_rank_trains():
    import deepep_b200
    from deepep_b200.models.moe import FusedMoE, MoEConfig
    from deepep_b200.parallel.local_cluster import SingleProcessGroup
    T, H, I, E, K = 128, 256, 128, 4, 2
    buf = deepep_b200.ElasticBuffer(SingleProcessGroup(), num_max_tokens_per_rank=T, hidden=H, num_topk=K, num_gpu_timeout_secs=5)
    layer = FusedMoE(buf, MoEConfig(hidden=H, intermediate=I, num_experts=E, num_topk=K, num_sms=4))
    x = torch.randn((T, H), device='cuda', generator=torch.Generator(device='cuda').manual_seed(4)).bfloat16().requires_grad_(True)
    y = layer(x)
    loss = (y.float() ** 2).mean()
    loss.backward()
    torch.cuda.synchronize()
    buf.check_status()
    assert y.shape == (T, H) and torch.isfinite(y.float()).all()
    for p in (x, layer.router, layer.w13, layer.w2):
        assert p.grad is not None and torch.isfinite(p.grad.float()).all() and p.grad.float().abs().sum() > 0
    buf.destroy()


@pytest.mark.parametrize('T,H,I,E,K,use_fp8', [(1, 256, 128, 4, 1, False), (77, 640, 128, 8, 3, False), (300, 1024, 256, 16, 8, False), (40, 256, 128, 120, 4, False),
                                               (129, 512, 256, 8, 4, True)])
def test_moe_module_gradients(T, H, I, E, K, use_fp8):
    """All gradients of the layer (router's share of dx and the router weights included) against fp32 autograd over the
    routing that the layer chose. bf16 intermediates bound the difference: every contraction sees operands rounded to 2^-9
    and four roundings lie between an input and a gradient, 4 * 2^-9 < 1e-2 of the norm; e4m3 operands (2^-4) in the
    forward products: the tolerance of the emulated-rank test above, plus its margins for gradients."""
    import deepep_b200
    from deepep_b200.models.moe import FusedMoE, MoEConfig, reference_moe
    from deepep_b200.parallel.local_cluster import SingleProcessGroup
    buf = deepep_b200.ElasticBuffer(SingleProcessGroup(), num_max_tokens_per_rank=T, hidden=H, num_topk=K, num_gpu_timeout_secs=5)
    layer = FusedMoE(buf, MoEConfig(hidden=H, intermediate=I, num_experts=E, num_topk=K, use_fp8=use_fp8, pow2_scales=use_fp8))
    g = torch.Generator(device='cuda').manual_seed(6)
    x = torch.randn((T, H), device='cuda', generator=g).bfloat16().requires_grad_(True)
    dy = torch.randn((T, H), device='cuda', generator=g).bfloat16()
    y = layer(x)
    y.backward(dy)
    buf.check_status()
    xr = x.detach().float().requires_grad_(True)
    wr, w13, w2 = (p.detach().bfloat16().float().requires_grad_(True) for p in (layer.router, layer.w13, layer.w2))
    logits = xr @ wr.t()
    idx = logits.bfloat16().float().topk(K, dim=1)[1]
    w = torch.softmax(logits.gather(1, idx), dim=1)
    ref = reference_moe([xr], [idx], [w], w13, w2)[0]
    ref.backward(dy.float())
    tol = 0.08 if use_fp8 else 0.02
    assert _rel(y, ref.detach()) < tol
    for got, want in ((x.grad, xr.grad), (layer.w13.grad, w13.grad), (layer.w2.grad, w2.grad)):
        assert _rel(got, want) < tol + 0.03
    if K > 1:
        assert _rel(layer.router.grad, wr.grad) < tol + 0.05
    else:
        assert layer.router.grad.abs().max() == 0       # the softmax over one expert does not depend on its logit
    assert layer.router.grad.dtype == layer.router.dtype
    buf.destroy()


def test_layers_of_several_threads():
    """Each thread has a buffer, a layer and a stream of its own; what the layers share (the launch set-up and the status word
    of the tensor-core kernels) is reached without the GIL. In a process of its own: the first calls are the ones that matter."""
    code = """
import threading, torch, deepep_b200
from deepep_b200.models.moe import FusedMoE, MoEConfig
from deepep_b200.parallel.local_cluster import SingleProcessGroup
N, T, H, I, E, K = 6, 100, 256, 128, 4, 2
layers = [FusedMoE(deepep_b200.ElasticBuffer(SingleProcessGroup(), num_max_tokens_per_rank=T, hidden=H, num_topk=K, num_gpu_timeout_secs=5),
                   MoEConfig(hidden=H, intermediate=I, num_experts=E, num_topk=K)) for _ in range(N)]
x = torch.randn((T, H), device='cuda').bfloat16()
streams, start, out = [torch.cuda.Stream() for _ in range(N)], threading.Barrier(N), [None] * N
torch.cuda.synchronize()
def work(i):
    with torch.cuda.stream(streams[i]):
        xi = x.clone().requires_grad_(True)
        start.wait()
        for _ in range(20):
            xi.grad = None
            y = layers[i](xi)
            y.backward(x)
        out[i] = (y.detach(), xi.grad)
        streams[i].synchronize()
threads = [threading.Thread(target=work, args=(i,)) for i in range(N)]
for t in threads: t.start()
for t in threads: t.join()
xi = x.clone().requires_grad_(True)
y = layers[0](xi)
y.backward(x)
assert all(torch.equal(a, y) and torch.equal(b, xi.grad) for a, b in out)
"""
    done = subprocess.run([sys.executable, '-c', code], cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))), capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]


def test_a_router_that_changes_before_the_backward_pass_is_noticed():
    """A bf16 router over a multiple of 128 experts is read where it lies; any other one is converted into a copy, which a
    change does not reach."""
    import deepep_b200
    from deepep_b200.models.moe import FusedMoE, MoEConfig
    from deepep_b200.parallel.local_cluster import SingleProcessGroup
    T, H, I, K = 64, 256, 128, 2
    for E, dtype in ((128, torch.bfloat16), (128, torch.float32), (8, torch.bfloat16)):
        buf = deepep_b200.ElasticBuffer(SingleProcessGroup(), num_max_tokens_per_rank=T, hidden=H, num_topk=K, num_gpu_timeout_secs=5)
        layer = FusedMoE(buf, MoEConfig(hidden=H, intermediate=I, num_experts=E, num_topk=K))
        layer.router = torch.nn.Parameter(layer.router.detach().to(dtype))
        x = torch.randn((T, H), device='cuda', generator=torch.Generator(device='cuda').manual_seed(2)).bfloat16().requires_grad_(True)
        layer(x).sum().backward()
        kept, x.grad = x.grad, None
        y = layer(x)
        with torch.no_grad():
            layer.router.mul_(2)
        if E == 128 and dtype == torch.bfloat16:
            with pytest.raises(RuntimeError, match='modified by an inplace operation'):
                y.sum().backward()
        else:
            y.sum().backward()
            assert torch.equal(x.grad, kept)
        buf.destroy()


@pytest.mark.parametrize('T,E,K,use_fp8,pow2', [(77, 8, 3, False, False), (1, 4, 1, False, False), (130, 16, 4, True, True), (64, 8, 2, True, False)])
def test_module_and_list_functions_give_the_same_bits(T, E, K, use_fp8, pow2):
    """The native calls of the module against moe_forward / moe_backward on the same routing."""
    import deepep_b200
    from deepep_b200 import ops
    from deepep_b200.models.moe import FusedMoE, MoEConfig, moe_backward, moe_forward, route
    from deepep_b200.parallel.local_cluster import SingleProcessGroup
    H, I = 512, 256
    buf = deepep_b200.ElasticBuffer(SingleProcessGroup(), num_max_tokens_per_rank=T, hidden=H, num_topk=K, num_gpu_timeout_secs=5)
    layer = FusedMoE(buf, MoEConfig(hidden=H, intermediate=I, num_experts=E, num_topk=K, use_fp8=use_fp8, pow2_scales=pow2))
    g = torch.Generator(device='cuda').manual_seed(T)
    x = torch.randn((T, H), device='cuda', generator=g).bfloat16().requires_grad_(True)
    dy = torch.randn((T, H), device='cuda', generator=g).bfloat16()
    y = layer(x)
    y.backward(dy)
    padded = torch.nn.functional.pad(layer.router.detach().bfloat16(), (0, 0, 0, -E % 128))
    idx, w = route(ops.gemm(x.detach(), padded)[:, :E], K)
    ys, ctxs = moe_forward(layer.comm, [layer.weights], [x.detach()], [idx], [w], layer.cfg)
    assert torch.equal(ys[0], y)
    dx, dw, d13, d2 = (t[0] for t in moe_backward(layer.comm, [layer.weights], ctxs, [dy], layer.cfg))
    d_router = deepep_b200._C.router_backward(x.detach(), padded, idx, w, dw, E, dx)       # (adds its share to dx)
    assert torch.equal(d13, layer.w13.grad) and torch.equal(d2, layer.w2.grad)
    assert torch.equal(dx, x.grad) and torch.equal(d_router.float(), layer.router.grad)
    buf.check_status()
    buf.destroy()
