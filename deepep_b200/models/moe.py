"""Fused expert-parallel MoE layer (forward and backward) on the kernels of this library.

Forward, per rank::

    router logits --router_topk--> (topk_idx, topk_weights)
    x --dispatch (expanded, expert-major, 128-aligned; optional in-kernel e4m3 cast)--> rows
    rows --grouped tcgen05 GEMM (W13: gate|up)--> h1 --SwiGLU * gate weight (optional fused cast)--> a
    a --grouped tcgen05 GEMM (W2)--> h2 --combine (sum over experts, fp32 accumulate)--> y

The expert GEMMs read the dispatch's device-resident prefix array as their group table, so nothing
but the dispatch itself synchronises with the host. The gate weight is applied inside the SwiGLU
kernel, which makes the combine a plain sum. Backward reverses the same pipeline: the gradient of
the combine is a cached (replayed) dispatch, the gradient of the dispatch is a combine, the data
gradients are grouped GEMMs with the transposed weights, the weight gradients are two GEMM launches
grouped along the contraction dimension (all experts at once, segment bounds read on the device), and
the gradient of the gate weights rides back with the combine. ``FusedMoE`` runs all of it, router included, as one
native call per direction (``_LayerFunction``).

The reference library has no model code; this is the "fused MoE layer fwd+bwd" workload that its
kernels exist to serve. ``moe_forward`` and ``moe_backward`` are written over LISTS of ranks, for the single-GPU emulation
(``LocalCluster``) and for layers put together by hand; the native calls of ``FusedMoE`` (``csrc/runtime/moe_layer.cpp``) take
the same steps in the same order for the rank of a process and give the same bits.
"""
from __future__ import annotations

from dataclasses import dataclass
from typing import Any, List, Optional, Sequence, Tuple

import torch

from .._native import _C, require_native
from ..utils.envs import check_torch_deterministic


@dataclass
class MoEConfig:
    hidden: int
    intermediate: int
    num_experts: int
    num_topk: int
    use_fp8: bool = False          # e4m3 dispatch + e4m3 expert GEMMs (weights 128x128 block scaled), bf16 gradients
    pow2_scales: bool = False      # with use_fp8: every scale is a power of two (UE8M0), applied by the tensor core itself
    expert_alignment: int = 128
    num_sms: int = 24


def quantize_weight_128x128(w: torch.Tensor, pow2: bool = False) -> Tuple[torch.Tensor, torch.Tensor]:
    """``[G, N, K]`` -> (e4m3 ``[G, N, K]``, fp32 scales ``[G, N / 128, K / 128]``); ``pow2`` rounds the scales up to
    powers of two."""
    if w.is_cuda and w.dtype == torch.bfloat16 and _C is not None:
        return _C.quant_weights_128x128(w.contiguous(), pow2)
    G, N, K = w.shape
    blocks = w.float().view(G, N // 128, 128, K // 128, 128)
    amax = blocks.abs().amax(dim=(2, 4)).clamp(1e-4)
    scale = torch.div(amax, torch.full_like(amax, 448.0))
    if pow2:
        scale = torch.exp2(torch.ceil(torch.log2(scale)))
    q = (blocks / scale[:, :, None, :, None]).clamp(-448, 448).to(torch.float8_e4m3fn).view(G, N, K)
    return q, scale.contiguous()


def _transposed(w: torch.Tensor) -> torch.Tensor:
    """``[G, N, K]`` -> contiguous ``[G, K, N]``."""
    if w.is_cuda and w.dtype == torch.bfloat16 and _C is not None and w.size(0) <= 65535:      # (the kernel's grid)
        return _C.transpose_bf16(w)
    return w.transpose(1, 2).contiguous()


class ExpertWeights:
    """This rank's experts: ``w13 [local experts, 2 * intermediate, hidden]`` (gate rows first, then up) and
    ``w2 [local experts, hidden, intermediate]`` in bf16, plus the derived copies the kernels read."""

    def __init__(self, w13: torch.Tensor, w2: torch.Tensor, use_fp8: bool, pow2_scales: bool = False):
        self.w13, self.w2, self.use_fp8, self.pow2_scales = w13.contiguous(), w2.contiguous(), use_fp8, pow2_scales
        self.refresh()

    def refresh(self) -> None:
        """Rebuilds the transposed (for data gradients) and quantised (for FP8 forward) copies after an update."""
        self.w13_t = _transposed(self.w13)                     # [EL, hidden, 2I]
        self.w2_t = _transposed(self.w2)                       # [EL, I, hidden]
        if self.use_fp8:
            self.w13_q, self.w13_sf = quantize_weight_128x128(self.w13, self.pow2_scales)
            self.w2_q, self.w2_sf = quantize_weight_128x128(self.w2, self.pow2_scales)

    def forward_operands(self) -> List[torch.Tensor]:
        """The tensors that the forward GEMMs read."""
        return [self.w13_q, self.w13_sf, self.w2_q, self.w2_sf] if self.use_fp8 else [self.w13, self.w2]


class _SingleRankComm:
    """Gives one ``ElasticBuffer`` the list interface of ``LocalCluster``: the ``comm`` of ``moe_forward`` and ``moe_backward``
    for the rank of a process."""

    def __init__(self, buffer):
        self.buffers = [buffer]

    def dispatch(self, per_rank_kwargs):
        check_torch_deterministic()
        buf, kw = self.buffers[0], per_rank_kwargs[0]
        call = buf._dispatch_call(**kw)
        return [buf._dispatch_result(_C.Runtime.dispatch([buf.runtime], [call])[0], call, kw.get('handle'))]

    def combine(self, per_rank_kwargs):
        return [self.buffers[0].combine(**per_rank_kwargs[0])]


def route(logits: torch.Tensor, num_topk: int) -> Tuple[torch.Tensor, torch.Tensor]:
    """Top-k experts and softmax weights over the selected logits (hand-written kernel)."""
    require_native()
    if logits.dtype not in (torch.float32, torch.bfloat16) or logits.stride(1) != 1:
        logits = logits.float().contiguous()
    return _C.router_topk(logits, num_topk)


def moe_forward(comm, weights: Sequence[ExpertWeights], xs: Sequence[torch.Tensor], topk_idx: Sequence[torch.Tensor],
                topk_weights: Sequence[torch.Tensor], cfg: MoEConfig):
    """Expert part of the layer for all ranks of ``comm``. Returns ``(ys, contexts)``."""
    R = len(xs)
    # Rows in the alignment gaps between the experts mean nothing on the way forward: nobody reads their results, so nobody
    # writes them. The backward pass contracts over rows and makes its own zeros there (for bf16 the dispatch does).
    out = comm.dispatch([dict(x=xs[r], topk_idx=topk_idx[r], topk_weights=topk_weights[r], num_experts=cfg.num_experts,
                              expert_alignment=cfg.expert_alignment, do_expand=True, do_zero_padding=not cfg.use_fp8, num_sms=cfg.num_sms,
                              fused_fp8=cfg.use_fp8, round_scale=cfg.use_fp8 and cfg.pow2_scales, defer_counts=True) for r in range(R)])
    ctxs, h2s = [], []
    for r in range(R):
        recv_x, _, recv_w, handle, _ = out[r]
        w = weights[r]
        groups = dict(group_end=handle.psum_num_recv_tokens_per_expert, group_alignment=cfg.expert_alignment)
        if cfg.use_fp8:
            xq, xsf = recv_x
            pow2 = cfg.pow2_scales and w.pow2_scales
            h1 = _C.gemm(xq, w.w13_q, sfa=xsf, sfb=w.w13_sf, pow2_scales=pow2, zero_gap=False, **groups)
            aq, asf = _C.swiglu(h1, recv_w, None, True, pow2, **groups)
            h2 = _C.gemm(aq, w.w2_q, sfa=asf, sfb=w.w2_sf, pow2_scales=pow2, zero_gap=False, **groups)
        else:
            h1 = _C.gemm(recv_x, w.w13, zero_gap=False, **groups)
            a, _ = _C.swiglu(h1, recv_w, **groups)
            h2 = _C.gemm(a, w.w2, zero_gap=False, **groups)
        h2s.append(h2)
        ctxs.append(dict(recv_x=recv_x, recv_w=recv_w, handle=handle, h1=h1))
    comb = comm.combine([dict(x=h2s[r], handle=ctxs[r]['handle']) for r in range(R)])
    # With one rank nothing above waited for the host to learn the row counts: the whole layer is queued by now.
    for r, c in enumerate(ctxs):
        if c['handle']._counts_pending:
            comm.buffers[r]._finish_counts(c['handle'])
            rows = c['handle'].num_expanded_tokens
            c['recv_x'] = tuple(t[:rows] for t in c['recv_x']) if isinstance(c['recv_x'], tuple) else c['recv_x'][:rows]
            c['recv_w'], c['h1'] = c['recv_w'][:rows], c['h1'][:rows]
    return [c[0] for c in comb], ctxs


def moe_backward(comm, weights: Sequence[ExpertWeights], ctxs, dys: Sequence[torch.Tensor], cfg: MoEConfig):
    """Gradients of :func:`moe_forward`: ``(dxs, d_topk_weights, dW13s, dW2s)`` (bf16 / fp32 weights grads).

    Nothing here synchronises with the host: the expert segments are read on the device from the dispatch's prefix
    array, both by the grouped data-gradient GEMMs and by the two weight-gradient launches (one GEMM over all experts
    each, grouped along the contraction dimension). The SwiGLU backward kernel also produces the weighted activation
    (operand of the W2 gradient) and the gradient of the gate weights in the same pass.
    """
    R = len(dys)
    # gradient of the combine (a sum): replay the dispatch routing with dy as payload
    out = comm.dispatch([dict(x=dys[r].contiguous(), handle=ctxs[r]['handle'], do_expand=True, do_zero_padding=True,
                              num_sms=cfg.num_sms, fused_fp8=False) for r in range(R)])
    dx_rows, dw_rows, dW13s, dW2s = [], [], [], []
    for r in range(R):
        dh2 = out[r][0]
        c, w = ctxs[r], weights[r]
        handle, h1, recv_w = c['handle'], c['h1'], c['recv_w']
        ends = handle.psum_num_recv_tokens_per_expert
        groups = dict(group_end=ends, group_alignment=cfg.expert_alignment)
        el = w.w13.size(0)
        x_rows = c['recv_x']
        if cfg.use_fp8:
            x_rows = _C.dequant_1x128(x_rows[0], x_rows[1], **groups)
        # data gradients (zeros in the gaps come from the SwiGLU backward: the contractions below run over the rows)
        da = _C.gemm(dh2, w.w2_t, zero_gap=False, **groups)                                         # [rows, I]
        dh1, a_w, dw_row = _C.swiglu_backward(h1, da, recv_w, True, **groups)                       # [rows, 2I], [rows, I], [rows]
        dw_rows.append(dw_row)
        dx_rows.append(_C.gemm(dh1, w.w13_t, zero_gap=False, **groups))
        # weight gradients: contraction over every expert's (zero padded) rows, all experts in one launch each, the operands
        # read as they lie in memory (rows outermost)
        dW2s.append(_C.gemm_k_grouped(dh2, a_w, ends, el, cfg.expert_alignment, mn_major=True))          # [EL, hidden, I]
        dW13s.append(_C.gemm_k_grouped(dh1, x_rows, ends, el, cfg.expert_alignment, mn_major=True))      # [EL, 2I, hidden]
    # gradient of the dispatch: a combine that also carries the gate-weight gradients back
    comb = comm.combine([dict(x=dx_rows[r], handle=ctxs[r]['handle'], topk_weights=dw_rows[r].contiguous()) for r in range(R)])
    return [c[0] for c in comb], [c[1] for c in comb], dW13s, dW2s


class _LayerFunction(torch.autograd.Function):
    """The whole layer as one node, one native call in each direction. The router runs on this library's kernels: logits =
    x @ W_r^T on the tcgen05 GEMM (bf16 operands, fp32 accumulation), top-k and softmax over the selected logits; its
    backward pass turns the gradient of the top-k weights into the gradient of the logits (softmax Jacobian over the
    selected experts, zero elsewhere), adds their share to dx and contracts them with x to dW_r."""

    @staticmethod
    def forward(ctx, x, router, w13, w2, layer):
        y, ctx.call = _C.moe_layer_forward(layer.buffer.runtime, layer._native_config(), x, router, layer.weights.forward_operands())
        ctx.layer, ctx.router_dtype = layer, router.dtype
        # where the kernels read the router as it is (no converted copy), autograd has to notice a change before the backward pass
        as_it_is = router.dtype == torch.bfloat16 and router.size(0) % 128 == 0 and router.is_contiguous()
        ctx.save_for_backward(x, *([router] if as_it_is else []))
        return y

    @staticmethod
    def backward(ctx, dy):
        check_torch_deterministic()
        w = ctx.layer.weights
        dx, d_router, d13, d2 = _C.moe_layer_backward(ctx.layer.buffer.runtime, ctx.call, ctx.saved_tensors[0], dy, w.w13_t, w.w2_t)
        return dx, d_router.to(ctx.router_dtype), d13, d2, None


class FusedMoE(torch.nn.Module):
    """Expert-parallel MoE layer of one rank: ``y = sum_k w_k * Expert_k(x)`` with SwiGLU experts.

    Arguments:
        buffer: the rank's ``ElasticBuffer`` (sized for the layer's tokens / hidden / top-k).
        cfg: layer shape.
    Weights are initialised N(0, 0.02).
    """

    def __init__(self, buffer, cfg: MoEConfig, device='cuda', seed: int = 0):
        super().__init__()
        require_native()
        self.cfg, self.buffer = cfg, buffer
        self.comm = _SingleRankComm(buffer)      # for moe_forward / moe_backward with this layer's weights
        el = cfg.num_experts // buffer.num_ranks
        g = torch.Generator(device='cpu').manual_seed(seed + buffer.rank_idx)
        self.router = torch.nn.Parameter((torch.randn((cfg.num_experts, cfg.hidden), generator=g) * 0.02).to(device))
        self.w13 = torch.nn.Parameter((torch.randn((el, 2 * cfg.intermediate, cfg.hidden), generator=g) * 0.02).bfloat16().to(device))
        self.w2 = torch.nn.Parameter((torch.randn((el, cfg.hidden, cfg.intermediate), generator=g) * 0.02).bfloat16().to(device))
        self.weights = ExpertWeights(self.w13.data, self.w2.data, cfg.use_fp8, cfg.pow2_scales)

    def refresh_weights(self) -> None:
        """Call after an optimizer step: rebuilds the transposed / quantised weight copies."""
        self.weights = ExpertWeights(self.w13.data, self.w2.data, self.cfg.use_fp8, self.cfg.pow2_scales)

    def _native_config(self):
        c, b = self.cfg, self.buffer
        num_sms = c.num_sms if c.num_sms > 0 else b.get_theoretical_num_sms(c.num_experts, c.num_topk)
        return _C.MoELayerConfig(c.num_experts, c.num_topk, b.num_max_tokens_per_rank, c.expert_alignment, num_sms, c.use_fp8,
                                 c.use_fp8 and c.pow2_scales and self.weights.pow2_scales, b.allow_multiple_reduction, b.fuse_combine_reduce)

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        check_torch_deterministic()
        return _LayerFunction.apply(x, self.router, self.w13, self.w2, self)


def reference_moe(xs, topk_idx, topk_weights, w13_all: torch.Tensor, w2_all: torch.Tensor):
    """Dense fp32 reference over ALL experts (``w13_all [E, 2I, H]``, ``w2_all [E, H, I]``): per-rank outputs."""
    outs = []
    inter = w13_all.size(1) // 2
    for x, idx, w in zip(xs, topk_idx, topk_weights):
        y = torch.zeros_like(x, dtype=torch.float32)
        for k in range(idx.size(1)):
            e = idx[:, k]
            ok = e >= 0
            ee = e.clamp(min=0)
            h = torch.einsum('th,tfh->tf', x.float(), w13_all[ee].float())
            a = torch.nn.functional.silu(h[:, :inter]) * h[:, inter:]
            o = torch.einsum('ti,thi->th', a, w2_all[ee].float())
            y = y + torch.where(ok[:, None], o * w[:, k:k + 1].float(), torch.zeros_like(o))
        outs.append(y)
    return outs
