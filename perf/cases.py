"""Performance cases of the library on one GPU: what programs built on it do, through its public entry points.

A case names one kind of work (`kind`) and its sizes:

* ``decode``   low-latency dispatch + weighted combine of a decode batch (``Buffer``), eager or replayed from a CUDA graph;
* ``exchange`` high-throughput dispatch + combine (``ElasticBuffer``), bf16 or FP8 payload;
* ``legacy``   the first-generation normal mode: layout query, dispatch, combine (``Buffer``);
* ``ranks``    dispatch + combine of several virtual ranks on one GPU (``LocalCluster``): the multi-rank kernels;
* ``forward``  router top-k and the forward pass of the MoE layer (``route``, ``moe_forward``): prefill or decode;
* ``train``    forward and backward of the MoE layer with explicit weights (``moe_forward``, ``moe_backward``);
* ``module``   one training iteration of ``FusedMoE``: router, forward, backward, refresh of the derived weight copies;
* ``experts``  an expert MLP put together from ``deepep_b200.ops``: cast, grouped GEMM, SwiGLU, grouped GEMM;
* ``engram``   rows of an Engram table fetched by index.

Tokens are N(0, 1), weights N(0, 0.02), routing is the top-k of N(0, 1) logits, or of logits with Zipf(1.2)
expert popularity where ``zipf`` is set.
"""
import math

import torch

import deepep_b200
from deepep_b200 import ops
from deepep_b200.models.moe import ExpertWeights, FusedMoE, MoEConfig, moe_backward, moe_forward, quantize_weight_128x128, route
from deepep_b200.parallel.local_cluster import LocalCluster, SingleProcessGroup
from deepep_b200.utils import gate


def listed():
    return [
        # the smallest serving step: four sequences decode one token each, bf16 rows, issued call by call
        dict(name='decode_4_bf16', kind='decode', tokens=4, max_tokens=128, hidden=7168, experts=256, topk=8, fp8=False, graph=False,
             hook=False),
        # the decode step that low-latency mode is made for: 128 tokens, FP8 dispatch, captured in a CUDA graph
        dict(name='decode_128_fp8_graph', kind='decode', tokens=128, max_tokens=128, hidden=7168, experts=256, topk=8, fp8=True, graph=True,
             hook=False),
        # a short prompt, or the tail of a batch: an odd token count, bf16, the host waits for the counts (the default)
        dict(name='exchange_133_bf16', kind='exchange', tokens=133, hidden=2048, experts=64, topk=6, fp8=False, expand=False,
             zero_copy=False, cpu_sync=True),
        # the benchmark's step: 8192 tokens of hidden 7168, 256 experts, top-8, cast to FP8 inside the dispatch
        dict(name='exchange_8192_fp8', kind='exchange', tokens=8192, hidden=7168, experts=256, topk=8, fp8=True, expand=False,
             zero_copy=False, cpu_sync=True),
        # a training batch on the first-generation API, a token count that divides by nothing
        dict(name='legacy_4001_bf16', kind='legacy', tokens=4001, hidden=4096, experts=64, topk=4),
        # four ranks: every kernel of the multi-rank path (count exchange, unpacking, reduction over ranks)
        dict(name='ranks4_1024_fp8', kind='ranks', ranks=4, tokens=1024, hidden=4096, experts=128, topk=8),
        # decode through the whole MoE layer on a rank that owns 32 of 256 experts: bound by reading the weights
        dict(name='forward_64_fp8', kind='forward', tokens=64, hidden=7168, intermediate=2048, experts=32, topk=8, fp8=True, zipf=False),
        # prefill through the whole MoE layer in bf16, ragged
        dict(name='forward_2011_bf16', kind='forward', tokens=2011, hidden=4096, intermediate=1536, experts=16, topk=4, fp8=False, zipf=False),
        # the fused MoE benchmark: 4096 tokens, skewed routing, FP8 forward, bf16 gradients, a rank's 32 experts
        dict(name='train_4096_fp8', kind='train', tokens=4096, hidden=7168, intermediate=2048, experts=32, topk=8, fp8=True, zipf=True),
        # a small model's layer trained as a torch module; the weights have changed, so their copies are rebuilt
        dict(name='module_1000_bf16', kind='module', tokens=1000, hidden=2048, intermediate=1024, experts=8, topk=2, fp8=False),
        # a prefill batch through FP8 experts with arbitrary (not power-of-two) scales, built from the operators
        dict(name='experts_8x700_fp8', kind='experts', rows=700, groups=8, hidden=4096, intermediate=2048, fp8=True),
        # memory look-up for a prefill batch: eight rows of 2048 bf16 values for each of 2048 tokens
        dict(name='engram_2048x8_bf16', kind='engram', tokens=2048, entries=8, hidden=2048, table=131072),
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], uniform over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(['decode', 'exchange', 'exchange', 'legacy', 'ranks', 'forward', 'forward', 'train', 'module', 'experts', 'engram'])
    if kind == 'decode':
        fp8 = rng.random() < 0.6
        graph = fp8 or rng.random() < 0.5
        return dict(kind=kind, tokens=_log(rng, 1, 128), max_tokens=128, hidden=_log(rng, 1024, 7168, 128), experts=rng.choice([32, 64, 160, 256]),
                    topk=rng.randint(1, 8), fp8=fp8, graph=graph, hook=not graph and rng.random() < 0.5)
    if kind == 'exchange':
        expand = rng.random() < 0.3
        return dict(kind=kind, tokens=_log(rng, 16, 8192), hidden=_log(rng, 1024, 7168, 256 if expand else 128), experts=rng.choice([16, 64, 128, 256]),
                    topk=rng.randint(1, 8), fp8=rng.random() < 0.6, expand=expand, zero_copy=rng.random() < 0.3, cpu_sync=rng.random() < 0.7)
    if kind == 'legacy':
        return dict(kind=kind, tokens=_log(rng, 16, 8192), hidden=_log(rng, 1024, 7168, 128), experts=rng.choice([16, 64, 256]), topk=rng.randint(1, 8))
    if kind == 'ranks':
        return dict(kind=kind, ranks=rng.choice([2, 4, 8]), tokens=_log(rng, 16, 1024), hidden=_log(rng, 1024, 7168, 512), experts=rng.choice([64, 128, 256]),
                    topk=rng.randint(2, 8))
    if kind == 'forward':
        return dict(kind=kind, tokens=_log(rng, 8, 4096), hidden=_log(rng, 1024, 7168, 256), intermediate=_log(rng, 512, 2048, 256),
                    experts=rng.choice([8, 16, 32]), topk=rng.randint(1, 8), fp8=rng.random() < 0.6, zipf=rng.random() < 0.3)
    if kind == 'train':
        return dict(kind=kind, tokens=_log(rng, 64, 4096), hidden=_log(rng, 1024, 7168, 256), intermediate=_log(rng, 512, 2048, 256),
                    experts=rng.choice([8, 16, 32]), topk=rng.randint(1, 8), fp8=rng.random() < 0.6, zipf=rng.random() < 0.5)
    if kind == 'module':
        return dict(kind=kind, tokens=_log(rng, 64, 4096), hidden=_log(rng, 1024, 2048, 256), intermediate=_log(rng, 512, 1024, 128),
                    experts=rng.choice([4, 8]), topk=rng.randint(1, 4), fp8=rng.random() < 0.5)
    if kind == 'experts':
        return dict(kind=kind, rows=_log(rng, 16, 2048), groups=rng.choice([1, 4, 8, 16]), hidden=_log(rng, 1024, 7168, 256),
                    intermediate=_log(rng, 512, 2048, 256), fp8=rng.random() < 0.6)
    return dict(kind=kind, tokens=_log(rng, 16, 4096), entries=rng.choice([1, 2, 4, 8]), hidden=_log(rng, 256, 4096, 64), table=131072)


# ---------------------------------------------------------------------------------------------------- inputs
def _tokens(gen, *shape):
    return torch.randn(shape, device='cuda', generator=gen, dtype=torch.bfloat16)


def _weights(gen, *shape):
    return torch.randn(shape, device='cuda', generator=gen, dtype=torch.bfloat16).mul_(0.02)


def _logits(gen, tokens, experts, zipf=False):
    if zipf:
        return gate.get_zipf_scores(tokens, experts, 1.2, device='cuda', generator=gen)
    return gate.get_balanced_scores(tokens, experts, device='cuda', generator=gen)


def _routing(gen, tokens, experts, topk):
    return gate.topk_from_scores(_logits(gen, tokens, experts), topk)


def _elastic(tokens, hidden, topk, fp8=False):
    return deepep_b200.ElasticBuffer(SingleProcessGroup(), num_max_tokens_per_rank=tokens, hidden=hidden, num_topk=topk, use_fp8_dispatch=fp8,
                                     num_gpu_timeout_secs=20)


def prepare(case, seed):
    gen = torch.Generator(device='cuda').manual_seed(seed)
    kind, s = case['kind'], dict(case=case)
    if kind == 'decode':
        T, H, E, K = case['tokens'], case['hidden'], case['experts'], case['topk']
        s['x'] = _tokens(gen, T, H)
        s['idx'], s['w'] = _routing(gen, T, E, K)
        s['buf'] = deepep_b200.Buffer(SingleProcessGroup(), num_rdma_bytes=deepep_b200.Buffer.get_low_latency_rdma_size_hint(
            case['max_tokens'], H, 1, E), low_latency_mode=True, num_gpu_timeout_secs=20)
        if case['fp8']:
            s['y'] = _tokens(gen, E, case['max_tokens'], H)         # the experts' output, in the packed layout
        if case['graph']:
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                _decode(s)
            torch.cuda.current_stream().wait_stream(side)
            torch.cuda.synchronize()
            s['graph'] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(s['graph']):
                s['out'] = _decode(s)
            for t in s['out'].values():                              # rows of the packed layout that no token fills stay zero
                t.zero_()
    elif kind in ('exchange', 'legacy'):
        T, H, E, K = case['tokens'], case['hidden'], case['experts'], case['topk']
        s['x'] = _tokens(gen, T, H)
        s['idx'], s['w'] = _routing(gen, T, E, K)
        if kind == 'exchange':
            s['buf'] = _elastic(T, H, K, case['fp8'])
            s['y'] = _tokens(gen, T * K if case['expand'] else T, H)
        else:
            s['buf'] = deepep_b200.Buffer(SingleProcessGroup(), num_nvl_bytes=deepep_b200.Buffer.get_dispatch_config(1).get_nvl_buffer_size_hint(
                2 * H, 1, T, K), num_gpu_timeout_secs=20)
            s['y'] = _tokens(gen, T, H)
    elif kind == 'ranks':
        R, T, H, E, K = case['ranks'], case['tokens'], case['hidden'], case['experts'], case['topk']
        s['cluster'] = LocalCluster(R, num_max_tokens_per_rank=T, hidden=H, num_topk=K, use_fp8_dispatch=True, num_gpu_timeout_secs=20)
        s['xs'] = [_tokens(gen, T, H) for _ in range(R)]
        # the order of the tokens comes from the seed, how many of them each rank gets from the sizes: outputs keep their shapes
        fixed = torch.Generator(device='cuda').manual_seed(T)
        s['routes'] = []
        for _ in range(R):
            order = torch.randperm(T, device='cuda', generator=gen)
            s['routes'].append(tuple(t[order] for t in _routing(fixed, T, E, K)))
        held = [sum(int((idx // (E // R) == r).any(dim=1).sum()) for idx, _ in s['routes']) for r in range(R)]
        s['ys'] = [_tokens(gen, n, H) for n in held]                 # what every rank's experts return for the tokens it holds
    elif kind in ('forward', 'train'):
        T, H, I, E, K = case['tokens'], case['hidden'], case['intermediate'], case['experts'], case['topk']
        s['cfg'] = MoEConfig(hidden=H, intermediate=I, num_experts=E, num_topk=K, use_fp8=case['fp8'], pow2_scales=case['fp8'])
        s['cluster'] = LocalCluster(1, num_max_tokens_per_rank=T, hidden=H, num_topk=K, num_gpu_timeout_secs=20)
        s['weights'] = ExpertWeights(_weights(gen, E, 2 * I, H), _weights(gen, E, H, I), case['fp8'], case['fp8'])
        s['x'] = _tokens(gen, T, H)
        s['logits'] = _logits(gen, T, E, case['zipf'])
        if kind == 'train':
            s['idx'], s['w'] = route(s['logits'], K)
            s['dy'] = _tokens(gen, T, H)
    elif kind == 'module':
        T, H, I, E, K = case['tokens'], case['hidden'], case['intermediate'], case['experts'], case['topk']
        cfg = MoEConfig(hidden=H, intermediate=I, num_experts=E, num_topk=K, use_fp8=case['fp8'], pow2_scales=case['fp8'])
        s['layer'] = FusedMoE(_elastic(T, H, K), cfg, seed=seed)
        s['x'] = _tokens(gen, T, H).requires_grad_(True)
        s['dy'] = _tokens(gen, T, H)
    elif kind == 'experts':
        G, H, I = case['groups'], case['hidden'], case['intermediate']
        # ragged groups; how many rows each has comes from the sizes, outputs keep their shapes
        counts = torch.randint(case['rows'] // 2, case['rows'] + case['rows'] // 2 + 1, (G,), generator=torch.Generator().manual_seed(case['rows'])).tolist()
        ends, start = [], 0
        for n in counts:
            ends.append(start + n)
            start = -(-(start + n) // 128) * 128
        s['ends'] = torch.tensor(ends, dtype=torch.int32, device='cuda')
        s['x'] = _tokens(gen, start, H)
        s['row_weight'] = torch.rand((start,), device='cuda', generator=gen)
        s['w13'], s['w2'] = _weights(gen, G, 2 * I, H), _weights(gen, G, H, I)
        if case['fp8']:
            s['w13'], s['w2'] = quantize_weight_128x128(s['w13']), quantize_weight_128x128(s['w2'])
    else:
        s['buf'] = deepep_b200.ElasticBuffer(SingleProcessGroup(), num_bytes=deepep_b200.ElasticBuffer.get_engram_storage_size_hint(
            case['table'], case['hidden']), num_gpu_timeout_secs=20)
        s['buf'].engram_write(_tokens(gen, case['table'], case['hidden']))
        s['idx'] = torch.randint(0, case['table'], (case['tokens'], case['entries']), device='cuda', generator=gen, dtype=torch.int32)
    return s


# ---------------------------------------------------------------------------------------------------- one pass
def _decode(s):
    case, buf = s['case'], s['buf']
    recv, count, handle, _, hook = buf.low_latency_dispatch(s['x'], s['idx'], case['max_tokens'], case['experts'], use_fp8=case['fp8'],
                                                            return_recv_hook=case['hook'])
    if hook is not None:
        hook()
    # bf16: the experts are the identity, so the result shows every received row; FP8: the experts' output is at hand
    out, _, hook = buf.low_latency_combine(s['y'] if case['fp8'] else recv, s['idx'], s['w'], handle, return_recv_hook=case['hook'])
    if hook is not None:
        hook()
    if case['fp8']:
        return dict(out=out, count=count, rows=recv[0], scales=recv[1], source=handle[0], layout=handle[1])
    return dict(out=out, count=count, layout=handle[1])


def run(state):
    s, case = state, state['case']
    kind = case['kind']
    if kind == 'decode':
        if case['graph']:
            s['graph'].replay()
            return s['out']
        return _decode(s)
    if kind == 'exchange':
        recv, idx, w, handle, _ = s['buf'].dispatch(s['x'], topk_idx=s['idx'], topk_weights=s['w'], num_experts=case['experts'],
                                                    do_expand=case['expand'], zero_copy=case['zero_copy'], do_cpu_sync=case['cpu_sync'])
        y, wc, _ = s['buf'].combine(s['y'], handle, topk_weights=w)
        rows, scales = recv if case['fp8'] else (recv, None)
        return dict(rows=rows, scales=scales, idx=idx, w=w, y=y, wc=wc, source=handle.recv_src_metadata, ends=handle.psum_num_recv_tokens_per_expert)
    if kind == 'legacy':
        buf = s['buf']
        per_rank, _, per_expert, in_rank, _ = buf.get_dispatch_layout(s['idx'], case['experts'])
        recv, idx, w, _, handle, _ = buf.dispatch(s['x'], num_tokens_per_rank=per_rank, is_token_in_rank=in_rank,
                                                  num_tokens_per_expert=per_expert, topk_idx=s['idx'], topk_weights=s['w'])
        y, wc, _ = buf.combine(s['y'], handle, topk_weights=w)
        return dict(rows=recv, idx=idx, w=w, y=y, wc=wc, handle=list(handle), per_rank=per_rank, per_expert=per_expert, in_rank=in_rank)
    if kind == 'ranks':
        out = s['cluster'].dispatch([dict(x=x, topk_idx=i, topk_weights=w, num_experts=case['experts'], num_sms=12, fused_fp8=True)
                                     for x, (i, w) in zip(s['xs'], s['routes'])])
        back = s['cluster'].combine([dict(x=y, handle=o[3], topk_weights=o[2]) for y, o in zip(s['ys'], out)])
        return [dict(rows=o[0][0], scales=o[0][1], idx=o[1], w=o[2], y=b[0], wc=b[1]) for o, b in zip(out, back)]
    if kind == 'forward':
        idx, w = route(s['logits'], case['topk'])
        ys, _ = moe_forward(s['cluster'], [s['weights']], [s['x']], [idx], [w], s['cfg'])
        return dict(y=ys[0], idx=idx, w=w)
    if kind == 'train':
        ys, ctxs = moe_forward(s['cluster'], [s['weights']], [s['x']], [s['idx']], [s['w']], s['cfg'])
        dx, dw, d13, d2 = moe_backward(s['cluster'], [s['weights']], ctxs, [s['dy']], s['cfg'])
        return dict(y=ys[0], dx=dx[0], dw=dw[0], d13=d13[0], d2=d2[0])
    if kind == 'module':
        layer, x = s['layer'], s['x']
        x.grad = None
        layer.zero_grad(set_to_none=True)
        y = layer(x)
        y.backward(s['dy'])
        layer.refresh_weights()
        w = layer.weights
        out = dict(y=y, dx=x.grad, router=layer.router.grad, d13=layer.w13.grad, d2=layer.w2.grad, w13_t=w.w13_t, w2_t=w.w2_t)
        return dict(out, w13_q=w.w13_q, w13_sf=w.w13_sf, w2_q=w.w2_q, w2_sf=w.w2_sf) if case['fp8'] else out
    if kind == 'experts':
        if not case['fp8']:
            h1 = ops.grouped_gemm(s['x'], s['w13'], s['ends'])
            a, _ = ops.swiglu(h1, s['row_weight'])
            return dict(h1=h1, a=a, y=ops.grouped_gemm(a, s['w2'], s['ends']))
        q, sf = ops.quant_1x128(s['x'])
        h1 = ops.grouped_gemm(q, s['w13'][0], s['ends'], sfa=sf, sfb=s['w13'][1])
        a, asf = ops.swiglu(h1, s['row_weight'], quant=True)
        return dict(q=q, sf=sf, h1=h1, a=a, asf=asf, y=ops.grouped_gemm(a, s['w2'][0], s['ends'], sfa=asf, sfb=s['w2'][1]))
    rows, _ = s['buf'].engram_fetch(s['idx'])()
    return rows


# ---------------------------------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    kind = case['kind']
    if kind == 'engram':
        n = case['tokens'] * case['entries']
        return dict(bytes=n * (4 * case['hidden'] + 4), flops=0)
    if kind == 'experts':
        rows, H, I = case['rows'] * case['groups'], case['hidden'], case['intermediate']
        elem = 1 if case['fp8'] else 2
        weights = 3 * case['groups'] * H * I * elem
        acts = rows * (2 * H + 2 * H + 4 * I + elem * I + (H if case['fp8'] else 0))             # x, y, h1, a and the cast x
        return dict(bytes=weights + acts, flops=6 * rows * H * I)
    T, H, K = case['tokens'], case['hidden'], case['topk']
    route_bytes = T * K * 12
    if kind == 'decode':
        per_row = H + H // 32 if case['fp8'] else 2 * H
        return dict(bytes=T * 2 * H + T * K * (per_row + 2 * H) + T * 2 * H + route_bytes, flops=2 * T * K * H)
    if kind in ('exchange', 'legacy'):
        per_row = H + H // 32 if kind == 'exchange' and case['fp8'] else 2 * H
        copies = K if kind == 'exchange' and case['expand'] else 1
        return dict(bytes=T * 2 * H + T * copies * (per_row + 2 * H) + T * 2 * H + 3 * route_bytes, flops=0)
    if kind == 'ranks':
        R, E = case['ranks'], case['experts']
        held = R * (1 - math.comb(E - E // R, K) / math.comb(E, K))                              # ranks that hold a copy of a token
        return dict(bytes=R * T * (2 * H + held * (H + H // 32 + 2 * H) + 2 * H) + 3 * R * route_bytes, flops=0)
    I, E = case['intermediate'], case['experts']
    rows = T * K
    elem = 1 if case['fp8'] else 2
    used = E * (1 - (1 - K / E) ** T)                                                            # experts that some token selects
    if kind == 'forward':
        return dict(bytes=3 * used * H * I * elem + 4 * T * H + 4 * T * E + route_bytes, flops=6 * rows * H * I)
    weights = 3 * E * H * I
    b = 3 * used * H * I * (elem + 2) + 2 * weights + 8 * T * H + 2 * route_bytes                # weights once each way, their gradients
    f = 18 * rows * H * I
    if kind == 'module':
        b += 2 * weights + (weights if case['fp8'] else 0) + 8 * E * H                           # the derived copies, the router
        f += 6 * T * E * H
    return dict(bytes=b, flops=f)


def tolerance(case):
    kind = case['kind']
    # payloads are moved as they are, casts round to nearest
    if kind in ('legacy', 'engram') or (kind == 'exchange' and not case['expand']):
        return 'exact'
    # fp32 sums of at most eight bf16 rows, rounded to bf16 once
    if kind in ('decode', 'ranks', 'exchange'):
        return dict(rel=4e-3)
    # bf16 results and intermediates of tensor-core contractions; a bf16 step in front of the e4m3 cast can move a value by an e4m3 step
    return dict(rel=1e-2)
