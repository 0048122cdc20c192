"""Dispatch / combine of a one-rank group (plan, move and combine kernels of their own) against the pure-torch oracle, at
the sizes where their work is cut: one and several planning blocks, more than one batch per warp, top-k beyond what a lane
keeps in registers, rows that end inside a warp's slice, alignment gaps."""
import pytest
import torch

from conftest import make_routed_inputs

pytestmark = pytest.mark.gpu


def _buffer(T, H, K, **kw):
    import deepep_b200
    from deepep_b200.parallel.local_cluster import SingleProcessGroup
    return deepep_b200.ElasticBuffer(SingleProcessGroup(), num_max_tokens_per_rank=T, hidden=H, num_topk=K, num_gpu_timeout_secs=5, **kw)


@pytest.mark.parametrize('T,H,E,K', [
    (1, 128, 4, 1),          # one token
    (31, 1152, 8, 3),        # 2304-byte rows: a slice and a quarter, rows not a multiple of 512 bytes
    (1025, 256, 256, 8),     # two planning blocks, the second with one token more than the first leaves
    (8300, 128, 64, 2),      # more than one batch of 32 tokens per warp
    (70, 512, 32, 9),        # more top-k lanes than a planning lane keeps in registers
    (1100, 128, 64, 32),     # the largest top-k, two planning blocks
    (9000, 128, 40, 17),     # an odd large top-k and two batches per warp
])
@pytest.mark.parametrize('expand', [False, True])
@pytest.mark.parametrize('mode', ['bf16', 'fused', 'fused_col_major', 'prequantised'])
def test_dispatch_combine_against_the_oracle(T, H, E, K, expand, mode):
    from deepep_b200.utils import refs
    from deepep_b200.utils.math import per_token_cast_to_fp8
    align = 16
    buf = _buffer(T, H, K)
    (x,), (idx,), (w,) = make_routed_inputs(1, T, H, E, K, seed=T, device='cuda', masked_ratio=0.2)
    idx[::5] = -1                                          # tokens that nobody takes
    q, sf = per_token_cast_to_fp8(x)
    xin, kw = {'bf16': (x, {}), 'fused': (x, dict(fused_fp8=True)), 'prequantised': ((q, sf), {}),
               'fused_col_major': (x, dict(fused_fp8=True, use_tma_aligned_col_major_sf=True))}[mode]
    raw = x.cpu() if mode == 'bf16' else q.view(torch.uint8).cpu()
    e = refs.dispatch_local([raw], [idx.cpu()], [w.cpu()], 0, E, T, sfs=[sf.cpu()])
    ex = refs.expand_local(e, E, align)
    stats = torch.zeros(E, dtype=torch.int32, device='cuda')
    for sync in (True, False):
        recv, ridx, rw, handle, _ = buf.dispatch(xin, topk_idx=idx, topk_weights=w, num_experts=E, do_expand=expand, expert_alignment=align,
                                                 do_zero_padding=True, do_cpu_sync=sync, cumulative_local_expert_recv_stats=stats, **kw)
        torch.cuda.synchronize()
        buf.check_status()
        rows, scales = recv if isinstance(recv, tuple) else (recv, None)
        rows = rows.view(torch.uint8).cpu() if mode != 'bf16' else rows.cpu()
        n = e['recv_x'].size(0)
        if sync:
            assert handle.num_recv_tokens == n and rows.size(0) == (ex['num_rows'] if expand else n)
            assert handle.num_recv_tokens_per_expert_list == [-(-int(c) // align) * align for c in ex['counts']]
        meta = handle.recv_src_metadata.cpu()
        assert torch.equal(meta[:n, 0], e['recv_src_token_idx']) and (meta[n:] == -1).all()
        assert torch.equal(handle.num_unaligned_recv_tokens_per_expert.cpu().long(), ex['counts'])
        assert torch.equal(handle.topk_idx, idx) and handle.topk_idx.data_ptr() != idx.data_ptr()
        if not expand:
            assert torch.equal(rows[:n], e['recv_x']) and torch.equal(ridx[:n].cpu(), e['recv_topk_idx']) and torch.equal(rw[:n].cpu(), e['recv_topk_weights'])
            assert scales is None or torch.equal(scales[:n].cpu(), e['recv_sf'])
            assert (ridx[n:] == -1).all() and (rw[n:] == 0).all() and (meta[:n, 2:] == -1).all()
        else:
            assert torch.equal(meta[:n, 2:].long(), ex['lane_rows'])
            for g in range(E):
                s, c = int(ex['starts'][g]), int(ex['counts'][g])
                pick = ex['row_of'][g]
                assert torch.equal(rows[s:s + c], e['recv_x'][pick])
                lane = (e['recv_topk_idx'][pick] == g).float().argmax(dim=1)
                assert torch.equal(rw[s:s + c].cpu(), e['recv_topk_weights'][pick, lane])
                end = -(-(s + c) // align) * align
                assert (rows[s + c:end] == 0).all() and (rw[s + c:end] == 0).all()
                assert scales is None or (torch.equal(scales[s:s + c].cpu(), e['recv_sf'][pick]) and (scales[s + c:end] == 0).all())
        if scales is not None and mode == 'fused_col_major':
            assert scales.stride(0) == 1 and scales.stride(1) % 4 == 0
    expect = torch.stack([(idx == g).sum() for g in range(E)]).int() * 2
    assert torch.equal(stats, expect)
    # replay of the routing with other payload
    x2 = (x.float() * 2 + 1).bfloat16()
    again = buf.dispatch(x2, handle=handle, do_expand=expand, do_zero_padding=True, fused_fp8=False)[0]
    torch.cuda.synchronize()
    keep = e['recv_src_token_idx'].long()
    if not expand:
        assert torch.equal(again[:n].cpu(), x2.cpu()[keep])
    else:
        for g in range(E):
            s, c = int(ex['starts'][g]), int(ex['counts'][g])
            assert torch.equal(again[s:s + c].cpu(), x2.cpu()[keep[ex['row_of'][g]]])
    # combine of what came in
    y = torch.randn((rows.size(0), H), device='cuda', generator=torch.Generator(device='cuda').manual_seed(T)).bfloat16()
    bias = torch.randn((T, H), device='cuda', generator=torch.Generator(device='cuda').manual_seed(T + 1)).bfloat16()
    part = torch.zeros((n, H))
    wpart = torch.zeros((n, H))
    yc, lanes = y.cpu().float(), ex['lane_rows'] if expand else torch.arange(n).view(n, 1)
    for k in range(lanes.size(1)):
        ok = lanes[:, k] >= 0
        part[ok] += yc[lanes[ok, k]]
        if expand:
            wpart[ok] = torch.addcmul(wpart[ok], yc[lanes[ok, k]], rw.cpu()[lanes[ok, k]].view(-1, 1))
    out, ow, _ = buf.combine(y, handle, topk_weights=rw)
    outb, _, _ = buf.combine(y, handle, bias=bias)
    ref = torch.zeros((T, H))
    ref[keep] = part.bfloat16().float()
    assert torch.equal(out.cpu(), ref.bfloat16())
    assert torch.equal(outb.cpu(), (ref + bias.cpu().float()).bfloat16())
    assert torch.equal(ow, torch.where(idx >= 0, w, torch.zeros_like(w)))
    if expand:
        got = buf.combine(y, handle, topk_weights=rw, weighted=True)[0].cpu().float()
        wref = torch.zeros((T, H))
        wref[keep] = wpart
        # fused multiply-adds against separate roundings, then one bf16 rounding: at most one bf16 step apart
        assert torch.allclose(got, wref, rtol=2 ** -7, atol=1e-5)
    torch.cuda.synchronize()
    buf.check_status()
    buf.destroy()


def test_expanded_dispatch_with_less_room_than_tokens():
    """`num_worst_tokens` below the received count: the routing outputs end there, and so do the tokens that a combine finds.
    Expanded rows have room of their own: all of them arrive, with their weights."""
    T, H, E, K, room = 300, 256, 8, 3, 171
    buf = _buffer(T, H, K)
    (x,), (idx,), (w,) = make_routed_inputs(1, T, H, E, K, seed=12, device='cuda')
    recv, _, rw, handle, _ = buf.dispatch(x, topk_idx=idx, topk_weights=w, num_experts=E, do_expand=True, do_cpu_sync=False, num_worst_tokens=room)
    assert handle.recv_src_metadata.size(0) == room
    rows = handle.dst_expanded_row_idx.long()
    assert torch.equal(recv[rows.flatten()].view(T, K, H), x[:, None].expand(T, K, H)) and torch.equal(rw[rows], w)
    out, ow, _ = buf.combine(recv, handle, topk_weights=rw)
    ref, wref = (x.float() * K).bfloat16(), w.clone()
    ref[room:], wref[room:] = 0, 0
    assert torch.equal(out, ref) and torch.equal(ow, wref)
    torch.cuda.synchronize()
    buf.check_status()
    buf.destroy()


def _zero_copy_dispatch(buf, x, idx, **kw):
    return buf.dispatch(x, topk_idx=idx, num_experts=16, zero_copy=True, do_cpu_sync=False, **kw)


@pytest.mark.parametrize('capture_between', [False, True])
@pytest.mark.parametrize('first', ['comm', 'side', 'external'])
def test_calls_that_change_streams_stay_in_order(first, capture_between):
    """A synchronous call runs on the caller's stream, an asynchronous one on the communication stream. All use the buffer's
    regions and must not overtake one another, whatever the caller does about its streams: here it orders nothing. A call that
    is held up on its stream is followed by calls on another one; the second of them writes the same half of the receive
    region and has to be the one that stays."""
    T, H = 512, 2048
    buf = _buffer(T, H, 4)
    (x,), (idx,), _ = make_routed_inputs(1, T, H, 16, 4, seed=3, device='cuda')
    xs = [(x.float() * (i + 1)).bfloat16() for i in range(4)]
    late, other = torch.cuda.Stream(), torch.cuda.Stream()
    if first == 'external':
        late, raw = _external_stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(late):
        torch.cuda._sleep(200_000_000)                       # about a tenth of a second
        _zero_copy_dispatch(buf, xs[1], idx, async_with_compute_stream=first == 'comm')
    if capture_between:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            _zero_copy_dispatch(buf, xs[2], idx)             # (never replayed: it only takes its turn in the double buffer)
    with torch.cuda.stream(other):
        if not capture_between:
            _zero_copy_dispatch(buf, xs[2], idx)
        recv, _, _, handle, _ = _zero_copy_dispatch(buf, xs[3], idx)
        combined = buf.combine(recv, handle)[0]
    torch.cuda.synchronize()
    buf.check_status()
    assert torch.equal(recv[:handle.psum_num_recv_tokens_per_scaleup_rank[0]], xs[3][(idx >= 0).any(dim=1)])
    assert torch.equal(combined, xs[3])
    if capture_between:
        graph.reset()
    if first == 'external':
        _destroy_stream(raw)
    buf.destroy()


def _external_stream():
    import ctypes
    lib = ctypes.CDLL('libcudart.so.12')
    raw = ctypes.c_void_p()
    assert lib.cudaStreamCreateWithFlags(ctypes.byref(raw), 1) == 0          # non-blocking, like PyTorch's own
    return torch.cuda.ExternalStream(raw.value), raw


def _destroy_stream(raw):
    import ctypes
    assert ctypes.CDLL('libcudart.so.12').cudaStreamDestroy(raw) == 0


def test_a_stream_of_the_caller_may_be_gone_by_the_next_call():
    import deepep_b200
    from deepep_b200.parallel.local_cluster import SingleProcessGroup
    T, H, E, K = 64, 1024, 16, 4
    buf = _buffer(T, H, K)
    ll = deepep_b200.Buffer(SingleProcessGroup(), num_rdma_bytes=deepep_b200.Buffer.get_low_latency_rdma_size_hint(T, H, 1, E), low_latency_mode=True,
                            num_gpu_timeout_secs=5)
    (x,), (idx,), (w,) = make_routed_inputs(1, T, H, E, K, seed=4, device='cuda')
    for _ in range(3):
        stream, raw = _external_stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            recv, _, _, handle, _ = buf.dispatch(x, topk_idx=idx, num_experts=E)
            rows, _, lh, _, _ = ll.low_latency_dispatch(x, idx, T, E, use_fp8=False)
        stream.synchronize()
        _destroy_stream(raw)
        assert torch.equal(buf.combine(recv, handle)[0], x)
        out = ll.low_latency_combine(rows, idx, w, lh)[0]
        assert (out.float() - x.float() * w.sum(dim=1, keepdim=True)).abs().max() <= 2 ** -7 * x.float().abs().max()
    torch.cuda.synchronize()
    buf.destroy()
    ll.destroy()


@pytest.mark.parametrize('T,H,E,K', [
    (1, 1024, 8, 2),         # one token: the extra blocks only count
    (33, 1152, 256, 9),      # a row that ends inside a warp's slice, more top-k lanes than four warps look up in one round
    (128, 7168, 32, 16),     # the largest top-k, experts that hold more rows than a warp has lanes
])
@pytest.mark.parametrize('mode', ['bf16', 'fp8', 'pow2', 'ue8m0'])
@pytest.mark.parametrize('hook', [False, True])
def test_low_latency_against_the_oracle(T, H, E, K, mode, hook):
    import deepep_b200
    from deepep_b200.parallel.local_cluster import SingleProcessGroup
    from deepep_b200.utils.math import per_token_cast_back, per_token_cast_to_fp8, unpack_ue8m0
    if mode == 'ue8m0' and H % 512 != 0:
        pytest.skip('UE8M0 scales need hidden % 512 == 0')
    Tm = 128
    buf = deepep_b200.Buffer(SingleProcessGroup(), num_rdma_bytes=deepep_b200.Buffer.get_low_latency_rdma_size_hint(Tm, H, 1, E),
                             low_latency_mode=True, num_gpu_timeout_secs=5)
    (x,), (idx,), (w,) = make_routed_inputs(1, T, H, E, K, seed=T + K, device='cuda', masked_ratio=0.2)
    stats = torch.zeros(E, dtype=torch.int32, device='cuda')
    fp8 = mode != 'bf16'
    q, sc = per_token_cast_to_fp8(x, round_scale=mode in ('pow2', 'ue8m0'))
    for _ in range(2):
        recv, count, handle, _, h = buf.low_latency_dispatch(x, idx, Tm, E, cumulative_local_expert_recv_stats=stats, use_fp8=fp8,
                                                             round_scale=mode in ('pow2', 'ue8m0'), use_ue8m0=mode == 'ue8m0', return_recv_hook=hook)
        if hook:
            h()
        torch.cuda.synchronize()
        buf.check_status()
        rows = torch.zeros((E, Tm, H), device='cuda', dtype=torch.bfloat16)
        for e in range(E):
            tok, lane = (idx == e).nonzero(as_tuple=True)
            n = tok.numel()
            assert int(count[e]) == n and int(handle[1][e, 0]) == n
            assert torch.equal(handle[0][e, :n], (tok | (lane << 16)).int())
            if n == 0:
                continue
            if not fp8:
                assert torch.equal(recv[e, :n], x[tok])
                rows[e, :n] = x[tok]
                continue
            assert torch.equal(recv[0][e, :n].view(torch.uint8), q[tok].view(torch.uint8)) and recv[1].stride(1) == 1
            sf = recv[1][e, :n]
            sf = unpack_ue8m0(sf.contiguous()).view(n, -1) if mode == 'ue8m0' else sf
            assert torch.equal(sf.float(), sc[tok])
            rows[e, :n] = per_token_cast_back(q[tok], sc[tok].contiguous())
        ref = torch.zeros((T, H), device='cuda')
        for k in range(K):
            for t in range(T):
                e = int(idx[t, k])
                if e >= 0:
                    j = int(((idx[:t] == e).any(dim=1)).sum())
                    ref[t] += w[t, k] * rows[e, j].float()
        for logfmt in (False, True):        # LogFMT takes the message path of the multi-rank kernels, on the same handle
            out, _, h = buf.low_latency_combine(rows, idx, w, handle, use_logfmt=logfmt, return_recv_hook=hook)
            if hook:
                h()
            torch.cuda.synchronize()
            buf.check_status()
            # one bf16 rounding of an fp32 sum; a 10-bit log code is within 2 % of a value
            tol = 3e-2 if logfmt else 2 ** -8
            assert (out.float() - ref).norm() <= tol * ref.norm() + 1e-6
    assert torch.equal(stats, torch.stack([(idx == e).sum() for e in range(E)]).int() * 2)
    buf.destroy()


@pytest.mark.parametrize('hidden,fp8', [(8, False), (520, False), (2048, False), (48, True), (1040, True)])
def test_engram_fetch_from_local_memory(hidden, fp8):
    """Rows that end inside a warp's kilobyte, on and off 32-byte boundaries; indices outside the table fetch nothing."""
    import deepep_b200
    from deepep_b200.parallel.local_cluster import SingleProcessGroup
    entries = 300
    dtype = torch.float8_e4m3fn if fp8 else torch.bfloat16
    buf = deepep_b200.ElasticBuffer(SingleProcessGroup(), num_bytes=deepep_b200.ElasticBuffer.get_engram_storage_size_hint(entries, hidden), num_gpu_timeout_secs=5)
    g = torch.Generator(device='cuda').manual_seed(hidden)
    table = torch.randn((entries, hidden), device='cuda', generator=g).to(dtype)
    sf = torch.rand((entries, 3), device='cuda', generator=g) if fp8 else None
    buf.engram_write(table, sf)
    idx = torch.randint(0, entries, (37, 3), device='cuda', generator=g, dtype=torch.int32)
    flat = idx.flatten().long()
    for _ in range(2):
        data, got = buf.engram_fetch(idx, use_tma_aligned_col_major_sf=fp8)()
        assert torch.equal(data.view(torch.uint8), table.view(torch.uint8)[flat])
        assert got is None or torch.equal(got, sf[flat].view(37, 9))
    bad = idx.clone()
    bad[5, 1], bad[6, 2] = -1, entries
    data, _ = buf.engram_fetch(bad)()
    keep = (bad.flatten() >= 0) & (bad.flatten() < entries)
    assert torch.equal(data.view(torch.uint8)[keep], table.view(torch.uint8)[flat[keep]])
    torch.cuda.synchronize()
    buf.check_status()
    buf.destroy()


def test_calls_refuse_to_run_under_filled_uninitialised_memory():
    """PyTorch's deterministic mode with filled memory would write over what arrives: every entry point says so."""
    import deepep_b200
    from deepep_b200.models.moe import FusedMoE, MoEConfig
    from deepep_b200.parallel.local_cluster import SingleProcessGroup
    T, H, E, K = 32, 256, 4, 2
    (x,), (idx,), (w,) = make_routed_inputs(1, T, H, E, K, seed=1, device='cuda')
    buf = _buffer(T, H, K)
    old = deepep_b200.Buffer(SingleProcessGroup(), num_nvl_bytes=deepep_b200.Buffer.get_dispatch_config(1).get_nvl_buffer_size_hint(2 * H, 1, T, K),
                             num_gpu_timeout_secs=5)
    layer = FusedMoE(buf, MoEConfig(hidden=H, intermediate=128, num_experts=E, num_topk=K))
    y = layer(x.requires_grad_(True))
    recv, _, _, handle, _ = buf.dispatch(x.detach(), topk_idx=idx, topk_weights=w, num_experts=E)
    calls = [lambda: buf.dispatch(x.detach(), topk_idx=idx, num_experts=E), lambda: buf.combine(recv, handle), lambda: layer(x), lambda: y.sum().backward(),
             lambda: old.dispatch(x.detach(), topk_idx=idx, topk_weights=w, num_experts=E)]
    torch.use_deterministic_algorithms(True)
    try:
        for call in calls:
            with pytest.raises(AssertionError, match='fill_uninitialized_memory'):
                call()
    finally:
        torch.use_deterministic_algorithms(False)
    buf.destroy()
    old.destroy()


@pytest.mark.parametrize('T,K', [(0, 2), (1, 8), (1025, 3), (8192, 8), (8193, 8), (65536, 1), (65537, 1), (5000, 32)])
def test_layout_query_on_both_sides_of_its_line(T, K):
    """One cluster up to 64k pairs, all SMs above."""
    import deepep_b200
    from deepep_b200.parallel.local_cluster import SingleProcessGroup
    E = 96
    buf = deepep_b200.Buffer(SingleProcessGroup(), num_nvl_bytes=1 << 24, num_gpu_timeout_secs=5)
    g = torch.Generator(device='cuda').manual_seed(T)
    idx = torch.randint(-1, E, (T, K), device='cuda', generator=g)
    for dtype in (torch.int64, torch.int32):
        per_rank, _, per_expert, in_rank, _ = buf.get_dispatch_layout(idx.to(dtype), E)
        assert torch.equal(per_expert.long(), torch.bincount(idx[idx >= 0], minlength=E))
        assert torch.equal(in_rank[:, 0], (idx >= 0).any(dim=1)) and per_rank.item() == int(in_rank.sum())
    buf.destroy()


@pytest.mark.parametrize('hook', [False, True])
def test_one_rank_waits_for_nobody(hook):
    """The statistics of the time spent waiting for each source stay as they are."""
    import deepep_b200
    from deepep_b200.parallel.local_cluster import SingleProcessGroup
    T, H, E, K = 16, 512, 8, 2
    buf = deepep_b200.Buffer(SingleProcessGroup(), num_rdma_bytes=deepep_b200.Buffer.get_low_latency_rdma_size_hint(T, H, 1, E), low_latency_mode=True,
                             num_gpu_timeout_secs=5)
    (x,), (idx,), (w,) = make_routed_inputs(1, T, H, E, K, seed=2, device='cuda')
    for shape in ((1,), (1, 1)):
        a, b = torch.full(shape, 7, dtype=torch.int64, device='cuda'), torch.full(shape, 9, dtype=torch.int64, device='cuda')
        rows, _, handle, _, recv = buf.low_latency_dispatch(x, idx, T, E, use_fp8=False, dispatch_wait_recv_cost_stats=a, return_recv_hook=hook)
        if hook:
            recv()
        _, _, recv = buf.low_latency_combine(rows, idx, w, handle, combine_wait_recv_cost_stats=b, return_recv_hook=hook)
        if hook:
            recv()
        assert (a == 7).all() and (b == 9).all()
    buf.destroy()
