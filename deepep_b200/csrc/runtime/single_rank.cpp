// Dispatch and combine drivers of a group of one rank (kernels/local_exchange.cu): the same arguments, checks and results
// as the multi-rank drivers (runtime.cpp), without the heap.
#include <ATen/ops/from_blob.h>

#include "runtime.hpp"
#include "stream_scope.hpp"

namespace ep {

namespace {

uint64_t* timeline_of(uint64_t* local_ws, int kernel) {
    return reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(local_ws) + kWsTimelineOffsetBytes) + 2 * kernel;
}

}  // namespace

DispatchResult Runtime::dispatch_single(DispatchArgs& a) {
    const int device = heap_->device();
    c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(device));
    StreamScope scope(a.sc, *this, /*may_stay=*/true);
    const cudaStream_t stream = scope.comm.stream();

    EP_HOST_ASSERT(a.topk_idx.has_value() && heap_->connected());
    const at::Tensor& topk_idx = *a.topk_idx;
    const int K = static_cast<int>(topk_idx.size(1)), H = static_cast<int>(a.x.size(1)), T = static_cast<int>(a.x.size(0));
    const int E = a.num_experts, T_max = a.num_max_tokens;
    EP_HOST_ASSERT(E > 0 && E <= kMaxExperts && E <= kMaxLocalExperts);
    EP_HOST_ASSERT(K >= 1 && K <= kMaxTopk && T_max > 0 && a.expert_alignment >= 1);
    const bool quant = a.quant_mode != kQuantNone;
    const int elem = static_cast<int>(a.x.element_size());
    if (quant) EP_HOST_ASSERT_MSG(a.x.scalar_type() == at::kBFloat16 && H % 128 == 0 && !a.sf.has_value(),
                                  "fused FP8 dispatch wants a bf16 input with hidden % 128 == 0 and no scales");
    else EP_HOST_ASSERT(a.x.scalar_type() == at::kBFloat16 || a.x.scalar_type() == at::kFloat8_e4m3fn);
    const int src_row_bytes = H * elem;
    const int x_row_bytes = quant ? H : src_row_bytes;
    const int sf_packs = quant ? H / 128 : (a.sf.has_value() ? static_cast<int>(a.sf->size(1)) : 0);
    EP_HOST_ASSERT_MSG(src_row_bytes % 16 == 0 && x_row_bytes % 16 == 0, "hidden bytes must be a multiple of 16");
    EP_HOST_ASSERT(sf_packs <= ceil_div(H, 128));
    const int rec_pitch = ht_record_pitch(x_row_bytes, sf_packs * 4, K);
    const HtLayout lay = ht_layout(1, T_max, H, K);
    EP_HOST_ASSERT_MSG(lay.end <= heap_->num_bytes(), "symmetric buffer too small for this dispatch");
    const at::ScalarType out_dtype = quant ? at::kFloat8_e4m3fn : a.x.scalar_type();
    const at::ScalarType idx_dtype = topk_idx.scalar_type();
    EP_HOST_ASSERT_MSG(idx_dtype == at::kLong || idx_dtype == at::kInt, "topk_idx must be int64 or int32");
    EP_HOST_ASSERT_MSG(a.num_sms > 0, "num_sms must be given (the Python front end fills in the SM model's value)");
    EP_HOST_ASSERT(a.x.dim() == 2 && a.x.is_cuda() && a.x.stride(1) == 1);
    EP_HOST_ASSERT((a.x.stride(0) * elem) % 16 == 0 && reinterpret_cast<uintptr_t>(a.x.data_ptr()) % 16 == 0);
    EP_HOST_ASSERT(topk_idx.is_contiguous() && T <= T_max && topk_idx.size(0) == T);
    if (a.topk_weights.has_value())
        EP_HOST_ASSERT(a.topk_weights->scalar_type() == at::kFloat && a.topk_weights->is_contiguous() && a.topk_weights->size(0) == T && a.topk_weights->size(1) == K);
    const bool has_sf = sf_packs > 0;
    if (has_sf && !quant) EP_HOST_ASSERT(a.sf->dim() == 2 && a.sf->size(0) == T && a.sf->element_size() == 4);
    const bool cached = a.cached;
    const bool sync = a.do_cpu_sync && !cached;

    DispatchResult r;
    r.num_sms = std::min(a.num_sms, num_device_sms_);
    const uint32_t epoch = dispatch_epoch + 1;
    prof_record(0, stream);
    if (cached) {
        EP_HOST_ASSERT(a.h_token_slot.has_value() && a.h_pair_row.has_value() && a.h_psum_rank.has_value() &&
                       a.h_psum_expert.has_value() && a.h_num_unaligned.has_value() && a.h_recv_src_metadata.has_value());
        EP_HOST_ASSERT(!a.cumulative_stats.has_value());
        r.token_slot = *a.h_token_slot;
        r.pair_row = *a.h_pair_row;
        r.psum_rank = *a.h_psum_rank;
        r.psum_expert = *a.h_psum_expert;
        r.num_unaligned = *a.h_num_unaligned;
        r.recv_src_metadata = *a.h_recv_src_metadata;
    } else {
        const int64_t idx_size = static_cast<int64_t>(c10::elementSize(idx_dtype)), pairs = static_cast<int64_t>(T) * K;
        TensorPack pack(2 * TensorPack::room(1, 4) + TensorPack::room(T, 4) + TensorPack::room(pairs, 4) + TensorPack::room(E + 1, 4) + TensorPack::room(E, 4) +
                        (a.copy_topk_idx ? TensorPack::room(pairs, idx_size) : 0), device);
        r.token_slot = pack.take({T, 1}, at::kInt);
        r.pair_row = pack.take({T, K}, at::kInt);
        r.psum_rank = pack.take({1}, at::kInt);
        r.psum_expert = pack.take({E + 1}, at::kInt);
        r.num_unaligned = pack.take({E}, at::kInt);
        r.count_matrix = pack.take({1, 1}, at::kInt);
        if (a.copy_topk_idx) r.topk_idx = pack.take({T, K}, idx_dtype);
        LocalPlanParams p = {};
        p.num_tokens = T;
        p.num_topk = K;
        p.num_experts = E;
        p.expert_alignment = a.expert_alignment;
        p.do_expand = a.do_expand;
        p.idx32 = idx_dtype == at::kInt ? 1 : 0;
        p.topk_idx = topk_idx.data_ptr();
        p.token_slot = r.token_slot.data_ptr<int>();
        p.pair_row = r.pair_row.data_ptr<int>();
        p.psum_rank = r.psum_rank.data_ptr<int>();
        p.psum_expert = r.psum_expert.data_ptr<int>();
        p.num_unaligned = r.num_unaligned.data_ptr<int>();
        p.count_matrix = r.count_matrix.data_ptr<int>();
        if (a.cumulative_stats.has_value()) {
            EP_HOST_ASSERT(a.cumulative_stats->scalar_type() == at::kInt && a.cumulative_stats->numel() == E && a.cumulative_stats->is_contiguous());
            p.recv_stats = a.cumulative_stats->data_ptr<int>();
        }
        p.host_counts = sync ? host_words_dev_ + kHostStatusWords : nullptr;
        p.epoch = epoch;
        p.timeline = timeline_of(local_ws_, kTlDispatch);
        p.stamps = local_ws_ + kWsStamps;
        CUDA_RUNTIME_CHECK(launch_local_plan(p, stream));
        ++num_launches_;
    }
    dispatch_epoch = epoch;

    // ---- sizes of the outputs
    const int worst_expanded = align_up(T_max * std::min(K, E) + E * (a.expert_alignment - 1), a.expert_alignment);
    auto read_counts = [&]() { std::tie(r.num_recv_tokens, r.num_expanded_tokens, r.num_recv_tokens_per_expert_list) = take_counts(E); };
    // The exact sizes are known when the plan kernel has run. The move kernel does not wait for the host to learn them:
    // it gets outputs that hold the most rows these tokens can have (every token, every pair plus the alignment gaps),
    // which are cut to their real length afterwards. Only where the row count is part of a stride (column-major scales) or
    // the bound is far off for an expanded output is the count awaited first.
    int rows_bound, idx_bound;
    bool cut = false;
    if (cached) {
        r.num_recv_tokens = a.h_num_recv_tokens;
        r.num_expanded_tokens = a.h_num_expanded_tokens;
        idx_bound = r.num_recv_tokens;
        rows_bound = a.do_expand ? r.num_expanded_tokens : r.num_recv_tokens;
    } else if (sync) {
        const int64_t expanded_bound = align_up<int64_t>(static_cast<int64_t>(T) * std::min(K, E) + static_cast<int64_t>(E) * (a.expert_alignment - 1), a.expert_alignment);
        cut = !(a.col_major_sf && has_sf) && expanded_bound * x_row_bytes < (1ll << 30);
        if (cut) {
            idx_bound = T;
            rows_bound = a.do_expand ? static_cast<int>(expanded_bound) : T;
        } else {
            read_counts();
            idx_bound = r.num_recv_tokens;
            rows_bound = a.do_expand ? r.num_expanded_tokens : r.num_recv_tokens;
        }
    } else {
        r.num_recv_tokens = a.num_worst_tokens > 0 ? a.num_worst_tokens : T_max;
        EP_HOST_ASSERT_MSG(r.num_recv_tokens <= T_max, "num_worst_tokens exceeds ranks x num_max_tokens_per_rank");
        r.num_expanded_tokens = worst_expanded;
        idx_bound = r.num_recv_tokens;
        rows_bound = a.do_expand ? r.num_expanded_tokens : r.num_recv_tokens;
    }

    const bool zero_copy = a.zero_copy && !a.do_expand;
    uint8_t* region = heap_->base() + lay.dispatch_rec[epoch & 1];
    if (zero_copy) r.recv_x = at::from_blob(region, {rows_bound, H}, {rec_pitch / static_cast<int64_t>(c10::elementSize(out_dtype)), 1}, opts(out_dtype, device));
    else r.recv_x = new_tensor({rows_bound, H}, out_dtype, device);
    if (has_sf) {
        const at::ScalarType sf_dtype = (!quant && a.sf->scalar_type() == at::kInt) ? at::kInt : at::kFloat;
        if (a.col_major_sf) {
            r.recv_sf = new_strided({rows_bound, sf_packs}, {1, align_up(std::max(rows_bound, 1), 4)}, sf_dtype, device);
        } else if (zero_copy) {
            r.recv_sf = at::from_blob(region + x_row_bytes, {rows_bound, sf_packs}, {rec_pitch / 4, 1}, opts(sf_dtype, device));
        } else {
            r.recv_sf = new_tensor({rows_bound, sf_packs}, sf_dtype, device);
        }
    }
    if (!a.do_expand) {
        r.recv_topk_idx = new_tensor({idx_bound, K}, idx_dtype, device);
        if (a.topk_weights.has_value()) r.recv_topk_weights = new_tensor({idx_bound, K}, at::kFloat, device);
    } else if (a.topk_weights.has_value()) {
        r.recv_topk_weights = new_tensor({rows_bound}, at::kFloat, device);
    }
    if (!cached) r.recv_src_metadata = new_tensor({idx_bound, K + 2}, at::kInt, device);

    LocalMoveParams q = {};
    q.num_tokens = T;
    q.num_topk = K;
    q.num_experts = E;
    q.expert_alignment = a.expert_alignment;
    q.do_expand = a.do_expand;
    q.do_zero_padding = a.do_zero_padding;
    q.write_metadata = cached ? 0 : 1;
    q.idx32 = idx_dtype == at::kInt ? 1 : 0;
    q.mask_weights = a.mask_weights ? 1 : 0;
    q.pow2 = a.quant_mode == kQuantE4M3Pow2;
    q.src_row_bytes = src_row_bytes;
    q.x = static_cast<const uint8_t*>(a.x.data_ptr());
    q.x_stride_bytes = a.x.stride(0) * elem;
    if (has_sf && !quant) {
        q.sf = static_cast<const uint32_t*>(a.sf->data_ptr());
        q.sf_token_stride = a.sf->stride(0);
        q.sf_pack_stride = a.sf->stride(1);
    }
    q.sf_packs = sf_packs;
    q.topk_idx = topk_idx.data_ptr();
    q.topk_idx_copy = r.topk_idx.has_value() ? r.topk_idx->data_ptr() : nullptr;
    q.topk_weights = a.topk_weights.has_value() ? a.topk_weights->data_ptr<float>() : nullptr;
    q.token_slot = r.token_slot.data_ptr<int>();
    q.pair_row = r.pair_row.data_ptr<int>();
    q.psum_rank = r.psum_rank.data_ptr<int>();
    q.psum_expert = r.psum_expert.data_ptr<int>();
    q.recv_x = static_cast<uint8_t*>(r.recv_x.data_ptr());
    q.recv_x_pitch = zero_copy ? rec_pitch : x_row_bytes;
    q.recv_sf = has_sf ? static_cast<uint32_t*>(r.recv_sf->data_ptr()) : nullptr;
    q.recv_sf_row_stride = has_sf ? r.recv_sf->stride(0) : 0;
    q.recv_sf_pack_stride = has_sf ? r.recv_sf->stride(1) : 0;
    q.recv_topk_idx = r.recv_topk_idx.has_value() ? r.recv_topk_idx->data_ptr() : nullptr;
    q.recv_topk_weights = r.recv_topk_weights.has_value() ? r.recv_topk_weights->data_ptr<float>() : nullptr;
    q.recv_src_metadata = r.recv_src_metadata.data_ptr<int>();
    q.num_out_rows = rows_bound;
    q.num_idx_rows = cached ? static_cast<int>(r.recv_src_metadata.size(0)) : idx_bound;
    q.timeline = timeline_of(local_ws_, kTlDispatch);
    const bool gated = a.sc.previous_event_before_epilogue.has_value();
    if (gated) a.sc.previous_event_before_epilogue->stream_wait(scope.comm);
    q.plan_ahead = !cached && !gated && use_pdl_ ? 1 : 0;
    CUDA_RUNTIME_CHECK(launch_local_move(q, quant, num_device_sms_, stream));
    ++num_launches_;
    prof_record(1, stream);
    prof_record(2, stream);
    prof_valid_[0] = profiling_ != 0;
    prof_split_[0] = profiling_ == 2;

    // the full-length tensors are what the streams have to know about; the views below share their memory
    std::vector<at::Tensor> touched;
    if (a.sc.async_with_compute_stream) {
        touched = {r.recv_x, r.token_slot, r.pair_row, r.psum_rank, r.psum_expert, r.num_unaligned, r.recv_src_metadata, a.x, topk_idx};
        for (const auto& t : {r.recv_sf, r.recv_topk_idx, r.recv_topk_weights, r.topk_idx, a.sf, a.topk_weights, a.cumulative_stats})
            if (t.has_value()) touched.push_back(*t);
    }
    if (cut && a.defer_counts) {
        r.counts_pending = true;
        r.num_recv_tokens = idx_bound;
        r.num_expanded_tokens = rows_bound;
    } else if (cut) {
        read_counts();
        const int rows = a.do_expand ? r.num_expanded_tokens : r.num_recv_tokens;
        auto shorten = [](at::Tensor& t, int n) { t = first_rows(t, n); };
        shorten(r.recv_x, rows);
        if (r.recv_sf.has_value()) shorten(*r.recv_sf, rows);
        if (r.recv_topk_idx.has_value()) shorten(*r.recv_topk_idx, r.num_recv_tokens);
        if (r.recv_topk_weights.has_value()) shorten(*r.recv_topk_weights, a.do_expand ? rows : r.num_recv_tokens);
        shorten(r.recv_src_metadata, r.num_recv_tokens);
    }
    r.event = scope.finish(a.sc, touched);
    return r;
}

std::tuple<int, int, std::vector<int>> Runtime::take_counts(int num_local_experts) {
    std::vector<int> per_expert(num_local_experts);
    const int tokens = wait_count(0, dispatch_epoch), rows = wait_count(1, dispatch_epoch);
    for (int e = 0; e < num_local_experts; ++e) per_expert[e] = wait_count(2 + e, dispatch_epoch);
    return {tokens, rows, std::move(per_expert)};
}

CombineResult Runtime::combine_single(CombineArgs& a) {
    const int device = heap_->device();
    c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(device));
    StreamScope scope(a.sc, *this, /*may_stay=*/true);
    const cudaStream_t stream = scope.comm.stream();

    const int K = static_cast<int>(a.topk_idx.size(1)), H = static_cast<int>(a.x.size(1)), T = static_cast<int>(a.topk_idx.size(0));
    const int E = a.num_experts, T_max = a.num_max_tokens;
    EP_HOST_ASSERT(heap_->connected());
    EP_HOST_ASSERT(a.x.scalar_type() == at::kBFloat16 && (H * 2) % 16 == 0);
    EP_HOST_ASSERT_MSG(ht_layout(1, T_max, H, K).end <= heap_->num_bytes(), "symmetric buffer too small for this combine");
    const at::ScalarType idx_dtype = a.topk_idx.scalar_type();
    EP_HOST_ASSERT_MSG(idx_dtype == at::kLong || idx_dtype == at::kInt, "topk_idx must be int64 or int32");
    EP_HOST_ASSERT_MSG(a.num_sms > 0, "num_sms must be given (the Python front end fills in the handle's value)");
    EP_HOST_ASSERT(a.x.dim() == 2 && a.x.is_cuda() && a.x.stride(1) == 1);
    EP_HOST_ASSERT((a.x.stride(0) * 2) % 16 == 0 && reinterpret_cast<uintptr_t>(a.x.data_ptr()) % 16 == 0);
    EP_HOST_ASSERT(a.recv_src_metadata.scalar_type() == at::kInt && a.recv_src_metadata.is_contiguous() && a.recv_src_metadata.size(1) == K + 2);
    EP_HOST_ASSERT(a.topk_idx.is_contiguous() && K <= kMaxTopk);
    EP_HOST_ASSERT(a.dst_slot.has_value() && a.dst_slot->scalar_type() == at::kInt && a.dst_slot->is_contiguous() && a.dst_slot->numel() == T);
    const bool weighted = a.weighted && a.do_expand;
    if (weighted) EP_HOST_ASSERT_MSG(a.topk_weights.has_value(), "a weighted combine needs the top-k weights of the expanded rows");
    if (a.topk_weights.has_value()) {
        EP_HOST_ASSERT(a.topk_weights->scalar_type() == at::kFloat && a.topk_weights->is_contiguous());
        if (a.do_expand) EP_HOST_ASSERT(a.topk_weights->dim() == 1);
        else EP_HOST_ASSERT(a.topk_weights->dim() == 2 && a.topk_weights->size(1) == K);
    }
    CombineResult r;
    r.combined_x = new_tensor({T, H}, at::kBFloat16, device);
    if (a.topk_weights.has_value()) r.combined_topk_weights = new_tensor({T, K}, at::kFloat, device);
    LocalCombineParams p = {};
    p.num_tokens = T;
    p.num_topk = K;
    p.num_experts = E;
    p.row_bytes = H * 2;
    p.do_expand = a.do_expand;
    p.weighted = weighted ? 1 : 0;
    p.idx32 = idx_dtype == at::kInt ? 1 : 0;
    p.round_partial = (!a.do_expand || a.allow_multiple_reduction) ? 1 : 0;
    p.num_x_rows = static_cast<int>(a.x.size(0));
    p.num_meta_rows = static_cast<int>(a.recv_src_metadata.size(0));
    p.x = static_cast<const uint8_t*>(a.x.data_ptr());
    p.x_stride_bytes = a.x.stride(0) * 2;
    p.topk_weights = a.topk_weights.has_value() ? a.topk_weights->data_ptr<float>() : nullptr;
    p.token_slot = a.dst_slot->data_ptr<int>();
    p.recv_src_metadata = a.recv_src_metadata.data_ptr<int>();
    p.topk_idx = a.topk_idx.data_ptr();
    const uint8_t** const bias_out[2] = {&p.bias0, &p.bias1};
    const std::optional<at::Tensor>* const bias_in[2] = {&a.bias0, &a.bias1};
    for (int i = 0; i < 2; ++i) {
        if (!bias_in[i]->has_value()) continue;
        const at::Tensor& b = **bias_in[i];
        EP_HOST_ASSERT(b.scalar_type() == at::kBFloat16 && b.is_contiguous() && b.size(0) == T && b.size(1) == H);
        *bias_out[i] = static_cast<const uint8_t*>(b.data_ptr());
    }
    p.combined_x = static_cast<uint8_t*>(r.combined_x.data_ptr());
    p.combined_topk_weights = r.combined_topk_weights.has_value() ? r.combined_topk_weights->data_ptr<float>() : nullptr;
    p.timeline = timeline_of(local_ws_, kTlCombine);
    if (a.sc.previous_event_before_epilogue.has_value()) a.sc.previous_event_before_epilogue->stream_wait(scope.comm);
    prof_record(3, stream);
    CUDA_RUNTIME_CHECK(launch_local_combine(p, num_device_sms_, stream));
    ++num_launches_;
    ++combine_epoch;
    prof_record(4, stream);
    prof_record(5, stream);
    prof_valid_[1] = profiling_ != 0;
    prof_split_[1] = profiling_ == 2;
    std::vector<at::Tensor> touched;
    if (a.sc.async_with_compute_stream) {
        touched = {r.combined_x, a.x, a.recv_src_metadata, a.topk_idx, a.psum_rank, *a.dst_slot};
        for (const auto& t : {r.combined_topk_weights, a.topk_weights, a.bias0, a.bias1})
            if (t.has_value()) touched.push_back(*t);
    }
    r.event = scope.finish(a.sc, touched);
    return r;
}

}  // namespace ep
