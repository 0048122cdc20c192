// Host drivers of the low-latency dispatch / combine kernels and of the rank-mask API.
//
// Parity: csrc/legacy/buffer.hpp:1431-1748 of the reference (clean_low_latency_buffer,
// low_latency_dispatch, low_latency_combine, get_next_low_latency_combine_buffer, mask API) and
// csrc/legacy/config.hpp:122-188 (LowLatencyLayout, size hint).
#include <ATen/ops/empty.h>
#include <ATen/ops/from_blob.h>
#include <pybind11/stl.h>
#include <torch/extension.h>

#include "py_tuples.hpp"
#include "runtime.hpp"
#include "stream_scope.hpp"

namespace py = pybind11;

namespace ep {

namespace {

struct LLDispatchIO {
    at::Tensor x, topk_idx;
    std::optional<at::Tensor> cumulative_stats, wait_stats;
    // outputs (allocated by the first call, passed again by the receive hook)
    at::Tensor packed_recv_x, packed_recv_count, src_info, layout_range;
    std::optional<at::Tensor> packed_recv_sf;
};

struct LLCombineIO {
    at::Tensor x, topk_idx, topk_weights, src_info, layout_range, combined_x;
    std::optional<at::Tensor> wait_stats;
    bool use_logfmt = false;   // send rows in the 10-bit log format (same for all emulated ranks of a call)
};

int64_t ll_buffer_size(int num_ranks, int num_max_tokens, int hidden, int num_experts) {
    return static_cast<int64_t>(ll_layout(num_ranks, num_max_tokens, hidden, num_experts).end);
}

// Launch-stream policy of the low-latency calls: a call that hands back an event runs on the communication stream, every
// other one on the caller's stream (with a receive hook the caller overlaps the kernels itself; a synchronous call would
// only go over the communication stream and back).
struct LLStreams {
    at::cuda::CUDAStream compute, launch;
    Runtime& runtime;
    LLStreams(Runtime& rt, bool async_finish, bool use_compute)
        : compute(at::cuda::getCurrentCUDAStream()), launch(async_finish && !use_compute ? rt.comm_stream() : compute), runtime(rt) {
        if (launch != compute) stream_wait(launch, compute);
        rt.order_behind_last_call(launch, compute);
    }
    std::optional<EventHandle> finish(bool async_finish) {
        runtime.call_ended(launch, std::nullopt);
        if (async_finish) return EventHandle(launch);
        return std::nullopt;
    }
};

std::optional<EventHandle> ll_dispatch(const std::vector<std::shared_ptr<Runtime>>& rts, std::vector<LLDispatchIO*>& ios,
                                       int num_max_tokens, int num_experts, bool use_fp8, bool round_scale, bool use_ue8m0,
                                       int phases, int num_sms, bool shrink, bool async_finish, bool on_compute_stream) {
    const int V = static_cast<int>(rts.size());
    EP_HOST_ASSERT(V >= 1 && V <= kMaxVRanks && static_cast<int>(ios.size()) == V);
    auto& rt0 = *rts[0];
    const int device = rt0.heap().device();
    c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(device));
    LLStreams streams(rt0, async_finish, on_compute_stream);
    const int R = rt0.num_ranks();
    const int H = static_cast<int>(ios[0]->x.size(1)), K = static_cast<int>(ios[0]->topk_idx.size(1));
    const int E = num_experts, EL = E / R, Tm = num_max_tokens;
    EP_HOST_ASSERT(E % R == 0 && E <= kMaxExperts && EL <= kMaxLocalExperts && K <= kMaxLLTopk && Tm >= 1 && Tm < 65536);
    EP_HOST_ASSERT_MSG(H % 128 == 0 && H <= 8192, "low-latency dispatch needs hidden % 128 == 0 and hidden <= 8192");
    if (use_ue8m0) EP_HOST_ASSERT_MSG(round_scale && use_fp8 && H % 512 == 0, "UE8M0 scales need round_scale, FP8 and hidden % 512 == 0");
    const LLLayout lay = ll_layout(R, Tm, H, E);
    EP_HOST_ASSERT_MSG(lay.end <= rt0.heap().num_bytes(), "symmetric buffer too small for low-latency mode");
    if (num_sms <= 0) num_sms = rt0.num_device_sms();   // latency-bound: one token / one (expert, source) pair per block
    if (num_sms * V > rt0.num_device_sms()) num_sms = rt0.num_device_sms() / V;

    Multi<LLDispatchParams> m;
    m.num_vranks = V;
    m.blocks_per_rank = num_sms;
    for (int v = 0; v < V; ++v) {
        auto& rt = *rts[v];
        auto& io = *ios[v];
        EP_HOST_ASSERT(io.x.scalar_type() == at::kBFloat16 && io.x.is_contiguous() && io.x.size(1) == H && io.x.size(0) <= Tm);
        EP_HOST_ASSERT((io.topk_idx.scalar_type() == at::kLong || io.topk_idx.scalar_type() == at::kInt) && io.topk_idx.is_contiguous() && io.topk_idx.size(0) == io.x.size(0) && io.topk_idx.size(1) == K);
        if (!io.packed_recv_x.defined()) {
            io.packed_recv_x = new_tensor({EL, R * Tm, H}, use_fp8 ? at::kFloat8_e4m3fn : at::kBFloat16, device);
            const int64_t rows = static_cast<int64_t>(R) * Tm;
            TensorPack pack(TensorPack::room(EL, 4) + TensorPack::room(EL * rows, 4) + TensorPack::room(EL * R, 8), device);
            io.packed_recv_count = pack.take({EL}, at::kInt);
            io.src_info = pack.take({EL, rows}, at::kInt);
            io.layout_range = pack.take({EL, R}, at::kLong);
            if (use_fp8) {
                const int64_t packs = use_ue8m0 ? H / 512 : H / 128;
                io.packed_recv_sf = new_strided({EL, rows, packs}, {packs * rows, 1, rows}, use_ue8m0 ? at::kInt : at::kFloat, device);
            }
        }
        LLDispatchParams& p = m.r[v];
        p.c = rt.ctx();
        p.num_tokens = static_cast<int>(io.x.size(0));
        p.hidden = H;
        p.num_topk = K;
        p.num_experts = E;
        p.num_local_experts = EL;
        p.num_max_tokens = Tm;
        p.use_fp8 = use_fp8;
        p.round_scale = round_scale;
        p.use_ue8m0 = use_ue8m0;
        p.phases = phases;
        p.shrink = shrink;
        p.x = static_cast<const uint8_t*>(io.x.data_ptr());
        p.topk_idx = io.topk_idx.data_ptr();
        p.idx32 = io.topk_idx.scalar_type() == at::kInt ? 1 : 0;
        p.packed_recv_x = static_cast<uint8_t*>(io.packed_recv_x.data_ptr());
        p.packed_recv_sf = io.packed_recv_sf.has_value() ? static_cast<uint8_t*>(io.packed_recv_sf->data_ptr()) : nullptr;
        p.packed_recv_src_info = io.src_info.data_ptr<int>();
        p.packed_recv_layout_range = io.layout_range.data_ptr<int64_t>();
        p.packed_recv_count = io.packed_recv_count.data_ptr<int>();
        p.cumulative_stats = io.cumulative_stats.has_value() ? io.cumulative_stats->data_ptr<int>() : nullptr;
        p.wait_stats = io.wait_stats.has_value() ? io.wait_stats->data_ptr<int64_t>() : nullptr;
        for (int h = 0; h < 2; ++h) {
            p.off_recv_x[h] = lay.recv_x[h];
            p.off_recv_count[h] = lay.recv_count[h];
        }
    }
    if (R == 1 && V == 1) {
        // one rank: both phases are one local kernel, a receive call has nothing left to do
        if (phases & kLLSend) CUDA_RUNTIME_CHECK(launch_ll_local_dispatch(m.r[0], num_sms, rt0.use_pdl(), streams.launch.stream()));
    } else {
        CUDA_RUNTIME_CHECK(launch_ll_dispatch(m, num_sms, streams.launch.stream()));
    }
    return streams.finish(async_finish);
}

std::optional<EventHandle> ll_combine(const std::vector<std::shared_ptr<Runtime>>& rts, std::vector<LLCombineIO*>& ios,
                                      int num_max_tokens, int num_experts, int phases, int num_sms, bool shrink,
                                      bool async_finish, bool on_compute_stream) {
    const int V = static_cast<int>(rts.size());
    EP_HOST_ASSERT(V >= 1 && V <= kMaxVRanks && static_cast<int>(ios.size()) == V);
    auto& rt0 = *rts[0];
    const int device = rt0.heap().device();
    c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(device));
    LLStreams streams(rt0, async_finish, on_compute_stream);
    const int R = rt0.num_ranks();
    const int H = static_cast<int>(ios[0]->x.size(2)), K = static_cast<int>(ios[0]->topk_idx.size(1));
    const int E = num_experts, EL = E / R, Tm = num_max_tokens;
    EP_HOST_ASSERT(E % R == 0 && K <= kMaxLLTopk && K <= kMaxTopk && (H * 2) % 16 == 0);
    EP_HOST_ASSERT_MSG(!ios[0]->use_logfmt || H % 128 == 0, "LogFMT needs a hidden size that is a multiple of 128");
    const LLLayout lay = ll_layout(R, Tm, H, E);
    EP_HOST_ASSERT_MSG(lay.end <= rt0.heap().num_bytes(), "symmetric buffer too small for low-latency mode");
    const bool limited = num_sms > 0;
    if (num_sms <= 0) num_sms = rt0.num_device_sms();   // latency-bound: one token / one (expert, source) pair per block
    if (num_sms * V > rt0.num_device_sms()) num_sms = rt0.num_device_sms() / V;

    Multi<LLCombineParams> m;
    m.num_vranks = V;
    m.blocks_per_rank = num_sms;
    for (int v = 0; v < V; ++v) {
        auto& rt = *rts[v];
        auto& io = *ios[v];
        EP_HOST_ASSERT(io.x.scalar_type() == at::kBFloat16 && io.x.is_contiguous() && io.x.dim() == 3 && io.x.size(0) == EL &&
                       io.x.size(1) == R * Tm && io.x.size(2) == H);
        EP_HOST_ASSERT((io.topk_idx.scalar_type() == at::kLong || io.topk_idx.scalar_type() == at::kInt) && io.topk_idx.is_contiguous());
        EP_HOST_ASSERT(io.topk_weights.scalar_type() == at::kFloat && io.topk_weights.is_contiguous() && io.topk_weights.size(1) == K);
        const int T = static_cast<int>(io.topk_idx.size(0));
        if (!io.combined_x.defined()) io.combined_x = new_tensor({T, H}, at::kBFloat16, device);
        EP_HOST_ASSERT(io.combined_x.scalar_type() == at::kBFloat16 && io.combined_x.is_contiguous() && io.combined_x.size(0) == T && io.combined_x.size(1) == H);
        LLCombineParams& p = m.r[v];
        p.c = rt.ctx();
        p.num_tokens = T;
        p.hidden = H;
        p.num_topk = K;
        p.num_experts = E;
        p.num_local_experts = EL;
        p.num_max_tokens = Tm;
        p.phases = phases;
        p.shrink = shrink;
        p.use_logfmt = ios[0]->use_logfmt ? 1 : 0;
        p.x = static_cast<const uint8_t*>(io.x.data_ptr());
        p.topk_idx = io.topk_idx.data_ptr();
        p.idx32 = io.topk_idx.scalar_type() == at::kInt ? 1 : 0;
        p.topk_weights = io.topk_weights.data_ptr<float>();
        p.src_info = io.src_info.data_ptr<int>();
        p.layout_range = io.layout_range.data_ptr<int64_t>();
        p.combined_x = static_cast<uint8_t*>(io.combined_x.data_ptr());
        p.wait_stats = io.wait_stats.has_value() ? io.wait_stats->data_ptr<int64_t>() : nullptr;
        for (int h = 0; h < 2; ++h) {
            p.off_combine_x[h] = lay.combine_x[h];
            p.off_combine_flag[h] = lay.combine_flag[h];
        }
    }
    if (R == 1 && V == 1 && !ios[0]->use_logfmt) {
        if (phases & kLLSend) CUDA_RUNTIME_CHECK(launch_ll_local_combine(m.r[0], num_sms, limited, rt0.use_pdl(), streams.launch.stream()));
    } else {
        CUDA_RUNTIME_CHECK(launch_ll_combine(m, num_sms, rt0.smem_optin(), streams.launch.stream()));
    }
    return streams.finish(async_finish);
}

// The calls of one process (one rank) without an IO object on the Python side: one trip into native code.
py::tuple ll_dispatch_one(const std::shared_ptr<Runtime>& rt, py::tuple call) {
    const TupleReader t(call.ptr(), 12);
    LLDispatchIO io;
    io.x = t.tensor(0);
    io.topk_idx = t.tensor(1);
    io.cumulative_stats = t.maybe_tensor(2);
    io.wait_stats = t.maybe_tensor(3);
    std::vector<LLDispatchIO*> ios = {&io};
    const auto event = ll_dispatch({rt}, ios, t.integer(4), t.integer(5), t.flag(6), t.flag(7), t.flag(8), kLLSend | kLLRecv, t.integer(9), t.flag(10), t.flag(11), false);
    TupleWriter out(6);
    out.put(io.packed_recv_x).put(io.packed_recv_sf).put(io.packed_recv_count).put(io.src_info).put(io.layout_range).put(event);
    return out.take();
}

py::tuple ll_combine_one(const std::shared_ptr<Runtime>& rt, py::tuple call) {
    const TupleReader t(call.ptr(), 13);
    LLCombineIO io;
    io.x = t.tensor(0);
    io.topk_idx = t.tensor(1);
    io.topk_weights = t.tensor(2);
    io.src_info = t.tensor(3);
    io.layout_range = t.tensor(4);
    if (!t.none(5)) io.combined_x = t.tensor(5);
    io.wait_stats = t.maybe_tensor(6);
    io.use_logfmt = t.flag(9);
    std::vector<LLCombineIO*> ios = {&io};
    const auto event = ll_combine({rt}, ios, t.integer(7), t.integer(8), kLLSend | kLLRecv, t.integer(10), t.flag(11), t.flag(12), false);
    TupleWriter out(2);
    out.put(io.combined_x).put(event);
    return out.take();
}

// bf16 [EL, R * T_max, H] view of the staging half that the NEXT combine send may read from
at::Tensor ll_next_combine_buffer(Runtime& rt, int num_max_tokens, int hidden, int num_experts) {
    const int R = rt.num_ranks(), EL = num_experts / R;
    const LLLayout lay = ll_layout(R, num_max_tokens, hidden, num_experts);
    EP_HOST_ASSERT(lay.end <= rt.heap().num_bytes());
    uint64_t calls = 0;
    CUDA_RUNTIME_CHECK(cudaMemcpy(&calls, rt.local_ws() + kWsLLCalls + 2, sizeof(calls), cudaMemcpyDeviceToHost));
    const int half = static_cast<int>((calls + 1) & 1);
    return at::from_blob(rt.heap().base() + lay.send_x[half], {EL, R * num_max_tokens, hidden}, opts(at::kBFloat16, rt.heap().device()));
}

void ll_mask_update(Runtime& rt, int rank, bool mask) {
    CUDA_RUNTIME_CHECK(ll_update_mask(rt.local_ws(), rank, mask ? 1 : 0, at::cuda::getCurrentCUDAStream().stream()));
}
void ll_mask_clean(Runtime& rt) {
    CUDA_RUNTIME_CHECK(ll_update_mask(rt.local_ws(), -1, 0, at::cuda::getCurrentCUDAStream().stream()));
}
void ll_mask_query(Runtime& rt, at::Tensor out) {
    EP_HOST_ASSERT(out.scalar_type() == at::kInt && out.is_cuda() && out.numel() >= rt.num_ranks());
    CUDA_RUNTIME_CHECK(ll_query_mask(rt.local_ws(), out.data_ptr<int>(), rt.num_ranks(), at::cuda::getCurrentCUDAStream().stream()));
}

// Routing layout of `topk_idx` on the communication stream (legacy Buffer.get_dispatch_layout).
std::tuple<at::Tensor, at::Tensor, at::Tensor, std::optional<EventHandle>> get_dispatch_layout(
    Runtime& rt, const at::Tensor& topk_idx, int num_experts, std::optional<EventHandle> previous_event, bool async_finish,
    bool allocate_on_comm_stream) {
    EP_HOST_ASSERT(topk_idx.dim() == 2 && topk_idx.is_contiguous() && (topk_idx.scalar_type() == at::kLong || topk_idx.scalar_type() == at::kInt) && topk_idx.is_cuda());
    EP_HOST_ASSERT(num_experts > 0 && num_experts % rt.num_ranks() == 0 && num_experts <= kMaxExperts);
    const int device = rt.heap().device();
    c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(device));
    const auto compute = at::cuda::getCurrentCUDAStream();
    const auto comm = rt.comm_stream();
    if (allocate_on_comm_stream) at::cuda::setCurrentCUDAStream(comm);
    // (it touches nothing of the runtime: a synchronous query stays on the caller's stream)
    const bool stay = !async_finish && !allocate_on_comm_stream && !previous_event.has_value();
    const auto launch = stay ? compute : comm;
    if (previous_event.has_value()) previous_event->stream_wait(comm);
    else if (!stay) stream_wait(comm, compute);
    const int T = static_cast<int>(topk_idx.size(0)), K = static_cast<int>(topk_idx.size(1)), R = rt.num_ranks();
    TensorPack pack(TensorPack::room(R, 4) + TensorPack::room(num_experts, 4) + TensorPack::room(static_cast<int64_t>(T) * R, 1), device);
    auto per_rank = pack.take({R}, at::kInt), per_expert = pack.take({num_experts}, at::kInt), in_rank = pack.take({T, R}, at::kBool);
    CUDA_RUNTIME_CHECK(launch_dispatch_layout(topk_idx.data_ptr(), topk_idx.scalar_type() == at::kInt, T, K, R, num_experts, per_rank.data_ptr<int>(),
                                              per_expert.data_ptr<int>(), in_rank.data_ptr<bool>(), launch.stream()));
    std::optional<EventHandle> event;
    if (async_finish) {
        event = EventHandle(comm);
        for (const auto& t : {topk_idx, per_rank, per_expert, in_rank}) {
            t.record_stream(comm);
            if (allocate_on_comm_stream) t.record_stream(compute);
        }
    } else if (!stay) {
        stream_wait(compute, comm);
    }
    if (allocate_on_comm_stream) at::cuda::setCurrentCUDAStream(compute);
    return {per_rank, per_expert, in_rank, event};
}

// (rank_prefix_matrix, channel_prefix_matrix, recv_channel_prefix_matrix, send_head, is_token_in_rank) of the
// first-generation handle, on the current stream
std::tuple<at::Tensor, at::Tensor, at::Tensor, at::Tensor, std::optional<at::Tensor>> legacy_handle(Runtime& rt, const at::Tensor& count_matrix,
                                                                                                    const at::Tensor& token_slot, bool with_in_rank) {
    const int R = rt.num_ranks(), T = static_cast<int>(token_slot.size(0)), device = rt.heap().device();
    EP_HOST_ASSERT(count_matrix.is_contiguous() && count_matrix.numel() == R * R && token_slot.is_contiguous() && token_slot.size(1) == R);
    c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(device));
    const int64_t slots = static_cast<int64_t>(T) * R;
    TensorPack pack(TensorPack::room(R * R, 4) + 2 * TensorPack::room(R, 4) + TensorPack::room(slots, 4) + TensorPack::room(slots, 1), device);
    auto prefix = pack.take({R, R}, at::kInt), sent = pack.take({R, 1}, at::kInt), received = pack.take({R, 1}, at::kInt), send_head = pack.take({T, R}, at::kInt);
    std::optional<at::Tensor> in_rank;
    if (with_in_rank) in_rank = pack.take({T, R}, at::kBool);
    CUDA_RUNTIME_CHECK(launch_legacy_handle(count_matrix.data_ptr<int>(), token_slot.data_ptr<int>(), rt.rank(), R, T, prefix.data_ptr<int>(),
                                            sent.data_ptr<int>(), received.data_ptr<int>(), send_head.data_ptr<int>(),
                                            with_in_rank ? in_rank->data_ptr<bool>() : nullptr, at::cuda::getCurrentCUDAStream().stream()));
    return {prefix, sent, received, send_head, in_rank};
}

}  // namespace

void register_ll_bindings(py::module_& m) {
    py::class_<LLDispatchIO>(m, "LLDispatchIO")
        .def(py::init<>())
        .def_readwrite("x", &LLDispatchIO::x)
        .def_readwrite("topk_idx", &LLDispatchIO::topk_idx)
        .def_readwrite("cumulative_stats", &LLDispatchIO::cumulative_stats)
        .def_readwrite("wait_stats", &LLDispatchIO::wait_stats)
        .def_readwrite("packed_recv_x", &LLDispatchIO::packed_recv_x)
        .def_readwrite("packed_recv_sf", &LLDispatchIO::packed_recv_sf)
        .def_readwrite("packed_recv_count", &LLDispatchIO::packed_recv_count)
        .def_readwrite("src_info", &LLDispatchIO::src_info)
        .def_readwrite("layout_range", &LLDispatchIO::layout_range);
    py::class_<LLCombineIO>(m, "LLCombineIO")
        .def(py::init<>())
        .def_readwrite("x", &LLCombineIO::x)
        .def_readwrite("topk_idx", &LLCombineIO::topk_idx)
        .def_readwrite("topk_weights", &LLCombineIO::topk_weights)
        .def_readwrite("src_info", &LLCombineIO::src_info)
        .def_readwrite("layout_range", &LLCombineIO::layout_range)
        .def_readwrite("combined_x", &LLCombineIO::combined_x)
        .def_readwrite("wait_stats", &LLCombineIO::wait_stats)
        .def_readwrite("use_logfmt", &LLCombineIO::use_logfmt);
    m.def("get_dispatch_layout", &get_dispatch_layout);
    m.def("legacy_handle", &legacy_handle);
    m.def("ll_buffer_size", &ll_buffer_size);
    m.def("ll_dispatch", &ll_dispatch);
    m.def("ll_combine", &ll_combine);
    m.def("ll_dispatch_one", &ll_dispatch_one);
    m.def("ll_combine_one", &ll_combine_one);
    m.def("ll_next_combine_buffer", &ll_next_combine_buffer);
    m.def("ll_mask_update", &ll_mask_update);
    m.def("ll_mask_clean", &ll_mask_clean);
    m.def("ll_mask_query", &ll_mask_query);
    m.attr("LL_SEND") = static_cast<int>(kLLSend);
    m.attr("LL_RECV") = static_cast<int>(kLLRecv);
}

}  // namespace ep
