// One rank's MoE layer, forward and backward, as one native call each (FusedMoE of models/moe.py): router, dispatch, expert
// GEMMs, combine. A training iteration of a small layer launches some twenty kernels of 2 to 30 us; issued one by one from
// Python, through two autograd functions, the host took longer than the GPU (1000 tokens, hidden 2048, 8 experts: 398 us
// per iteration of which the GPU worked 270).
#include <c10/cuda/CUDAGuard.h>
#include <pybind11/stl.h>
#include <torch/extension.h>

#include "ops_runtime.hpp"
#include "runtime.hpp"
#include "tensors.hpp"

namespace py = pybind11;

namespace ep {

namespace {

using OptTensor = std::optional<at::Tensor>;

struct LayerConfig {
    int num_experts = 0, num_topk = 0, num_max_tokens = 0, expert_alignment = 1, num_sms = 0, fuse_reduce = 1;
    bool fp8 = false, pow2 = false, allow_multiple_reduction = true;
};

// what the backward pass needs of the forward pass (the input aside)
struct LayerCall {
    LayerConfig cfg;
    at::Tensor router, topk_idx, topk_weights, h1, ends;
    DispatchResult d;
};

CombineArgs combine_args(const LayerCall& c, const at::Tensor& rows, const OptTensor& weights) {
    CombineArgs a;
    a.x = rows;
    a.topk_weights = weights;
    a.recv_src_metadata = c.d.recv_src_metadata;
    a.topk_idx = c.topk_idx;
    a.psum_rank = c.d.psum_rank;
    a.dst_slot = c.d.token_slot;
    if (c.d.count_matrix.defined()) a.count_matrix = c.d.count_matrix;
    a.num_experts = c.cfg.num_experts;
    a.num_max_tokens = c.cfg.num_max_tokens;
    a.num_sms = c.d.num_sms;
    a.do_expand = true;
    a.allow_multiple_reduction = c.cfg.allow_multiple_reduction;
    a.fuse_reduce = c.cfg.fuse_reduce;
    return a;
}

// `weights`: (w13, w2) in bf16, or (w13_q, w13_sf, w2_q, w2_sf) for e4m3
std::tuple<at::Tensor, std::shared_ptr<LayerCall>> layer_forward(const std::shared_ptr<Runtime>& rt, const LayerConfig& cfg, const at::Tensor& input,
                                                                 const at::Tensor& router, const std::vector<at::Tensor>& weights) {
    c10::cuda::CUDAGuard guard(input.device());
    auto c = std::make_shared<LayerCall>();
    c->cfg = cfg;
    const at::Tensor x = input.contiguous();
    std::tie(c->topk_idx, c->topk_weights, c->router) = router_forward(x, router.contiguous(), cfg.num_topk);

    std::vector<DispatchArgs> args(1);
    DispatchArgs& a = args[0];
    a.x = x;
    a.topk_idx = c->topk_idx;
    a.topk_weights = c->topk_weights;
    a.num_experts = cfg.num_experts;
    a.num_max_tokens = cfg.num_max_tokens;
    a.expert_alignment = cfg.expert_alignment;
    a.num_sms = cfg.num_sms;
    a.quant_mode = cfg.fp8 ? (cfg.pow2 ? kQuantE4M3Pow2 : kQuantE4M3) : kQuantNone;
    a.do_expand = true;
    a.do_zero_padding = !cfg.fp8;       // (the backward pass contracts over the rows of x; with e4m3 it makes its own zeros)
    a.defer_counts = true;
    c->d = std::move(Runtime::dispatch({rt}, args)[0]);
    DispatchResult& d = c->d;
    const int el = static_cast<int>(d.num_unaligned.size(0));
    c->ends = first_rows(d.psum_expert, el);

    auto gemm = [&](const at::Tensor& rows, const OptTensor& sf, int w) {
        const OptTensor wsf = cfg.fp8 ? OptTensor(weights[w + 1]) : std::nullopt;
        return gemm_impl(rows, weights[w], sf, wsf, c->ends, cfg.expert_alignment, std::nullopt, 0, cfg.pow2, /*zero_gap=*/false);
    };
    c->h1 = gemm(d.recv_x, d.recv_sf, 0);
    const auto [act, act_sf] = swiglu(c->h1, d.recv_topk_weights, std::nullopt, cfg.fp8, cfg.pow2, c->ends, cfg.expert_alignment);
    std::vector<CombineArgs> back{combine_args(*c, gemm(act, act_sf, cfg.fp8 ? 2 : 1), std::nullopt)};
    at::Tensor y = Runtime::combine({rt}, back)[0].combined_x;

    if (d.counts_pending) {         // the whole pass is queued: now the host may wait for the row counts
        std::tie(d.num_recv_tokens, d.num_expanded_tokens, d.num_recv_tokens_per_expert_list) = rt->take_counts(el);
        d.counts_pending = false;
        const int64_t rows = d.num_expanded_tokens;
        d.recv_x = first_rows(d.recv_x, rows);
        if (d.recv_sf.has_value()) d.recv_sf = first_rows(*d.recv_sf, rows);
        d.recv_topk_weights = first_rows(*d.recv_topk_weights, rows);
        c->h1 = first_rows(c->h1, rows);
        d.recv_src_metadata = first_rows(d.recv_src_metadata, d.num_recv_tokens);
    }
    return {y, c};
}

// (dx, d router, dW13, dW2) from dy and the transposed weights
std::tuple<at::Tensor, at::Tensor, at::Tensor, at::Tensor> layer_backward(const std::shared_ptr<Runtime>& rt, const std::shared_ptr<LayerCall>& c, const at::Tensor& x,
                                                                          const at::Tensor& dy, const at::Tensor& w13_t, const at::Tensor& w2_t) {
    c10::cuda::CUDAGuard guard(x.device());
    const LayerConfig& cfg = c->cfg;
    const DispatchResult& d = c->d;
    // the gradient of the combine (a sum) replays the dispatch with dy as payload
    std::vector<DispatchArgs> args(1);
    DispatchArgs& a = args[0];
    a.x = dy.contiguous();
    a.topk_idx = c->topk_idx;
    a.num_experts = cfg.num_experts;
    a.num_max_tokens = cfg.num_max_tokens;
    a.expert_alignment = cfg.expert_alignment;
    a.num_sms = cfg.num_sms;
    a.do_expand = a.do_zero_padding = true;
    a.do_cpu_sync = false;
    a.cached = true;
    a.h_token_slot = d.token_slot;
    a.h_pair_row = d.pair_row;
    a.h_psum_rank = d.psum_rank;
    a.h_psum_expert = d.psum_expert;
    a.h_num_unaligned = d.num_unaligned;
    a.h_recv_src_metadata = d.recv_src_metadata;
    a.h_num_recv_tokens = d.num_recv_tokens;
    a.h_num_expanded_tokens = d.num_expanded_tokens;
    const at::Tensor dh2 = Runtime::dispatch({rt}, args)[0].recv_x;

    const int el = static_cast<int>(w13_t.size(0)), align = cfg.expert_alignment;
    const at::Tensor x_rows = cfg.fp8 ? dequant_1x128(d.recv_x, *d.recv_sf, c->ends, align) : d.recv_x;
    auto data_gradient = [&](const at::Tensor& rows, const at::Tensor& w) {
        return gemm_impl(rows, w, std::nullopt, std::nullopt, c->ends, align, std::nullopt, 0, false, /*zero_gap=*/false);
    };
    const auto [dh1, act, dw_row] = swiglu_backward(c->h1, data_gradient(dh2, w2_t), d.recv_topk_weights, true, c->ends, align);
    const at::Tensor dx_rows = data_gradient(dh1, w13_t);
    at::Tensor d2 = gemm_k_grouped(dh2, act, c->ends, el, align, std::nullopt, 0, true);
    at::Tensor d13 = gemm_k_grouped(dh1, x_rows, c->ends, el, align, std::nullopt, 0, true);
    // the gradient of the dispatch is a combine, which carries the gradients of the gate weights back as well
    std::vector<CombineArgs> back{combine_args(*c, dx_rows, dw_row)};
    const CombineResult r = Runtime::combine({rt}, back)[0];
    at::Tensor d_router = router_backward(x.contiguous(), c->router, c->topk_idx, c->topk_weights, *r.combined_topk_weights, cfg.num_experts, r.combined_x);
    return {r.combined_x, d_router, d13, d2};
}

}  // namespace

void register_moe_bindings(py::module_& m) {
    py::class_<LayerCall, std::shared_ptr<LayerCall>>(m, "MoELayerCall");
    py::class_<LayerConfig>(m, "MoELayerConfig")
        .def(py::init([](int num_experts, int num_topk, int num_max_tokens, int expert_alignment, int num_sms, bool fp8, bool pow2, bool allow_multiple_reduction,
                         int fuse_reduce) {
            return LayerConfig{num_experts, num_topk, num_max_tokens, expert_alignment, num_sms, fuse_reduce, fp8, pow2, allow_multiple_reduction};
        }), py::arg("num_experts"), py::arg("num_topk"), py::arg("num_max_tokens"), py::arg("expert_alignment"), py::arg("num_sms"), py::arg("fp8"),
            py::arg("pow2"), py::arg("allow_multiple_reduction"), py::arg("fuse_reduce"));
    // (both may wait on the host for peers or counts: without the GIL, like dispatch and combine)
    m.def("moe_layer_forward", &layer_forward, py::call_guard<py::gil_scoped_release>());
    m.def("moe_layer_backward", &layer_backward, py::call_guard<py::gil_scoped_release>());
}

}  // namespace ep
