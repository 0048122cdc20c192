// PyTorch-facing wrappers of the compute kernels (tcgen05 GEMM family, and the small hot ops).
// The reference library has no compute kernels; these exist for the fused MoE layer and the
// tensor-parallel fused operators built on the same runtime.
#include <ATen/cuda/CUDAContext.h>
#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAGuard.h>
#include <pybind11/stl.h>
#include <torch/extension.h>

#include <optional>

#include "../common/exception.hpp"
#include "../common/layout.hpp"
#include "../kernels/gemm_api.hpp"
#include "../kernels/ops_api.hpp"
#include "ops_runtime.hpp"
#include "tensors.hpp"

namespace py = pybind11;

namespace ep {

namespace {

// A contiguous tensor that starts on a 16-byte boundary (the wide loads of the kernels); a view into a flat buffer may not.
at::Tensor on_16_bytes(const at::Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0 ? t : t.clone(); }

cudaStream_t cur_stream() { return at::cuda::getCurrentCUDAStream().stream(); }

// the status word of the GEMM pipelines on the current device (0 = healthy)
int* gemm_status() {
    int* word = nullptr;
    CUDA_RUNTIME_CHECK(gemm::status_word(&word));
    return word;
}

int gemm_check_status() {
    int value = 0;
    CUDA_RUNTIME_CHECK(cudaMemcpyAsync(&value, gemm_status(), sizeof(value), cudaMemcpyDeviceToHost, cur_stream()));
    CUDA_RUNTIME_CHECK(cudaStreamSynchronize(cur_stream()));
    return value;
}

}  // namespace

at::Tensor gemm_impl(const at::Tensor& a, const at::Tensor& b, const std::optional<at::Tensor>& sfa, const std::optional<at::Tensor>& sfb,
                     const std::optional<at::Tensor>& group_end, int group_alignment, std::optional<at::Tensor> out, int num_sms,
                     bool pow2_scales, bool zero_gap) {
    EP_HOST_ASSERT(a.is_cuda() && b.is_cuda() && a.dim() == 2 && a.stride(1) == 1 && b.stride(-1) == 1);
    EP_HOST_ASSERT(b.dim() == 2 || b.is_contiguous());
    const bool fp8 = a.scalar_type() == at::kFloat8_e4m3fn;
    EP_HOST_ASSERT(fp8 || a.scalar_type() == at::kBFloat16);
    EP_HOST_ASSERT(b.scalar_type() == a.scalar_type());
    const bool grouped = b.dim() == 3;
    EP_HOST_ASSERT(b.dim() == 2 || b.dim() == 3);
    const int G = grouped ? static_cast<int>(b.size(0)) : 1;
    const int N = static_cast<int>(b.size(grouped ? 1 : 0)), K = static_cast<int>(b.size(grouped ? 2 : 1));
    const int M = static_cast<int>(a.size(0));
    EP_HOST_ASSERT(a.size(1) == K);
    const int elem = fp8 ? 1 : 2;
    EP_HOST_ASSERT((a.stride(0) * elem) % 16 == 0 && reinterpret_cast<uintptr_t>(a.data_ptr()) % 16 == 0);
    EP_HOST_ASSERT_MSG(N % 128 == 0 && K % (fp8 ? 128 : 64) == 0, "N must be a multiple of 128 and K of 64 (bf16) / 128 (fp8)");
    const int device = a.get_device();
    c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(device));
    if (!out.has_value()) out = new_tensor({M, N}, at::kBFloat16, device);
    EP_HOST_ASSERT(out->scalar_type() == at::kBFloat16 && out->size(0) == M && out->size(1) == N && out->stride(1) == 1 &&
                   (out->stride(0) * 2) % 16 == 0);
    if (M == 0) return *out;

    gemm::GemmParams p = {};
    p.M = M;
    p.N = N;
    p.K = K;
    p.num_groups = G;
    p.group_end = nullptr;
    p.group_alignment = std::max(group_alignment, 1);
    p.zero_gap = (zero_gap && grouped && p.group_alignment % 128 == 0) ? 1 : 0;
    if (grouped) {
        EP_HOST_ASSERT(group_end.has_value() && group_end->scalar_type() == at::kInt && group_end->is_contiguous() && group_end->numel() >= G);
        p.group_end = group_end->data_ptr<int>();
    }
    p.C = reinterpret_cast<__nv_bfloat16*>(out->data_ptr());
    p.ldc = out->stride(0);
    if (fp8) {
        EP_HOST_ASSERT(sfa.has_value() && sfb.has_value() && sfa->scalar_type() == at::kFloat && sfb->scalar_type() == at::kFloat);
        EP_HOST_ASSERT(sfa->dim() == 2 && sfa->size(0) == M && sfa->size(1) == K / 128);
        EP_HOST_ASSERT(sfb->is_contiguous() && sfb->numel() == static_cast<int64_t>(G) * (N / 128) * (K / 128));
        p.sfa = sfa->data_ptr<float>();
        p.sfa_row_stride = sfa->stride(0);
        p.sfa_k_stride = sfa->stride(1);
        p.sfb = sfb->data_ptr<float>();
        p.scales_pow2 = pow2_scales ? 1 : 0;
    }
    p.error = gemm_status();
    p.timeout_ns = 10ull * 1000 * 1000 * 1000;
    const int sms = num_sms > 0 ? num_sms : at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
    const int64_t b_stride = (grouped ? b.stride(1) : b.stride(0)) * elem;
    EP_HOST_ASSERT(b_stride % 16 == 0 && reinterpret_cast<uintptr_t>(b.data_ptr()) % 16 == 0);
    CUDA_RUNTIME_CHECK(gemm::launch_gemm(p, a.data_ptr(), a.stride(0) * elem, b.data_ptr(), b_stride, fp8, sms,
                                         at::cuda::getCurrentCUDAStream().stream()));
    return *out;
}

// out[g] = a[:, range g] @ b[:, range g]^T for all groups in one launch (bf16): the k range of group g is
// [align(group_end[g-1], group_alignment), group_end[g]), read from the device array, no host synchronisation.
// mn_major: the operands are given as [K, M] and [K, N] (the rows of an expert are the contraction dimension and lie in
// memory as the forward pass left them): no transposed copies.
at::Tensor gemm_k_grouped(const at::Tensor& a, const at::Tensor& b, const at::Tensor& group_end, int num_groups, int group_alignment,
                          std::optional<at::Tensor> out, int num_sms, bool mn_major) {
    EP_HOST_ASSERT(a.is_cuda() && b.is_cuda() && a.dim() == 2 && b.dim() == 2 && a.stride(1) == 1 && b.stride(1) == 1);
    const int kd = mn_major ? 0 : 1;
    EP_HOST_ASSERT(a.scalar_type() == at::kBFloat16 && b.scalar_type() == at::kBFloat16 && a.size(kd) == b.size(kd));
    const int M = static_cast<int>(a.size(1 - kd)), N = static_cast<int>(b.size(1 - kd)), K = static_cast<int>(a.size(kd));
    EP_HOST_ASSERT_MSG(N % 128 == 0 && K % 64 == 0 && group_alignment % 64 == 0, "N must be a multiple of 128, K and the group alignment of 64");
    EP_HOST_ASSERT((a.stride(0) * 2) % 16 == 0 && (b.stride(0) * 2) % 16 == 0 && reinterpret_cast<uintptr_t>(a.data_ptr()) % 16 == 0 &&
                   reinterpret_cast<uintptr_t>(b.data_ptr()) % 16 == 0);
    EP_HOST_ASSERT(group_end.scalar_type() == at::kInt && group_end.is_contiguous() && group_end.numel() >= num_groups && num_groups >= 1);
    const int device = a.get_device();
    c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(device));
    if (!out.has_value()) out = new_tensor({num_groups, M, N}, at::kBFloat16, device);
    EP_HOST_ASSERT(out->scalar_type() == at::kBFloat16 && out->is_contiguous() && out->numel() == static_cast<int64_t>(num_groups) * M * N);
    gemm::GemmParams p = {};
    p.M = M;
    p.N = N;
    p.K = K;
    p.num_groups = num_groups;
    p.group_end = group_end.data_ptr<int>();
    p.group_alignment = group_alignment;
    p.zero_gap = 0;
    p.k_grouped = 1;
    p.a_mn = p.b_mn = mn_major ? 1 : 0;
    p.c_group_stride = static_cast<int64_t>(M) * N;
    p.C = reinterpret_cast<__nv_bfloat16*>(out->data_ptr());
    p.ldc = N;
    p.error = gemm_status();
    p.timeout_ns = 10ull * 1000 * 1000 * 1000;
    const int sms = num_sms > 0 ? num_sms : at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
    CUDA_RUNTIME_CHECK(gemm::launch_gemm(p, a.data_ptr(), a.stride(0) * 2, b.data_ptr(), b.stride(0) * 2, false, sms, cur_stream()));
    return *out;
}

// bf16 a @ b with b as it lies in memory: b [K, N]; a [M, K], or a^T @ b with a [K, M] (any K then: the weight gradient of a
// linear layer, rows of both being the tokens).
static at::Tensor gemm_mn(const at::Tensor& a, const at::Tensor& b, bool a_transposed) {
    EP_HOST_ASSERT(a.is_cuda() && b.is_cuda() && a.dim() == 2 && b.dim() == 2 && a.stride(1) == 1 && b.stride(1) == 1);
    EP_HOST_ASSERT(a.scalar_type() == at::kBFloat16 && b.scalar_type() == at::kBFloat16);
    const int M = static_cast<int>(a.size(a_transposed ? 1 : 0)), K = static_cast<int>(a.size(a_transposed ? 0 : 1)), N = static_cast<int>(b.size(1));
    EP_HOST_ASSERT(b.size(0) == K);
    EP_HOST_ASSERT_MSG(N % 128 == 0 && (a_transposed || K % 64 == 0), "N must be a multiple of 128, K of 64 unless a is transposed");
    EP_HOST_ASSERT((a.stride(0) * 2) % 16 == 0 && (b.stride(0) * 2) % 16 == 0 && reinterpret_cast<uintptr_t>(a.data_ptr()) % 16 == 0 &&
                   reinterpret_cast<uintptr_t>(b.data_ptr()) % 16 == 0);
    const int device = a.get_device();
    c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(device));
    at::Tensor out = new_tensor({M, N}, at::kBFloat16, device);
    if (M == 0) return out;
    if (K == 0) return out.zero_();
    gemm::GemmParams p = {};
    p.M = M;
    p.N = N;
    p.K = K;
    p.num_groups = 1;
    p.group_alignment = 1;
    p.a_mn = a_transposed ? 1 : 0;
    p.b_mn = 1;
    p.C = reinterpret_cast<__nv_bfloat16*>(out.data_ptr());
    p.ldc = N;
    p.error = gemm_status();
    p.timeout_ns = 10ull * 1000 * 1000 * 1000;
    CUDA_RUNTIME_CHECK(gemm::launch_gemm(p, a.data_ptr(), a.stride(0) * 2, b.data_ptr(), b.stride(0) * 2, false,
                                         at::cuda::getCurrentDeviceProperties()->multiProcessorCount, cur_stream()));
    return out;
}

static std::tuple<at::Tensor, at::Tensor> router_topk(const at::Tensor& logits, int num_topk) {
    const bool bf16 = logits.scalar_type() == at::kBFloat16;
    EP_HOST_ASSERT(logits.is_cuda() && logits.dim() == 2 && (bf16 || logits.scalar_type() == at::kFloat) && logits.stride(1) == 1);
    c10::cuda::CUDAGuard guard(logits.device());
    const int T = static_cast<int>(logits.size(0)), E = static_cast<int>(logits.size(1)), device = logits.get_device();
    auto idx = new_tensor({T, num_topk}, at::kLong, device), w = new_tensor({T, num_topk}, at::kFloat, device);
    CUDA_RUNTIME_CHECK(ops::router_topk(logits.data_ptr(), bf16, logits.stride(0), T, E, num_topk, idx.data_ptr<int64_t>(), w.data_ptr<float>(), cur_stream()));
    return {idx, w};
}

// Router of the MoE layer: (topk_idx, topk_weights, bf16 weights padded to a multiple of 128 experts) from x [T, hidden] and
// the fp32 or bf16 router weights [experts, hidden]
std::tuple<at::Tensor, at::Tensor, at::Tensor> router_forward(const at::Tensor& x, const at::Tensor& router, int num_topk) {
    EP_HOST_ASSERT(router.is_cuda() && router.dim() == 2 && router.is_contiguous() && router.size(1) == x.size(1) && router.size(1) % 8 == 0);
    c10::cuda::CUDAGuard guard(x.device());
    const int E = static_cast<int>(router.size(0)), H = static_cast<int>(router.size(1)), padded = align_up(E, 128), device = x.get_device();
    at::Tensor w = router;
    if (router.scalar_type() != at::kBFloat16 || padded != E) {
        w = new_tensor({padded, H}, at::kBFloat16, device);
        const at::Tensor f = on_16_bytes(router.scalar_type() == at::kFloat ? router : router.to(at::kFloat));
        CUDA_RUNTIME_CHECK(ops::router_weights(f.data_ptr<float>(), E, padded, H, w.data_ptr(), cur_stream()));
    }
    const at::Tensor logits = gemm_impl(x, w, std::nullopt, std::nullopt, std::nullopt, 1, std::nullopt, 0, false, true);
    const int T = static_cast<int>(x.size(0));
    auto idx = new_tensor({T, num_topk}, at::kLong, device), tw = new_tensor({T, num_topk}, at::kFloat, device);
    CUDA_RUNTIME_CHECK(ops::router_topk(logits.data_ptr(), true, logits.stride(0), T, E, num_topk, idx.data_ptr<int64_t>(), tw.data_ptr<float>(), cur_stream()));
    return {idx, tw, w};
}

// d_router [experts, hidden] in bf16 from the gradient of the top-k weights; the router's share of the input gradient is
// added to dx [T, hidden] in place
at::Tensor router_backward(const at::Tensor& x, const at::Tensor& router_padded, const at::Tensor& topk_idx, const at::Tensor& w,
                           const at::Tensor& dw, int num_experts, const at::Tensor& dx) {
    EP_HOST_ASSERT(topk_idx.scalar_type() == at::kLong && topk_idx.is_contiguous() && w.is_contiguous() && w.scalar_type() == at::kFloat &&
                   dw.scalar_type() == at::kFloat && dw.is_contiguous() && dw.numel() == w.numel());
    EP_HOST_ASSERT(dx.scalar_type() == at::kBFloat16 && dx.is_contiguous() && dx.sizes() == x.sizes() && router_padded.is_contiguous() &&
                   router_padded.scalar_type() == at::kBFloat16 && router_padded.size(1) == dx.size(1) && dx.size(1) % 8 == 0);
    c10::cuda::CUDAGuard guard(x.device());
    const int T = static_cast<int>(topk_idx.size(0)), K = static_cast<int>(topk_idx.size(1)), padded = static_cast<int>(router_padded.size(0));
    at::Tensor dlogits = new_tensor({T, padded}, at::kBFloat16, x.get_device());
    CUDA_RUNTIME_CHECK(ops::router_backward(topk_idx.data_ptr<int64_t>(), w.data_ptr<float>(), dw.data_ptr<float>(), T, K, num_experts, padded,
                                            static_cast<int>(dx.size(1)), router_padded.data_ptr(), dx.data_ptr(), dlogits.data_ptr(), cur_stream()));
    return first_rows(gemm_mn(dlogits, x, true), num_experts);
}

// bf16 [G, N, K] -> (e4m3 [G, N, K], fp32 scales [G, N / 128, K / 128])
static std::tuple<at::Tensor, at::Tensor> quant_weights_128x128(const at::Tensor& w, bool pow2) {
    EP_HOST_ASSERT(w.is_cuda() && w.dim() == 3 && w.scalar_type() == at::kBFloat16 && w.is_contiguous() && w.size(1) % 128 == 0 && w.size(2) % 128 == 0);
    c10::cuda::CUDAGuard guard(w.device());
    const int G = static_cast<int>(w.size(0)), N = static_cast<int>(w.size(1)), K = static_cast<int>(w.size(2)), device = w.get_device();
    auto q = new_tensor({G, N, K}, at::kFloat8_e4m3fn, device), sf = new_tensor({G, N / 128, K / 128}, at::kFloat, device);
    const at::Tensor aligned = on_16_bytes(w);
    CUDA_RUNTIME_CHECK(ops::quant_weights_128x128(aligned.data_ptr(), G, N, K, pow2, q.data_ptr(), sf.data_ptr<float>(), cur_stream()));
    return {q, sf};
}

static std::tuple<at::Tensor, at::Tensor> quant_1x128(const at::Tensor& x, bool pow2, bool col_major_sf) {
    EP_HOST_ASSERT(x.is_cuda() && x.dim() == 2 && x.scalar_type() == at::kBFloat16 && x.stride(1) == 1 && (x.stride(0) * 2) % 16 == 0);
    c10::cuda::CUDAGuard guard(x.device());
    const int M = static_cast<int>(x.size(0)), H = static_cast<int>(x.size(1));
    EP_HOST_ASSERT(H % 128 == 0);
    auto q = new_tensor({M, H}, at::kFloat8_e4m3fn, x.get_device());
    at::Tensor sf = col_major_sf ? at::empty({H / 128, align_up(std::max(M, 1), 4)}, x.options().dtype(at::kFloat)).t().slice(0, 0, M)
                                 : new_tensor({M, H / 128}, at::kFloat, x.get_device());
    CUDA_RUNTIME_CHECK(ops::quant_1x128(x.data_ptr(), x.stride(0) * 2, M, H, pow2, q.data_ptr(), sf.data_ptr<float>(), sf.stride(0),
                                        sf.stride(1), cur_stream()));
    return {q, sf};
}

// the row groups of an expanded dispatch (null = none)
static ops::RowGroups row_groups(const std::optional<at::Tensor>& group_end, int group_alignment) {
    ops::RowGroups g;
    if (!group_end.has_value()) return g;
    EP_HOST_ASSERT(group_end->is_cuda() && group_end->scalar_type() == at::kInt && group_end->is_contiguous() && group_alignment >= 1);
    g.ends = group_end->data_ptr<int>();
    g.num = static_cast<int>(group_end->numel());
    g.alignment = group_alignment;
    return g;
}

at::Tensor dequant_1x128(const at::Tensor& q, const at::Tensor& sf, const std::optional<at::Tensor>& group_end, int group_alignment) {
    EP_HOST_ASSERT(q.is_cuda() && q.dim() == 2 && q.scalar_type() == at::kFloat8_e4m3fn && q.is_contiguous() && sf.scalar_type() == at::kFloat);
    c10::cuda::CUDAGuard guard(q.device());
    const int M = static_cast<int>(q.size(0)), H = static_cast<int>(q.size(1));
    EP_HOST_ASSERT(H % 128 == 0 && sf.size(0) == M && sf.size(1) == H / 128);
    auto out = new_tensor({M, H}, at::kBFloat16, q.get_device());
    const at::Tensor aligned = on_16_bytes(q);
    CUDA_RUNTIME_CHECK(ops::dequant_1x128(aligned.data_ptr(), sf.data_ptr<float>(), sf.stride(0), sf.stride(1), M, H, row_groups(group_end, group_alignment),
                                          out.data_ptr(), cur_stream()));
    return out;
}

// returns (out, scales or None)
std::tuple<at::Tensor, std::optional<at::Tensor>> swiglu(const at::Tensor& x, const std::optional<at::Tensor>& row_weight,
                                                          const std::optional<at::Tensor>& num_valid_rows, bool quant, bool pow2,
                                                          const std::optional<at::Tensor>& group_end, int group_alignment) {
    EP_HOST_ASSERT(x.is_cuda() && x.dim() == 2 && x.scalar_type() == at::kBFloat16 && x.is_contiguous() && x.size(1) % 16 == 0);
    c10::cuda::CUDAGuard guard(x.device());
    const int M = static_cast<int>(x.size(0)), I = static_cast<int>(x.size(1) / 2);
    const float* rw = nullptr;
    if (row_weight.has_value()) {
        EP_HOST_ASSERT(row_weight->scalar_type() == at::kFloat && row_weight->is_contiguous() && row_weight->numel() >= M);
        rw = row_weight->data_ptr<float>();
    }
    const int* nv = num_valid_rows.has_value() ? num_valid_rows->data_ptr<int>() : nullptr;
    at::Tensor out = new_tensor({M, I}, quant ? at::kFloat8_e4m3fn : at::kBFloat16, x.get_device());
    std::optional<at::Tensor> sf;
    if (quant) sf = new_tensor({M, I / 128}, at::kFloat, x.get_device());
    CUDA_RUNTIME_CHECK(ops::swiglu(x.data_ptr(), M, I, rw, nv, row_groups(group_end, group_alignment), out.data_ptr(), quant, quant ? sf->data_ptr<float>() : nullptr,
                                   quant ? sf->stride(0) : 0, quant ? sf->stride(1) : 0, pow2, cur_stream()));
    return {out, sf};
}

std::tuple<at::Tensor, at::Tensor, at::Tensor> swiglu_backward(const at::Tensor& x, const at::Tensor& dout, const std::optional<at::Tensor>& row_weight, bool with_byproducts,
                           const std::optional<at::Tensor>& group_end, int group_alignment) {
    EP_HOST_ASSERT(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.is_contiguous() && dout.scalar_type() == at::kBFloat16 && dout.is_contiguous());
    c10::cuda::CUDAGuard guard(x.device());
    const int M = static_cast<int>(x.size(0)), I = static_cast<int>(x.size(1) / 2);
    EP_HOST_ASSERT(dout.size(0) == M && dout.size(1) == I);
    if (row_weight.has_value()) EP_HOST_ASSERT(row_weight->scalar_type() == at::kFloat && row_weight->is_contiguous() && row_weight->numel() >= M);
    auto dx = new_tensor({M, 2 * I}, at::kBFloat16, x.get_device());
    at::Tensor act, dweight;
    if (with_byproducts) {
        act = new_tensor({M, I}, at::kBFloat16, x.get_device());
        dweight = new_tensor({M}, at::kFloat, x.get_device());
    }
    CUDA_RUNTIME_CHECK(ops::swiglu_backward(x.data_ptr(), dout.data_ptr(), M, I, row_weight.has_value() ? row_weight->data_ptr<float>() : nullptr,
                                            row_groups(group_end, group_alignment), dx.data_ptr(), with_byproducts ? act.data_ptr() : nullptr,
                                            with_byproducts ? dweight.data_ptr<float>() : nullptr, cur_stream()));
    return {dx, act, dweight};
}

// [rows, cols] -> [cols, rows], or the same for every matrix of a batch [n, rows, cols]
static at::Tensor transpose_bf16(const at::Tensor& x) {
    EP_HOST_ASSERT(x.is_cuda() && (x.dim() == 2 || x.dim() == 3) && x.scalar_type() == at::kBFloat16 && x.stride(-1) == 1);
    c10::cuda::CUDAGuard guard(x.device());
    const bool batched = x.dim() == 3;
    const int n = batched ? static_cast<int>(x.size(0)) : 1, rows = static_cast<int>(x.size(-2)), cols = static_cast<int>(x.size(-1));
    EP_HOST_ASSERT(n <= 65535);
    auto out = batched ? new_tensor({n, cols, rows}, at::kBFloat16, x.get_device()) : new_tensor({cols, rows}, at::kBFloat16, x.get_device());
    CUDA_RUNTIME_CHECK(ops::transpose_bf16(x.data_ptr(), x.stride(-2), batched ? x.stride(0) : 0, n, rows, cols, out.data_ptr(), rows,
                                           static_cast<int64_t>(rows) * cols, cur_stream()));
    return out;
}

void register_ops_bindings(py::module_& m) {
    m.def("router_topk", &router_topk);
    m.def("router_backward", &router_backward);
    m.def("quant_weights_128x128", &quant_weights_128x128, py::arg("w"), py::arg("pow2") = false);
    m.def("quant_1x128", &quant_1x128, py::arg("x"), py::arg("pow2") = false, py::arg("col_major_sf") = false);
    m.def("dequant_1x128", &dequant_1x128, py::arg("q"), py::arg("sf"), py::arg("group_end") = py::none(), py::arg("group_alignment") = 1);
    m.def("swiglu", &swiglu, py::arg("x"), py::arg("row_weight") = py::none(), py::arg("num_valid_rows") = py::none(), py::arg("quant") = false,
          py::arg("pow2") = false, py::arg("group_end") = py::none(), py::arg("group_alignment") = 1);
    // returns dx, or with `with_byproducts` (dx, weighted activation [rows, inter] bf16, gradient of the row weight [rows] fp32)
    m.def("swiglu_backward", [](const at::Tensor& x, const at::Tensor& dout, const std::optional<at::Tensor>& row_weight, bool with_byproducts,
                                const std::optional<at::Tensor>& group_end, int group_alignment) -> py::object {
        const auto [dx, act, dweight] = swiglu_backward(x, dout, row_weight, with_byproducts, group_end, group_alignment);
        return with_byproducts ? py::object(py::make_tuple(dx, act, dweight)) : py::cast(dx);
    }, py::arg("x"), py::arg("dout"), py::arg("row_weight") = py::none(),
          py::arg("with_byproducts") = false, py::arg("group_end") = py::none(), py::arg("group_alignment") = 1);
    m.def("transpose_bf16", &transpose_bf16);
    m.def("gemm", &gemm_impl, py::arg("a"), py::arg("b"), py::arg("sfa") = py::none(), py::arg("sfb") = py::none(),
          py::arg("group_end") = py::none(), py::arg("group_alignment") = 1, py::arg("out") = py::none(), py::arg("num_sms") = 0,
          py::arg("pow2_scales") = false, py::arg("zero_gap") = true,
          "C = A @ B^T on the tcgen05 tensor cores (bf16, or e4m3 with 1x128 / 128x128 block scales); 3-D B = grouped. "
          "pow2_scales: every scale is an exact power of two (round_scale quantisation), which lets the tensor core apply "
          "them itself (kind::mxf8f6f4.block_scale) when N is a multiple of 256 and K at most 8192. "
          "zero_gap: rows in the alignment gaps of a grouped problem are written as zeros (alignment a multiple of 128), else left alone");
    m.def("gemm_k_grouped", &gemm_k_grouped, py::arg("a"), py::arg("b"), py::arg("group_end"), py::arg("num_groups"),
          py::arg("group_alignment") = 128, py::arg("out") = py::none(), py::arg("num_sms") = 0, py::arg("mn_major") = false,
          "C[g] = A[:, k range g] @ B[:, k range g]^T for all groups in one launch (bf16; the ranges come from a device array)");
    m.def("gemm_mn", &gemm_mn, py::arg("a"), py::arg("b"), py::arg("a_transposed") = false,
          "a @ b, or a^T @ b, with b [K, N] row-major (bf16)");
    m.def("gemm_check_status", &gemm_check_status);
}

}  // namespace ep
