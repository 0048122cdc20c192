// The tensor-level operators (ops_runtime.cpp) as other drivers of the runtime call them.
#pragma once

#include <ATen/core/Tensor.h>

#include <optional>
#include <tuple>

namespace ep {

at::Tensor gemm_impl(const at::Tensor& a, const at::Tensor& b, const std::optional<at::Tensor>& sfa, const std::optional<at::Tensor>& sfb,
                     const std::optional<at::Tensor>& group_end, int group_alignment, std::optional<at::Tensor> out, int num_sms,
                     bool pow2_scales, bool zero_gap);
at::Tensor gemm_k_grouped(const at::Tensor& a, const at::Tensor& b, const at::Tensor& group_end, int num_groups, int group_alignment,
                          std::optional<at::Tensor> out, int num_sms, bool mn_major);
std::tuple<at::Tensor, at::Tensor, at::Tensor> router_forward(const at::Tensor& x, const at::Tensor& router, int num_topk);
at::Tensor router_backward(const at::Tensor& x, const at::Tensor& router_padded, const at::Tensor& topk_idx, const at::Tensor& w,
                           const at::Tensor& dw, int num_experts, const at::Tensor& dx);
at::Tensor dequant_1x128(const at::Tensor& q, const at::Tensor& sf, const std::optional<at::Tensor>& group_end, int group_alignment);
std::tuple<at::Tensor, std::optional<at::Tensor>> swiglu(const at::Tensor& x, const std::optional<at::Tensor>& row_weight,
                                                          const std::optional<at::Tensor>& num_valid_rows, bool quant, bool pow2,
                                                          const std::optional<at::Tensor>& group_end, int group_alignment);
// (dx, weighted activation, gradient of the row weight); the last two are undefined without `with_byproducts`
std::tuple<at::Tensor, at::Tensor, at::Tensor> swiglu_backward(const at::Tensor& x, const at::Tensor& dout, const std::optional<at::Tensor>& row_weight,
                                                               bool with_byproducts, const std::optional<at::Tensor>& group_end, int group_alignment);

}  // namespace ep
