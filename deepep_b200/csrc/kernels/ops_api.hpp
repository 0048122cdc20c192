// Launch interface of the small MoE operators (no torch types).
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace ep {
namespace ops {

// Rows of the expanded (expert-major) layout: group g ends at ends[g] (device), the next one starts at the next multiple of
// `alignment`; the rows in between mean nothing. ends = null: every row counts.
struct RowGroups {
    const int* ends = nullptr;
    int num = 0;
    int alignment = 1;
};

// top-k experts per token (ties: lowest id) and softmax weights over the selected logits
// (logits fp32 or bf16, rows `row_stride` elements apart)
cudaError_t router_topk(const void* logits, bool bf16, int64_t row_stride, int num_tokens, int num_experts, int num_topk, int64_t* topk_idx,
                        float* topk_weights, cudaStream_t stream);
// fp32 [experts, hidden] -> bf16 [padded experts, hidden] with zero rows at the end
cudaError_t router_weights(const float* w, int num_experts, int padded_experts, int hidden, void* out, cudaStream_t stream);
// bf16 dlogits [tokens, padded experts] from the top-k weights and their gradient
cudaError_t router_backward(const int64_t* topk_idx, const float* w, const float* dw, int num_tokens, int num_topk, int num_experts, int padded_experts,
                            int hidden, const void* router, void* dx, void* dlogits, cudaStream_t stream);
// bf16 [groups, rows, cols] -> e4m3 + one fp32 scale per 128 x 128 block
cudaError_t quant_weights_128x128(const void* w, int groups, int rows, int cols, bool pow2, void* q, float* scales, cudaStream_t stream);
// bf16 [rows, hidden] -> e4m3 [rows, hidden] + fp32 scales (element (row, block) at scales[row * row_stride + block * col_stride])
cudaError_t quant_1x128(const void* x, int64_t x_stride_bytes, int rows, int hidden, bool pow2, void* out, float* scales,
                        int64_t sf_row_stride, int64_t sf_col_stride, cudaStream_t stream);
cudaError_t dequant_1x128(const void* q, const float* scales, int64_t sf_row_stride, int64_t sf_col_stride, int rows, int hidden,
                          const RowGroups& groups, void* out, cudaStream_t stream);     // (rows in gaps become zeros)
// x [rows, 2 * inter] bf16 (gate | up) -> out [rows, inter]: silu(gate) * up * row_weight; bf16, or e4m3 + 1x128 scales with `quant`.
// Rows in gaps of `groups` are not written. `num_valid_rows` (device, optional) limits the work to the first rows. `pow2`: scales rounded up to powers of two.
cudaError_t swiglu(const void* x, int rows, int inter, const float* row_weight, const int* num_valid_rows, const RowGroups& groups, void* out, bool quant,
                   float* scales, int64_t sf_row_stride, int64_t sf_col_stride, bool pow2, cudaStream_t stream);
// dx [rows, 2 * inter] from dout [rows, inter]; optional by-products of the same pass: act_out [rows, inter] bf16 =
// silu(gate) * up * row_weight and dweight [rows] fp32 = sum_i dout_i * silu(gate_i) * up_i (gradient of the row weight); rows in gaps of `groups` give zeros
cudaError_t swiglu_backward(const void* x, const void* dout, int rows, int inter, const float* row_weight, const RowGroups& groups, void* dx, void* act_out,
                            float* dweight, cudaStream_t stream);
// [batch][rows, cols] -> [batch][cols, rows]
cudaError_t transpose_bf16(const void* in, int64_t in_stride, int64_t in_batch, int batch, int rows, int cols, void* out, int64_t out_stride,
                           int64_t out_batch, cudaStream_t stream);

}  // namespace ops
}  // namespace ep
