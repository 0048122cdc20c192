// Routing layout of one rank: tokens per destination rank (a token counts once per rank),
// (token, expert) pairs per expert, and the token x rank membership matrix.
//
// Parity: csrc/kernels/legacy/layout.cu:10-122 (get_dispatch_layout) of the reference,
// which splits experts and ranks over separate SM groups; here every block histograms its
// own slice of tokens in shared memory and merges with one atomic per non-zero bin (into the first block of a cluster, or
// into global memory).
#include <cooperative_groups.h>

#include "api.hpp"
#include "../common/device_utils.cuh"
#include "../common/launch.hpp"

namespace ep {

namespace {

constexpr int kLayoutThreads = 1024, kLayoutMaxCtas = 8;
constexpr int kLayoutWideThreads = 256;

// This block's share of the tokens (grid-strided): histogram in shared memory, one row of the mask per token.
__device__ __forceinline__ void count_tokens(const void* __restrict__ topk_idx, bool idx32, int num_tokens, int num_topk, int num_ranks, int num_experts,
                                             int* s_expert, int* s_rank, bool* is_token_in_rank) {
    const int experts_per_rank = num_experts / num_ranks;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < num_tokens; t += gridDim.x * blockDim.x) {
        uint32_t mask = 0;
        for (int k = 0; k < num_topk; ++k) {
            const int e = load_topk_idx(topk_idx, idx32, static_cast<int64_t>(t) * num_topk + k, num_experts);
            if (e >= 0) {
                atomicAdd(s_expert + e, 1);
                mask |= 1u << (e / experts_per_rank);
            }
        }
        for (int r = 0; r < num_ranks; ++r) {
            const bool in = (mask >> r) & 1u;
            is_token_in_rank[static_cast<int64_t>(t) * num_ranks + r] = in;
            if (in) atomicAdd(s_rank + r, 1);
        }
    }
}

// One thread-block cluster counts everything: a histogram per CTA in shared memory, summed into the first CTA's through
// distributed shared memory. Counting with global atomics wants two cleared arrays first, i.e. three launches.
__global__ void __launch_bounds__(kLayoutThreads) layout_kernel(const void* __restrict__ topk_idx, bool idx32, int num_tokens, int num_topk, int num_ranks,
                                                     int num_experts, int* num_tokens_per_rank, int* num_tokens_per_expert,
                                                     bool* is_token_in_rank) {
    extern __shared__ int s_hist[];   // [num_experts + num_ranks]
    int* s_expert = s_hist;
    int* s_rank = s_hist + num_experts;
    for (int i = threadIdx.x; i < num_experts + num_ranks; i += blockDim.x) s_hist[i] = 0;
    auto cluster = cooperative_groups::this_cluster();
    cluster.sync();                   // every CTA's histogram is cleared, and every CTA is there
    count_tokens(topk_idx, idx32, num_tokens, num_topk, num_ranks, num_experts, s_expert, s_rank, is_token_in_rank);
    __syncthreads();
    if (blockIdx.x != 0) {
        int* first = cluster.map_shared_rank(s_hist, 0);
        for (int i = threadIdx.x; i < num_experts + num_ranks; i += blockDim.x)
            if (s_hist[i] != 0) atomicAdd(first + i, s_hist[i]);
    }
    cluster.sync();
    if (blockIdx.x == 0) {
        for (int i = threadIdx.x; i < num_experts; i += blockDim.x) num_tokens_per_expert[i] = s_expert[i];
        for (int i = threadIdx.x; i < num_ranks; i += blockDim.x) num_tokens_per_rank[i] = s_rank[i];
    }
}

// The same on all SMs, added up in global memory (cleared before).
__global__ void __launch_bounds__(kLayoutWideThreads) layout_wide_kernel(const void* __restrict__ topk_idx, bool idx32, int num_tokens, int num_topk, int num_ranks,
                                                                         int num_experts, int* num_tokens_per_rank, int* num_tokens_per_expert,
                                                                         bool* is_token_in_rank) {
    extern __shared__ int s_hist[];
    int* s_expert = s_hist;
    int* s_rank = s_hist + num_experts;
    for (int i = threadIdx.x; i < num_experts + num_ranks; i += blockDim.x) s_hist[i] = 0;
    __syncthreads();
    count_tokens(topk_idx, idx32, num_tokens, num_topk, num_ranks, num_experts, s_expert, s_rank, is_token_in_rank);
    __syncthreads();
    for (int i = threadIdx.x; i < num_experts; i += blockDim.x)
        if (s_expert[i] != 0) atomicAdd(num_tokens_per_expert + i, s_expert[i]);
    for (int i = threadIdx.x; i < num_ranks; i += blockDim.x)
        if (s_rank[i] != 0) atomicAdd(num_tokens_per_rank + i, s_rank[i]);
}

// A thousand small words: one launch instead of the ten elementwise launches that the same takes in PyTorch.
__global__ void __launch_bounds__(256) legacy_handle_kernel(const int* __restrict__ count_matrix, const int* __restrict__ token_slot, int rank, int num_ranks,
                                                            int num_tokens, int* rank_prefix, int* sent, int* received, int* send_head, bool* in_rank) {
    __shared__ int s_base[kMaxRanks];
    const int R = num_ranks;
    launch_dependents();
    dependency_wait();
    if (threadIdx.x < R) {
        const int d = threadIdx.x;
        int acc = 0;
        for (int s = 0; s < R; ++s) {
            if (s == rank) s_base[d] = acc;
            acc += count_matrix[s * R + d];
            if (blockIdx.x == 0) rank_prefix[s * R + d] = acc;
        }
        if (blockIdx.x == 0) {
            sent[d] = count_matrix[rank * R + d];
            received[d] = count_matrix[d * R + rank];
        }
    }
    __syncthreads();
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < static_cast<int64_t>(num_tokens) * R; i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int slot = token_slot[i];
        send_head[i] = slot >= 0 ? slot - s_base[i % R] : slot;
        if (in_rank != nullptr) in_rank[i] = slot >= 0;
    }
}

}  // namespace

cudaError_t launch_dispatch_layout(const void* topk_idx, bool idx32, int num_tokens, int num_topk, int num_ranks, int num_experts,
                                   int* num_tokens_per_rank, int* num_tokens_per_expert, bool* is_token_in_rank,
                                   cudaStream_t stream) {
    // Up to 64k pairs one cluster is the shorter way (one launch; 8.4 us for 8192 x 8), above that its eight SMs are the longer
    // one (16384 x 8: 10.4 us, 8192 x 16: 14.4, 32768 x 8: 16.2, 131072 x 8: 47; on all SMs 32768 x 8 takes 9.2 us with the two
    // memsets, 131072 x 8 13.5).
    const size_t smem_bytes = static_cast<size_t>(num_experts + num_ranks) * sizeof(int);
    if (static_cast<int64_t>(num_tokens) * num_topk > (1 << 16)) {
        cudaError_t err = cudaMemsetAsync(num_tokens_per_rank, 0, sizeof(int) * num_ranks, stream);
        if (err != cudaSuccess) return err;
        err = cudaMemsetAsync(num_tokens_per_expert, 0, sizeof(int) * num_experts, stream);
        if (err != cudaSuccess) return err;
        const int blocks = ceil_div(num_tokens, kLayoutWideThreads);
        layout_wide_kernel<<<blocks < 148 ? blocks : 148, kLayoutWideThreads, smem_bytes, stream>>>(
            topk_idx, idx32, num_tokens, num_topk, num_ranks, num_experts, num_tokens_per_rank, num_tokens_per_expert, is_token_in_rank);
        return cudaGetLastError();
    }
    int ctas = 1;
    while (ctas < kLayoutMaxCtas && ctas * kLayoutThreads < num_tokens) ctas *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(kLayoutThreads);
    cfg.dynamicSmemBytes = smem_bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ctas;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, layout_kernel, topk_idx, idx32, num_tokens, num_topk, num_ranks, num_experts, num_tokens_per_rank,
                              num_tokens_per_expert, is_token_in_rank);
}

cudaError_t launch_legacy_handle(const int* count_matrix, const int* token_slot, int rank, int num_ranks, int num_tokens, int* rank_prefix,
                                 int* sent, int* received, int* send_head, bool* in_rank, cudaStream_t stream) {
    const int64_t want = ceil_div<int64_t>(static_cast<int64_t>(num_tokens) * num_ranks, 256);
    return launch_early(legacy_handle_kernel, dim3(static_cast<int>(want < 1 ? 1 : (want > 148 ? 148 : want))), dim3(256), 0, stream, count_matrix, token_slot,
                        rank, num_ranks, num_tokens, rank_prefix, sent, received, send_head, in_rank);
}

}  // namespace ep
