// Dispatch and combine of a group of ONE rank (sm_100a): every token stays on this GPU, so nothing is exchanged and
// nothing has to travel through the symmetric heap.
//
//   plan     one thread-block cluster ranks the (token, expert) pairs in token order (shared memory and distributed
//            shared memory only, no grid-wide barrier through global memory) and writes the routing description: rows
//            of the tokens and pairs, per-expert counts and prefixes, the counts that the host waits for;
//   move     all SMs: every payload row goes from the caller's tensor straight to its row(s) of the output, cast to
//            e4m3 with 1x128 scales on the way when asked to, with the routing words and scale factors beside it. It is
//            a programmatic dependent of the plan kernel: its blocks are resident when the plan is done;
//   combine  all SMs: every token's row(s) are summed (fp32, ascending top-k order) straight into the result.
//
// The multi-rank kernels (dispatch_ht.cu, combine_ht.cu) stage rows in the receive regions because peers write them;
// with one rank that is a second pass over the payload, and their cooperative grid is bound by its barriers: the
// 8192 x 7168 FP8 dispatch took 70 + 33 us and a 64-token one 32 + 34 us, the expanded combine of 32768 rows 680 us on
// 24 SMs.
//
// Results (row order, metadata, rounding) are those of the multi-rank kernels with one rank.
#include <cooperative_groups.h>

#include <algorithm>

#include "api.hpp"
#include "../common/device_utils.cuh"
#include "../common/launch.hpp"

namespace ep {

namespace {

namespace cg = cooperative_groups;

constexpr int kPlanThreads = 1024, kPlanWarps = kPlanThreads / 32;
constexpr int kPlanMaxCtas = 8;         // portable cluster size
constexpr int kPlanRegTopk = 8;         // top-k entries that a lane keeps in registers between the two passes

// Words of shared memory: counters [warps][E + 1] (column E counts tokens with a valid expert), token masks [warps][E],
// totals of all CTAs [kPlanMaxCtas][E + 1], this CTA's bases [E + 1].
__host__ __device__ inline int plan_smem_words(int E) {
    return kPlanWarps * (E + 1) + kPlanWarps * E + kPlanMaxCtas * (E + 1) + (E + 1);
}

// A CTA of the cluster owns a contiguous range of tokens, a warp a contiguous part of it, a lane one token of 32. A
// pair's position = tokens of earlier CTAs + of earlier warps + of earlier batches + of lower lanes that chose the same
// expert. The chain is latency-bound (a few hundred nanoseconds per step, whatever the batch), which is why it runs in
// one cluster: a cluster barrier costs about a microsecond less than a grid barrier through L2, and eight CTAs already
// hold 8192 tokens in one batch per warp.
__global__ void __launch_bounds__(kPlanThreads, 1) local_plan_kernel(const __grid_constant__ LocalPlanParams p) {
    extern __shared__ __align__(16) int s_plan[];
    const int E = p.num_experts, K = p.num_topk, T = p.num_tokens;
    int* s_cnt = s_plan;                                    // [warps][E + 1]
    uint32_t* s_mask = reinterpret_cast<uint32_t*>(s_cnt + kPlanWarps * (E + 1));   // [warps][E]
    int* s_all = reinterpret_cast<int*>(s_mask + kPlanWarps * E);                   // [CTAs][E + 1]
    int* s_base = s_all + kPlanMaxCtas * (E + 1);           // [E + 1]
    const int tid = threadIdx.x, lane = lane_id(), warp = warp_id();
    const int cta = blockIdx.x, num_ctas = gridDim.x;       // the grid is one cluster
    if (cta == 0 && tid == 0) {
        const uint64_t now = globaltimer_ns();
        p.timeline[0] = now;
        p.stamps[0] = now;
    }
    // The move kernel reads its input before its own wait: it may become resident once everything ahead of this kernel is done.
    dependency_wait();
    launch_dependents();
    // (first half of the barrier after which the other CTAs' shared memory may be written)
    if (num_ctas > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");

    const int chunk = ceil_div(T, num_ctas);
    const int t0 = min(T, cta * chunk), t1 = min(T, t0 + chunk);
    const int tpw = align_up(ceil_div(max(t1 - t0, 1), kPlanWarps), 32);        // tokens per warp
    const int a = min(t1, t0 + warp * tpw), b = min(t1, a + tpw);
    const bool in_regs = tpw == 32 && K <= kPlanRegTopk;
    // In registers a lane holds pairs lane, lane + 32, ... of the warp's 32 x K, so that loads and stores are contiguous
    // over the warp (a lane per token strides by the row: 16.5 us instead of 9 for 8192 x 8 pairs).
    int e_reg[kPlanRegTopk], pos_reg[kPlanRegTopk];
    int slot_reg = -1;
    const int pairs = (b - a) * K;
    if (in_regs) {
#pragma unroll
        for (int i = 0; i < kPlanRegTopk; ++i)
            e_reg[i] = (i < K && lane + 32 * i < pairs) ? load_topk_idx(p.topk_idx, p.idx32 != 0, static_cast<int64_t>(a) * K + lane + 32 * i, E) : -1;
    }
    for (int i = tid; i < kPlanWarps * (2 * E + 1) / 4; i += kPlanThreads) reinterpret_cast<int4*>(s_cnt)[i] = make_int4(0, 0, 0, 0);     // counters and masks
    __syncthreads();

    int* mine = s_cnt + warp * (E + 1);
    uint32_t* mask_of = s_mask + warp * E;
    int tokens_before = 0;
    // token of pair i: i / K for i < 32 K <= 1024, as a product (sixteen divisions a lane were a fifth of this kernel's issue slots)
    const uint32_t inv_k = 65536u / static_cast<uint32_t>(K) + 1u;
    auto token_of = [&](int i) { return (static_cast<uint32_t>(i) * inv_k) >> 16; };
    // All pairs of the 32 tokens from `base` on, in the same contiguous order, eight loads in flight (a lane that walked along
    // its own token's row waited for one load at a time: 239 against 101 us for a dispatch of 8192 tokens with top-32).
    auto walk_pairs = [&](int base, auto&& visit) {
        const int64_t first = static_cast<int64_t>(base) * K;
        const int n = min(32, b - base) * K;
        for (int i0 = lane; i0 - lane < n; i0 += 256) {
            int e[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) e[u] = i0 + 32 * u < n ? load_topk_idx(p.topk_idx, p.idx32 != 0, first + i0 + 32 * u, E) : -1;
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (i0 + 32 * u < n) visit(first + i0 + 32 * u, i0 + 32 * u, e[u]);
        }
    };
    if (in_regs) {
        uint32_t taken = 0;         // tokens of the warp with a valid expert
#pragma unroll
        for (int i = 0; i < kPlanRegTopk; ++i)
            if (e_reg[i] >= 0) {
                const uint32_t bit = 1u << token_of(lane + 32 * i);
                atomicOr(mask_of + e_reg[i], bit);
                taken |= bit;
            }
        __syncwarp();               // the masks of all lanes are in
        taken = __reduce_or_sync(0xffffffffu, taken);
        slot_reg = (taken >> lane) & 1u ? __popc(taken & lanemask_lt()) : -1;
        tokens_before = __popc(taken);
#pragma unroll
        for (int i = 0; i < kPlanRegTopk; ++i) {
            pos_reg[i] = 0;
            if (e_reg[i] >= 0) {
                const uint32_t m = mask_of[e_reg[i]];
                pos_reg[i] = __popc(m & ((1u << token_of(lane + 32 * i)) - 1u));
                if (pos_reg[i] == 0) mine[e_reg[i]] = __popc(m);      // the first token of a mask writes the count
            }
        }
    } else {
        // any number of batches per warp, any top-k: relative positions go to global memory and are completed below
        for (int base = a; base < b; base += 32) {
            uint32_t taken = 0;
            walk_pairs(base, [&](int64_t, int i, int e) {
                if (e < 0) return;
                const uint32_t bit = 1u << token_of(i);
                atomicOr(mask_of + e, bit);
                taken |= bit;
            });
            __syncwarp();
            taken = __reduce_or_sync(0xffffffffu, taken);
            if (base + lane < b) p.token_slot[base + lane] = (taken >> lane) & 1u ? tokens_before + __popc(taken & lanemask_lt()) : -1;
            tokens_before += __popc(taken);
            walk_pairs(base, [&](int64_t at, int i, int e) { p.pair_row[at] = e >= 0 ? mine[e] + __popc(mask_of[e] & ((1u << token_of(i)) - 1u)) : -1; });
            __syncwarp();
            walk_pairs(base, [&](int64_t, int i, int e) {       // the first token of a mask adds the count and clears it
                const uint32_t m = e >= 0 ? mask_of[e] : 0u;
                if (m != 0 && (m & ((1u << token_of(i)) - 1u)) == 0 && atomicExch(mask_of + e, 0u) != 0) mine[e] += __popc(m);
            });
            __syncwarp();
        }
    }
    if (lane == 0) mine[E] = tokens_before;
    __syncthreads();

    // counts of the warps -> exclusive prefix per column, totals of this CTA to every CTA of the cluster
    const int live_warps = min(kPlanWarps, ceil_div(max(t1 - t0, 1), tpw));
    if (num_ctas > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    for (int e = tid; e <= E; e += kPlanThreads) {
        int acc = 0;
        for (int w0 = 0; w0 < live_warps; w0 += 8) {
            int v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = w0 + u < live_warps ? s_cnt[(w0 + u) * (E + 1) + e] : 0;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                if (w0 + u < live_warps) s_cnt[(w0 + u) * (E + 1) + e] = acc;
                acc += v[u];
            }
        }
        if (num_ctas > 1) {
            auto cluster = cg::this_cluster();
            for (int c = 0; c < num_ctas; ++c) cluster.map_shared_rank(s_all, c)[cta * (E + 1) + e] = acc;
        } else {
            s_all[e] = acc;
        }
    }
    if (num_ctas > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        __syncthreads();
    }
    // first row of every expert (alignment applied): a thread per expert, prefix over the warps' sums; the column of the
    // tokens has no start to add
    __shared__ int s_warp_sum[kMaxLocalExperts / 32];
    static_assert(kMaxLocalExperts < kPlanThreads, "a thread per expert and one for the tokens");
    int total = 0, before = 0;
    if (tid <= E)
        for (int c = 0; c < num_ctas; ++c) {
            const int v = s_all[c * (E + 1) + tid];
            total += v;
            if (c < cta) before += v;
        }
    const int aligned = tid < E ? align_up(total, p.expert_alignment) : 0;
    int incl = aligned;
    if (warp < kMaxLocalExperts / 32) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
        }
        if (lane == 31) s_warp_sum[warp] = incl;
    }
    __syncthreads();
    if (tid < E) {
        int start = incl - aligned;
        for (int w = 0; w < warp; ++w) start += s_warp_sum[w];
        s_base[tid] = start + before;
        if (cta == 0) {
            if (p.host_counts != nullptr) {
                p.host_counts[2 + tid] = pack_epoch(p.epoch, static_cast<uint32_t>(aligned));
                if (tid == E - 1) p.host_counts[1] = pack_epoch(p.epoch, static_cast<uint32_t>(start + aligned));
            }
            p.num_unaligned[tid] = total;
            p.psum_expert[tid] = p.do_expand ? start + total : start + aligned;
            if (tid == E - 1) p.psum_expert[E] = start + aligned;
            if (p.recv_stats != nullptr) p.recv_stats[tid] += total;
        }
    } else if (tid == E) {
        s_base[E] = before;
        if (cta == 0) {
            if (p.host_counts != nullptr) p.host_counts[0] = pack_epoch(p.epoch, static_cast<uint32_t>(total));
            p.psum_rank[0] = total;
            p.count_matrix[0] = total;
        }
    }
    __syncthreads();
    const int slot_base = s_base[E] + mine[E];
    if (in_regs) {
        if (a + lane < b) p.token_slot[a + lane] = slot_reg < 0 ? -1 : slot_base + slot_reg;
#pragma unroll
        for (int i = 0; i < kPlanRegTopk; ++i)
            if (i < K && lane + 32 * i < pairs)
                p.pair_row[static_cast<int64_t>(a) * K + lane + 32 * i] = e_reg[i] < 0 ? -1 : s_base[e_reg[i]] + mine[e_reg[i]] + pos_reg[i];
    } else {
        for (int base = a; base < b; base += 32) {      // (every lane completes what it wrote itself)
            if (base + lane < b && p.token_slot[base + lane] >= 0) p.token_slot[base + lane] += slot_base;
            walk_pairs(base, [&](int64_t at, int, int e) {
                if (e >= 0) p.pair_row[at] += s_base[e] + mine[e];
            });
        }
    }
    if (cta == 0 && tid < 7) p.stamps[1 + tid] = globaltimer_ns();
}

// ==================================================================== move
constexpr int kMoveThreads = 256;
constexpr int kMoveSlice = 1024;            // input bytes of a row that a warp moves (32 per lane)
constexpr int kPadRows = 4;                 // padding rows per zeroing work item

// One warp per (token, 1 KB slice of its row) and nothing else: neighbouring warps have neighbouring slices, and a grid of
// many short blocks keeps the memory system busier than a resident grid that loops (8192 x 7168 bf16: copy 38 against
// 41-43 us, cast to e4m3 29 against 31-34 us, whatever the unrolling or prefetching inside the loop). The warps of column 0
// also write the tokens' routing words. The slice is requested before the plan is awaited (the input was there before the
// plan kernel started).
template <bool kQuant, bool kExpand>
__global__ void __launch_bounds__(kMoveThreads, kExpand ? 6 : 8) local_move_kernel(const __grid_constant__ LocalMoveParams p) {
    const int lane = lane_id();
    const int K = p.num_topk, T = p.num_tokens;
    const uint32_t warp_global = blockIdx.x * (kMoveThreads / 32) + warp_id(), num_warps = gridDim.x * (kMoveThreads / 32);
    const bool wide_in = p.wide_in != 0, wide_out = p.wide_out != 0;
    const int t = static_cast<int>(warp_global / static_cast<uint32_t>(p.columns)), col = static_cast<int>(warp_global % static_cast<uint32_t>(p.columns));
    const int off = col * kMoveSlice + lane * 32;
    int4 lo, hi;
    launch_dependents();
    if (!p.plan_ahead) dependency_wait();
    if (t < T) load_32(p.x + static_cast<int64_t>(t) * p.x_stride_bytes + off, p.src_row_bytes - off, wide_in, lo, hi);
    if (p.plan_ahead) dependency_wait();
    if (t < T) {
        // expanded: the row of top-k lane `lane`; else the token's row
        int row = kExpand ? (lane < K ? p.pair_row[static_cast<int64_t>(t) * K + lane] : -1) : p.token_slot[t];
        if (row >= p.num_out_rows) row = -1;
        const uint32_t rows = kExpand ? __ballot_sync(0xffffffffu, row >= 0) : (row >= 0 ? 1u : 0u);

        if (col == 0) {
            // ---- routing words
            int e = -1;
            if (lane < K) {
                const int64_t i = static_cast<int64_t>(t) * K + lane;
                e = load_topk_idx(p.topk_idx, p.idx32 != 0, i, p.num_experts);
                if (p.topk_idx_copy != nullptr) {
                    if (p.idx32) reinterpret_cast<int*>(p.topk_idx_copy)[i] = reinterpret_cast<const int*>(p.topk_idx)[i];
                    else reinterpret_cast<int64_t*>(p.topk_idx_copy)[i] = reinterpret_cast<const int64_t*>(p.topk_idx)[i];
                }
            }
            const uint32_t valid = __ballot_sync(0xffffffffu, e >= 0);
            const int slot = p.token_slot[t];
            // (the weights of an expanded row go with the row, also where the token has no place in the routing outputs)
            if (kExpand && row >= 0 && p.recv_topk_weights != nullptr) p.recv_topk_weights[row] = p.topk_weights[static_cast<int64_t>(t) * K + lane];
            if (slot >= 0 && slot < p.num_idx_rows && lane < K) {
                const int64_t o = static_cast<int64_t>(slot) * K + lane;
                if (!kExpand) {
                    if (p.recv_topk_idx != nullptr) {
                        if (p.idx32) reinterpret_cast<int*>(p.recv_topk_idx)[o] = e;
                        else reinterpret_cast<int64_t*>(p.recv_topk_idx)[o] = e;
                    }
                    if (p.recv_topk_weights != nullptr)
                        p.recv_topk_weights[o] = p.mask_weights && e < 0 ? 0.f : p.topk_weights[static_cast<int64_t>(t) * K + lane];
                }
                if (p.write_metadata) {
                    int* md = p.recv_src_metadata + static_cast<int64_t>(slot) * (K + 2);
                    md[2 + lane] = kExpand ? row : -1;
                    if (lane == 0) {
                        md[0] = t;
                        md[1] = valid != 0 ? __ffs(valid) - 1 : 0;
                    }
                }
            }
            // ---- scale factors that the caller made
            if (!kQuant && p.sf_packs > 0) {
                for (int i = lane; i < align_up(p.sf_packs, 32); i += 32) {
                    const bool in = i < p.sf_packs;
                    const uint32_t v = in ? p.sf[static_cast<int64_t>(t) * p.sf_token_stride + static_cast<int64_t>(i) * p.sf_pack_stride] : 0u;
                    for (uint32_t todo = rows; todo != 0; todo &= todo - 1) {
                        const int r = kExpand ? __shfl_sync(0xffffffffu, row, __ffs(todo) - 1) : row;
                        if (in) p.recv_sf[static_cast<int64_t>(r) * p.recv_sf_row_stride + static_cast<int64_t>(i) * p.recv_sf_pack_stride] = v;
                    }
                }
            }
        }

        // ---- payload
        if constexpr (!kQuant) {
            for (uint32_t todo = rows; todo != 0; todo &= todo - 1) {
                const int r = kExpand ? __shfl_sync(0xffffffffu, row, __ffs(todo) - 1) : row;
                store_32(p.recv_x + static_cast<int64_t>(r) * p.recv_x_pitch + off, p.src_row_bytes - off, wide_out, lo, hi);
            }
        } else {
            // a lane holds 16 channels, eight lanes a scale group of 128 (hidden is a multiple of 128: a group is all in or all out)
            float scale;
            const int4 q = cast16_e4m3(lo, hi, p.pow2 != 0, scale);
            for (uint32_t todo = rows; todo != 0; todo &= todo - 1) {
                const int r = kExpand ? __shfl_sync(0xffffffffu, row, __ffs(todo) - 1) : row;
                if (off >= p.src_row_bytes) continue;
                st_na_int4(p.recv_x + static_cast<int64_t>(r) * p.recv_x_pitch + off / 2, q);
                if ((lane & 7) == 0)
                    reinterpret_cast<float*>(p.recv_sf)[static_cast<int64_t>(r) * p.recv_sf_row_stride + (off >> 8) * p.recv_sf_pack_stride] = scale;
            }
        }
    }

    // ---- routing rows past the received count
    const int n = p.psum_rank[0];
    for (int64_t j = static_cast<int64_t>(n) * K + static_cast<int64_t>(warp_global) * 32 + lane; j < static_cast<int64_t>(p.num_idx_rows) * K; j += static_cast<int64_t>(num_warps) * 32) {
        const int i = static_cast<int>(j / K), k = static_cast<int>(j % K);
        if (!kExpand) {
            if (p.recv_topk_idx != nullptr) {
                if (p.idx32) reinterpret_cast<int*>(p.recv_topk_idx)[j] = -1;
                else reinterpret_cast<int64_t*>(p.recv_topk_idx)[j] = -1;
            }
            if (p.recv_topk_weights != nullptr) p.recv_topk_weights[j] = 0.f;
        }
        if (p.write_metadata) {
            int* md = p.recv_src_metadata + static_cast<int64_t>(i) * (K + 2);
            md[2 + k] = -1;
            if (k == 0) md[0] = md[1] = -1;
        }
    }

    // ---- alignment gaps of the expanded layout, kPadRows rows per item so that the few experts keep every SM busy
    if (kExpand && p.do_zero_padding) {
        const int out_row_bytes = kQuant ? p.src_row_bytes / 2 : p.src_row_bytes;
        const int per_expert = ceil_div(p.expert_alignment, kPadRows);
        for (int64_t it = warp_global; it < static_cast<int64_t>(p.num_experts) * per_expert; it += num_warps) {
            const int e = static_cast<int>(it / per_expert), part = static_cast<int>(it % per_expert);
            const int begin = p.psum_expert[e];                                     // start + real count
            const int end = min(align_up(begin, p.expert_alignment), p.num_out_rows);
            const int r0 = begin + part * kPadRows, r1 = min(end, r0 + kPadRows);
            for (int r = r0; r < r1; ++r) {
                uint8_t* dst = p.recv_x + static_cast<int64_t>(r) * p.recv_x_pitch;
                for (int v = lane * 16; v < out_row_bytes; v += 512) st_na_int4(dst + v, make_int4(0, 0, 0, 0));
                if (lane == 0 && p.recv_topk_weights != nullptr) p.recv_topk_weights[r] = 0.f;
                // the scales too: 0 x (whatever was in memory) would not be 0 for a NaN or an infinity
                if (p.recv_sf != nullptr)
                    for (int i = lane; i < p.sf_packs; i += 32) p.recv_sf[static_cast<int64_t>(r) * p.recv_sf_row_stride + static_cast<int64_t>(i) * p.recv_sf_pack_stride] = 0u;
            }
        }
    }
    if (threadIdx.x == 0 && (blockIdx.x == 0 || blockIdx.x == gridDim.x - 1))
        atomicMax(reinterpret_cast<unsigned long long*>(p.timeline + 1), static_cast<unsigned long long>(globaltimer_ns()));
}

// ==================================================================== combine
__device__ __forceinline__ void add_bf16x8(float (&acc)[8], const int4& raw) {
    const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 v = __bfloat1622float2(h2[i]);
        acc[2 * i] += v.x;
        acc[2 * i + 1] += v.y;
    }
}
__device__ __forceinline__ void fma_bf16x8(float (&acc)[8], const int4& raw, float w) {
    const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 v = __bfloat1622float2(h2[i]);
        acc[2 * i] = fmaf(w, v.x, acc[2 * i]);
        acc[2 * i + 1] = fmaf(w, v.y, acc[2 * i + 1]);
    }
}

constexpr int kCombineThreads = 128;

// Like the move kernel: a warp owns a column (NV x 512 bytes) of the rows and walks over tokens, so that neighbouring warps
// read neighbouring bytes of the same rows (a warp that walked along its own token's rows left every DRAM page after 512
// bytes: 121 us for 32768 rows of hidden 7168 against 81 us that the bytes take). NR rows x NV vectors = up to 128 bytes are
// in flight per lane before the first add; the rows of the next token are looked up meanwhile. The adds run in ascending
// top-k order.
// One row per token and nothing to add: the row is the result. One warp per KB of a row, as in the move kernel (in the
// kernel below, whose registers leave a third of the warps resident, the same copy took 45 instead of 39 us).
__global__ void __launch_bounds__(256, 8) local_return_kernel(const __grid_constant__ LocalCombineParams p) {
    const int lane = lane_id(), K = p.num_topk;
    launch_dependents();
    dependency_wait();
    if (blockIdx.x == 0 && threadIdx.x == 0) p.timeline[0] = globaltimer_ns();
    const uint32_t warp_global = blockIdx.x * 8 + warp_id();
    const int t = static_cast<int>(warp_global / static_cast<uint32_t>(p.columns)), col = static_cast<int>(warp_global % static_cast<uint32_t>(p.columns));
    if (t < p.num_tokens) {
        int row = p.token_slot[t];
        if (row >= p.num_x_rows) row = -1;
        const int off = col * 1024 + lane * 32;
        int4 lo = make_int4(0, 0, 0, 0), hi = lo;
        if (row >= 0) load_32(p.x + static_cast<int64_t>(row) * p.x_stride_bytes + off, p.row_bytes - off, p.wide != 0, lo, hi);
        store_32(p.combined_x + static_cast<int64_t>(t) * p.row_bytes + off, p.row_bytes - off, p.wide != 0, lo, hi);
        if (col == 0 && p.combined_topk_weights != nullptr && lane < K) {
            float v = 0.f;
            if (p.topk_weights != nullptr && row >= 0 && load_topk_idx(p.topk_idx, p.idx32 != 0, static_cast<int64_t>(t) * K + lane, p.num_experts) >= 0)
                v = p.topk_weights[static_cast<int64_t>(row) * K + lane];
            p.combined_topk_weights[static_cast<int64_t>(t) * K + lane] = v;
        }
    }
    if (threadIdx.x == 0 && blockIdx.x == gridDim.x - 1)
        atomicMax(reinterpret_cast<unsigned long long*>(p.timeline + 1), static_cast<unsigned long long>(globaltimer_ns()));
}

template <int NV, int NR, bool kExpand, bool kWeighted>
__global__ void __launch_bounds__(kCombineThreads) local_combine_kernel(const __grid_constant__ LocalCombineParams p) {
    const int lane = lane_id();
    const int K = p.num_topk, T = p.num_tokens;
    const int vec_per_row = p.row_bytes / 16;
    const int warp_global = blockIdx.x * (kCombineThreads / 32) + warp_id();
    const int col = warp_global % p.columns, step = p.warps / p.columns;
    const int v0 = col * 32 * NV + lane;
    launch_dependents();
    dependency_wait();
    if (blockIdx.x == 0 && threadIdx.x == 0) p.timeline[0] = globaltimer_ns();
    int t = warp_global < p.warps ? warp_global / p.columns : T;
    int next_row = -1, later_slot = -1;     // row of the next token (this lane's, when expanded), slot of the one after it
    auto request_row = [&](int slot) {
        // (a token beyond the rows that the caller made room for has no metadata)
        if (kExpand) next_row = lane < K && slot >= 0 && slot < p.num_meta_rows ? p.recv_src_metadata[static_cast<int64_t>(slot) * (K + 2) + 2 + lane] : -1;
        else next_row = slot;
    };
    if (t < T) request_row(p.token_slot[t]);
    if (t + step < T) later_slot = p.token_slot[t + step];
    for (; t < T; t += step) {
        const int row = next_row < p.num_x_rows ? next_row : -1;
        if (t + step < T) request_row(later_slot);
        if (t + 2 * step < T) later_slot = p.token_slot[t + 2 * step];
        uint8_t* dst = p.combined_x + static_cast<int64_t>(t) * p.row_bytes;
        if (col == 0 && p.combined_topk_weights != nullptr && lane < K) {
            float v = 0.f;
            if (p.topk_weights != nullptr && row >= 0) {
                if (kExpand) v = p.topk_weights[row];
                else if (load_topk_idx(p.topk_idx, p.idx32 != 0, static_cast<int64_t>(t) * K + lane, p.num_experts) >= 0)
                    v = p.topk_weights[static_cast<int64_t>(row) * K + lane];
            }
            p.combined_topk_weights[static_cast<int64_t>(t) * K + lane] = v;
        }
        const uint32_t rows = kExpand ? __ballot_sync(0xffffffffu, row >= 0) : (row >= 0 ? 1u : 0u);
        const float wt = kWeighted && row >= 0 ? p.topk_weights[row] : 0.f;
        float acc[NV][8];
#pragma unroll
        for (int j = 0; j < NV; ++j)
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[j][i] = 0.f;
        for (uint32_t todo = rows; todo != 0;) {        // (uniform over the warp: lanes past the row's end take part in the shuffles)
            int4 raw[NR][NV];
            const uint32_t batch = todo;
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const int rr = kExpand ? __shfl_sync(0xffffffffu, row, todo != 0 ? __ffs(todo) - 1 : 0) : row;
                const uint8_t* src = p.x + static_cast<int64_t>(rr) * p.x_stride_bytes;
#pragma unroll
                for (int j = 0; j < NV; ++j)
                    if (todo != 0 && v0 + 32 * j < vec_per_row) raw[r][j] = ld_nc_int4(src + (v0 + 32 * j) * 16);
                todo &= todo - 1;       // 0 stays 0
            }
            uint32_t now = batch;
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const float wr = kWeighted ? __shfl_sync(0xffffffffu, wt, now != 0 ? __ffs(now) - 1 : 0) : 1.f;
#pragma unroll
                for (int j = 0; j < NV; ++j)
                    if (now != 0 && v0 + 32 * j < vec_per_row) {
                        if (kWeighted) fma_bf16x8(acc[j], raw[r][j], wr);
                        else add_bf16x8(acc[j], raw[r][j]);
                    }
                now &= now - 1;
            }
        }
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const int v = v0 + 32 * j;
            if (v >= vec_per_row) continue;
            if (p.bias0 != nullptr || p.bias1 != nullptr) {
                if (p.round_partial) {
                    // a rank's partial sum is rounded once before it leaves the rank, then the biases are added
#pragma unroll
                    for (int i = 0; i < 8; ++i) acc[j][i] = __bfloat162float(__float2bfloat16_rn(acc[j][i]));
                }
                const int64_t off = static_cast<int64_t>(t) * p.row_bytes + v * 16;
                if (p.bias0 != nullptr) add_bf16x8(acc[j], ld_nc_int4(p.bias0 + off));
                if (p.bias1 != nullptr) add_bf16x8(acc[j], ld_nc_int4(p.bias1 + off));
            }
            int4 out;
            __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&out);
#pragma unroll
            for (int i = 0; i < 4; ++i) o2[i] = __floats2bfloat162_rn(acc[j][2 * i], acc[j][2 * i + 1]);
            st_na_int4(dst + v * 16, out);
        }
    }
    if (threadIdx.x == 0 && (blockIdx.x == 0 || blockIdx.x == gridDim.x - 1))
        atomicMax(reinterpret_cast<unsigned long long*>(p.timeline + 1), static_cast<unsigned long long>(globaltimer_ns()));
}

// Blocks that fit an SM at once, looked up once per kernel.
template <typename Kernel>
int resident_blocks(Kernel kernel, int threads, std::atomic<int>& known) {
    int n = known.load(std::memory_order_relaxed);
    if (n == 0) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, 0) != cudaSuccess || n < 1) n = 1;
        known.store(n, std::memory_order_relaxed);
    }
    return n;
}

// Warps for `tokens` x `columns` items on at most `most` resident warps: a multiple of the columns, such that every warp
// takes the same number of tokens (give or take one).
int balanced_warps(int tokens, int columns, int most) {
    const int64_t items = static_cast<int64_t>(tokens) * columns;
    const int rounds = static_cast<int>(ceil_div<int64_t>(items, most));
    int per_column = ceil_div(tokens, rounds < 1 ? 1 : rounds);
    return (per_column < 1 ? 1 : per_column) * columns;
}

}  // namespace

cudaError_t launch_local_plan(const LocalPlanParams& p, cudaStream_t stream) {
    const int smem_bytes = plan_smem_words(p.num_experts) * 4;
    static PreparedKernel prepared;
    cudaError_t err = prepared.prepare(local_plan_kernel, plan_smem_words(kMaxLocalExperts) * 4);
    if (err != cudaSuccess) return err;
    // one batch of 32 tokens per warp where the cluster can hold the tokens; a CTA that would stay empty only costs barrier time
    int ctas = 1;
    while (ctas < kPlanMaxCtas && ctas * kPlanThreads < p.num_tokens) ctas *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(kPlanThreads);
    cfg.dynamicSmemBytes = smem_bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ctas;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = programmatic_launches() ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, local_plan_kernel, p);
}

template <bool kQuant, bool kExpand>
static cudaError_t launch_move_cfg(LocalMoveParams& p, int num_sms, cudaStream_t stream) {
    static PreparedKernel prepared;
    cudaError_t err = prepared.prepare(local_move_kernel<kQuant, kExpand>, 0);
    if (err != cudaSuccess) return err;
    p.columns = ceil_div(p.src_row_bytes, kMoveSlice);
    int64_t warps = static_cast<int64_t>(p.num_tokens) * p.columns;
    if (warps >= (1ll << 31)) return cudaErrorInvalidValue;
    // (a few tokens can leave more padding rows to clear than there are slices to move)
    if (kExpand && p.do_zero_padding)
        warps = std::max<int64_t>(warps, std::min<int64_t>(num_sms * 32, static_cast<int64_t>(p.num_experts) * ceil_div(p.expert_alignment, kPadRows)));
    const int grid = std::max(1, static_cast<int>(ceil_div<int64_t>(warps, kMoveThreads / 32)));
    return launch_early(local_move_kernel<kQuant, kExpand>, dim3(grid), dim3(kMoveThreads), 0, stream, p);
}

cudaError_t launch_local_move(const LocalMoveParams& params, bool quant, int num_sms, cudaStream_t stream) {
    LocalMoveParams p = params;
    const uint64_t in_bits = reinterpret_cast<uintptr_t>(p.x) | static_cast<uint64_t>(p.x_stride_bytes);
    const uint64_t out_bits = reinterpret_cast<uintptr_t>(p.recv_x) | static_cast<uint64_t>(p.recv_x_pitch);
    p.wide_in = in_bits % 32 == 0;
    p.wide_out = out_bits % 32 == 0;
    if (quant) return p.do_expand ? launch_move_cfg<true, true>(p, num_sms, stream) : launch_move_cfg<true, false>(p, num_sms, stream);
    return p.do_expand ? launch_move_cfg<false, true>(p, num_sms, stream) : launch_move_cfg<false, false>(p, num_sms, stream);
}

template <int NV, int NR, bool kExpand, bool kWeighted>
static cudaError_t launch_combine_cfg(LocalCombineParams& p, int num_sms, cudaStream_t stream) {
    static PreparedKernel prepared;
    static std::atomic<int> per_sm{0};
    auto kernel = local_combine_kernel<NV, NR, kExpand, kWeighted>;
    cudaError_t err = prepared.prepare(kernel, 0);
    if (err != cudaSuccess) return err;
    const int warps_per_block = kCombineThreads / 32, most = num_sms * resident_blocks(kernel, kCombineThreads, per_sm) * warps_per_block;
    p.columns = ceil_div(p.row_bytes / 16, 32 * NV);
    p.warps = balanced_warps(p.num_tokens, p.columns, most);
    return launch_early(kernel, dim3(ceil_div(p.warps, warps_per_block)), dim3(kCombineThreads), 0, stream, p);
}

cudaError_t launch_local_combine(const LocalCombineParams& params, int num_sms, cudaStream_t stream) {
    if (params.num_tokens == 0) return cudaSuccess;
    LocalCombineParams p = params;
    if (!p.do_expand && p.bias0 == nullptr && p.bias1 == nullptr) {
        static PreparedKernel prepared;
        const cudaError_t err = prepared.prepare(local_return_kernel, 0);
        if (err != cudaSuccess) return err;
        p.columns = ceil_div(p.row_bytes, 1024);
        p.wide = (reinterpret_cast<uintptr_t>(p.x) | static_cast<uint64_t>(p.x_stride_bytes) | reinterpret_cast<uintptr_t>(p.combined_x) | static_cast<uint64_t>(p.row_bytes)) % 32 == 0;
        const int64_t warps = static_cast<int64_t>(p.num_tokens) * p.columns;
        if (warps >= (1ll << 31)) return cudaErrorInvalidValue;
        return launch_early(local_return_kernel, dim3(static_cast<int>(ceil_div<int64_t>(warps, 8))), dim3(256), 0, stream, p);
    }
    // Otherwise a resident grid, since looking up the rows of a token is a chain of two loads that the loop hides; up to four
    // rows two vectors at a time, more than four one (128 bytes in flight per lane either way).
    if (!p.do_expand) return launch_combine_cfg<2, 1, false, false>(p, num_sms, stream);
    if (p.num_topk <= 4) return p.weighted ? launch_combine_cfg<2, 4, true, true>(p, num_sms, stream) : launch_combine_cfg<2, 4, true, false>(p, num_sms, stream);
    return p.weighted ? launch_combine_cfg<1, 8, true, true>(p, num_sms, stream) : launch_combine_cfg<1, 8, true, false>(p, num_sms, stream);
}

}  // namespace ep
