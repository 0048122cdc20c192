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

#include "api.hpp"
#include "../common/device_utils.cuh"

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
    launch_dependents();            // the move kernel's blocks may become resident; they wait for this grid's end
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
    for (int i = tid; i < kPlanWarps * (E + 1) + kPlanWarps * E; i += kPlanThreads) s_cnt[i] = 0;     // counters and masks
    __syncthreads();

    int* mine = s_cnt + warp * (E + 1);
    uint32_t* mask_of = s_mask + warp * E;
    int tokens_before = 0;
    if (in_regs) {
        uint32_t taken = 0;         // tokens of the warp with a valid expert
#pragma unroll
        for (int i = 0; i < kPlanRegTopk; ++i)
            if (e_reg[i] >= 0) {
                const uint32_t bit = 1u << ((lane + 32 * i) / K);
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
                pos_reg[i] = __popc(m & ((1u << ((lane + 32 * i) / K)) - 1u));
                if (pos_reg[i] == 0) mine[e_reg[i]] = __popc(m);      // the first token of a mask writes the count
            }
        }
    } else {
        // any number of batches per warp, any top-k: relative positions go to global memory and are completed below
        for (int base = a; base < b; base += 32) {
            const int t = base + lane;
            bool any = false;
            if (t < b) {
                for (int k = 0; k < K; ++k) {
                    const int e = load_topk_idx(p.topk_idx, p.idx32 != 0, static_cast<int64_t>(t) * K + k, E);
                    if (e >= 0) {
                        atomicOr(mask_of + e, 1u << lane);
                        any = true;
                    }
                }
            }
            __syncwarp();
            const uint32_t bal = __ballot_sync(0xffffffffu, any);
            if (t < b) {
                p.token_slot[t] = any ? tokens_before + __popc(bal & lanemask_lt()) : -1;
                for (int k = 0; k < K; ++k) {
                    const int64_t i = static_cast<int64_t>(t) * K + k;
                    const int e = load_topk_idx(p.topk_idx, p.idx32 != 0, i, E);
                    p.pair_row[i] = e >= 0 ? mine[e] + __popc(mask_of[e] & lanemask_lt()) : -1;
                }
            }
            tokens_before += __popc(bal);
            __syncwarp();
            if (t < b) {
                for (int k = 0; k < K; ++k) {
                    const int e = load_topk_idx(p.topk_idx, p.idx32 != 0, static_cast<int64_t>(t) * K + k, E);
                    if (e < 0) continue;
                    const uint32_t m = mask_of[e];
                    if (m != 0 && (m & lanemask_lt()) == 0) {
                        mine[e] += __popc(m);
                        mask_of[e] = 0;
                    }
                }
            }
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
    // first row of every expert (alignment applied): one warp scans; the column of the tokens has no start to add
    if (warp == 0) {
        int carry = 0;
        for (int e0 = 0; e0 < E; e0 += 32) {
            const int e = e0 + lane;
            int total = 0, before = 0;
            if (e < E)
                for (int c = 0; c < num_ctas; ++c) {
                    const int v = s_all[c * (E + 1) + e];
                    total += v;
                    if (c < cta) before += v;
                }
            const int aligned = align_up(total, p.expert_alignment);
            int incl = aligned;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += up;
            }
            const int start = carry + incl - aligned;
            if (e < E) {
                s_base[e] = start + before;
                if (cta == 0) {
                    if (p.host_counts != nullptr) p.host_counts[2 + e] = pack_epoch(p.epoch, static_cast<uint32_t>(aligned));
                    p.num_unaligned[e] = total;
                    p.psum_expert[e] = p.do_expand ? start + total : start + aligned;
                    if (p.recv_stats != nullptr) p.recv_stats[e] += total;
                }
            }
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0 && cta == 0) {
            p.psum_expert[E] = carry;
            if (p.host_counts != nullptr) p.host_counts[1] = pack_epoch(p.epoch, static_cast<uint32_t>(carry));
        }
    } else if (tid == 32) {
        int total = 0, before = 0;
        for (int c = 0; c < num_ctas; ++c) {
            const int v = s_all[c * (E + 1) + E];
            total += v;
            if (c < cta) before += v;
        }
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
        for (int t = a + lane; t < b; t += 32) {        // (every lane wrote the positions of the same tokens itself)
            if (p.token_slot[t] >= 0) p.token_slot[t] += slot_base;
            for (int k = 0; k < K; ++k) {
                const int64_t i = static_cast<int64_t>(t) * K + k;
                const int e = load_topk_idx(p.topk_idx, p.idx32 != 0, i, E);
                if (e >= 0) p.pair_row[i] += s_base[e] + mine[e];
            }
        }
    }
    if (cta == 0 && tid < 7) p.stamps[1 + tid] = globaltimer_ns();
}

// ==================================================================== move
// Sixteen bytes twice (or 32 bytes at once when the row allows it): a lane owns 32 consecutive bytes of the row.
__device__ __forceinline__ void load_32(const uint8_t* src, int bytes_left, bool wide, int4& lo, int4& hi) {
    lo = hi = make_int4(0, 0, 0, 0);
    if (wide && bytes_left >= 32) {
        asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(lo.x), "=r"(lo.y), "=r"(lo.z), "=r"(lo.w), "=r"(hi.x), "=r"(hi.y), "=r"(hi.z), "=r"(hi.w) : "l"(src));
        return;
    }
    if (bytes_left >= 16) lo = *reinterpret_cast<const int4*>(src);
    if (bytes_left >= 32) hi = *reinterpret_cast<const int4*>(src + 16);
}
__device__ __forceinline__ void store_32(uint8_t* dst, int bytes_left, bool wide, const int4& lo, const int4& hi) {
    if (wide && bytes_left >= 32) {
        asm volatile("st.global.L1::no_allocate.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                     ::"l"(dst), "r"(lo.x), "r"(lo.y), "r"(lo.z), "r"(lo.w), "r"(hi.x), "r"(hi.y), "r"(hi.z), "r"(hi.w) : "memory");
        return;
    }
    if (bytes_left >= 16) st_na_int4(dst, lo);
    if (bytes_left >= 32) st_na_int4(dst + 16, hi);
}

constexpr int kMoveThreads = 256;
constexpr int kMoveSlice = 1024;            // input bytes of a row that a warp takes at once (32 per lane)
constexpr int kMoveUnroll = 2;              // slices in flight per warp
constexpr int kPadRows = 4;                 // padding rows per zeroing work item

// Work item = (token, kMoveUnroll slices of its row), one warp each: whatever the number of tokens, the row is cut so
// that all SMs take part (64 tokens of hidden 7168 are 448 items). The item of the first slices also writes the token's
// routing words. Rows are streamed: every byte is read once and written once per destination row, 32 bytes per lane.
template <bool kQuant>
__global__ void __launch_bounds__(kMoveThreads) local_move_kernel(const __grid_constant__ LocalMoveParams p) {
    const int lane = lane_id();
    const int K = p.num_topk, T = p.num_tokens;
    const int slices = ceil_div(p.src_row_bytes, kMoveSlice * kMoveUnroll);
    const int64_t items = static_cast<int64_t>(T) * slices;
    const int warp_global = blockIdx.x * (kMoveThreads / 32) + warp_id(), num_warps = gridDim.x * (kMoveThreads / 32);
    const bool wide_in = p.wide_in != 0, wide_out = p.wide_out != 0;
    if (p.plan_ahead) dependency_wait();

    for (int64_t it = warp_global; it < items; it += num_warps) {
        const int t = static_cast<int>(it / slices), s = static_cast<int>(it % slices);
        const uint8_t* src = p.x + static_cast<int64_t>(t) * p.x_stride_bytes;
        const int off = s * kMoveSlice * kMoveUnroll + lane * 32;
        int4 lo[kMoveUnroll], hi[kMoveUnroll];
#pragma unroll
        for (int u = 0; u < kMoveUnroll; ++u) load_32(src + off + u * kMoveSlice, p.src_row_bytes - off - u * kMoveSlice, wide_in, lo[u], hi[u]);
        const int slot = p.token_slot[t];
        int row = -1;                                   // expanded layout: the row of top-k lane `lane`
        if (p.do_expand && lane < K) {
            row = p.pair_row[static_cast<int64_t>(t) * K + lane];
            if (row >= p.num_out_rows) row = -1;
        }
        uint32_t rows = p.do_expand ? __ballot_sync(0xffffffffu, row >= 0) : (slot >= 0 && slot < p.num_out_rows ? 1u : 0u);
        if (!p.do_expand) row = slot;                   // the same on every lane

        if (s == 0) {
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
            if (slot >= 0 && slot < p.num_idx_rows && lane < K) {
                const int64_t o = static_cast<int64_t>(slot) * K + lane;
                if (!p.do_expand) {
                    if (p.recv_topk_idx != nullptr) {
                        if (p.idx32) reinterpret_cast<int*>(p.recv_topk_idx)[o] = e;
                        else reinterpret_cast<int64_t*>(p.recv_topk_idx)[o] = e;
                    }
                    if (p.recv_topk_weights != nullptr)
                        p.recv_topk_weights[o] = p.mask_weights && e < 0 ? 0.f : p.topk_weights[static_cast<int64_t>(t) * K + lane];
                } else if (row >= 0 && p.recv_topk_weights != nullptr) {
                    p.recv_topk_weights[row] = p.topk_weights[static_cast<int64_t>(t) * K + lane];
                }
                if (p.write_metadata) {
                    int* md = p.recv_src_metadata + static_cast<int64_t>(slot) * (K + 2);
                    md[2 + lane] = p.do_expand ? row : -1;
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
                        const int r = __shfl_sync(0xffffffffu, row, __ffs(todo) - 1);
                        if (in) p.recv_sf[static_cast<int64_t>(r) * p.recv_sf_row_stride + static_cast<int64_t>(i) * p.recv_sf_pack_stride] = v;
                    }
                }
            }
        }

        // ---- payload
        if constexpr (!kQuant) {
            for (uint32_t todo = rows; todo != 0; todo &= todo - 1) {
                const int r = __shfl_sync(0xffffffffu, row, __ffs(todo) - 1);
                uint8_t* dst = p.recv_x + static_cast<int64_t>(r) * p.recv_x_pitch;
#pragma unroll
                for (int u = 0; u < kMoveUnroll; ++u)
                    store_32(dst + off + u * kMoveSlice, p.src_row_bytes - off - u * kMoveSlice, wide_out, lo[u], hi[u]);
            }
        } else {
            // a lane holds 16 channels, eight lanes a scale group of 128 (hidden is a multiple of 128: a group is all in or all out)
            float scale[kMoveUnroll];
            int4 q[kMoveUnroll];
#pragma unroll
            for (int u = 0; u < kMoveUnroll; ++u) {
                float amax = fmaxf(amax_bf16x8(lo[u]), amax_bf16x8(hi[u]));
                amax = warp_reduce_max_width(amax, 8);
                float inv;
                fp8_scale_from_amax(amax, p.pow2 != 0, scale[u], inv);
                uint32_t* qw = reinterpret_cast<uint32_t*>(&q[u]);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(h == 0 ? &lo[u] : &hi[u]);
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const float2 f0 = __bfloat1622float2(h2[2 * j]), f1 = __bfloat1622float2(h2[2 * j + 1]);
                        qw[2 * h + j] = pack4_e4m3(f0.x * inv, f0.y * inv, f1.x * inv, f1.y * inv);
                    }
                }
            }
            for (uint32_t todo = rows; todo != 0; todo &= todo - 1) {
                const int r = __shfl_sync(0xffffffffu, row, __ffs(todo) - 1);
                uint8_t* dst = p.recv_x + static_cast<int64_t>(r) * p.recv_x_pitch;
                float* sf = reinterpret_cast<float*>(p.recv_sf) + static_cast<int64_t>(r) * p.recv_sf_row_stride;
#pragma unroll
                for (int u = 0; u < kMoveUnroll; ++u) {
                    const int o = off + u * kMoveSlice;
                    if (o < p.src_row_bytes) {
                        st_na_int4(dst + o / 2, q[u]);
                        if ((lane & 7) == 0) sf[static_cast<int64_t>(o >> 8) * p.recv_sf_pack_stride] = scale[u];
                    }
                }
            }
        }
    }

    // ---- routing rows past the received count
    const int n = p.psum_rank[0];
    for (int64_t j = static_cast<int64_t>(n) * K + warp_global * 32 + lane; j < static_cast<int64_t>(p.num_idx_rows) * K; j += static_cast<int64_t>(num_warps) * 32) {
        const int i = static_cast<int>(j / K), k = static_cast<int>(j % K);
        if (!p.do_expand) {
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
    if (p.do_expand && p.do_zero_padding) {
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

constexpr int kCombineThreads = 256;

// Work item = (token, NV columns of 16 bytes per lane), a warp takes a run of consecutive items, so that the rows of a
// token are looked up once per token and not once per column. NR rows x NV columns = 128 bytes are in flight per lane
// before the first add; the adds run in ascending top-k order.
template <int NV, int NR, bool kWeighted>
__global__ void __launch_bounds__(kCombineThreads) local_combine_kernel(const __grid_constant__ LocalCombineParams p) {
    const int lane = lane_id();
    const int K = p.num_topk;
    const int vec_per_row = p.row_bytes / 16;
    const int cols = ceil_div(vec_per_row, 32 * NV);
    const int64_t items = static_cast<int64_t>(p.num_tokens) * cols;
    const int64_t num_warps = static_cast<int64_t>(gridDim.x) * (kCombineThreads / 32);
    const int64_t w = static_cast<int64_t>(blockIdx.x) * (kCombineThreads / 32) + warp_id();
    const int64_t first = items * w / num_warps, last = items * (w + 1) / num_warps;
    if (blockIdx.x == 0 && threadIdx.x == 0) p.timeline[0] = globaltimer_ns();
    int cur = -1, row = -1;         // token whose rows are held, this lane's row
    float wt = 1.f;
    uint32_t rows = 0;
    for (int64_t it = first; it < last; ++it) {
        const int t = static_cast<int>(it / cols), c = static_cast<int>(it % cols);
        if (t != cur) {
            cur = t;
            const int slot = p.token_slot[t];
            row = -1;
            if (lane < K && slot >= 0) row = p.do_expand ? p.recv_src_metadata[static_cast<int64_t>(slot) * (K + 2) + 2 + lane] : (lane == 0 ? slot : -1);
            if (row >= p.num_x_rows) row = -1;
            rows = __ballot_sync(0xffffffffu, row >= 0);
            if (kWeighted) wt = row >= 0 ? p.topk_weights[row] : 0.f;
            if (c == 0 && p.combined_topk_weights != nullptr && lane < K) {
                float v = 0.f;
                if (p.topk_weights != nullptr) {
                    if (p.do_expand) v = row >= 0 ? p.topk_weights[row] : 0.f;
                    else if (slot >= 0 && load_topk_idx(p.topk_idx, p.idx32 != 0, static_cast<int64_t>(t) * K + lane, p.num_experts) >= 0)
                        v = p.topk_weights[static_cast<int64_t>(slot) * K + lane];
                }
                p.combined_topk_weights[static_cast<int64_t>(t) * K + lane] = v;
            }
        }
        float acc[NV][8];
#pragma unroll
        for (int j = 0; j < NV; ++j)
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[j][i] = 0.f;
        const int v0 = c * 32 * NV + lane;
        for (uint32_t todo = rows; todo != 0;) {        // (uniform over the warp: lanes past the row's end take part in the shuffles)
            int4 raw[NR][NV];
            int rr[NR];
            float ww[NR];
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const int k = todo != 0 ? __ffs(todo) - 1 : 0;
                const int got = __shfl_sync(0xffffffffu, row, k);
                rr[r] = todo != 0 ? got : -1;
                if (kWeighted) ww[r] = __shfl_sync(0xffffffffu, wt, k);
                todo &= todo - 1;       // 0 stays 0
#pragma unroll
                for (int j = 0; j < NV; ++j)
                    if (rr[r] >= 0 && v0 + 32 * j < vec_per_row) raw[r][j] = ld_nc_int4(p.x + static_cast<int64_t>(rr[r]) * p.x_stride_bytes + (v0 + 32 * j) * 16);
            }
#pragma unroll
            for (int r = 0; r < NR; ++r)
#pragma unroll
                for (int j = 0; j < NV; ++j)
                    if (rr[r] >= 0 && v0 + 32 * j < vec_per_row) {
                        if (kWeighted) fma_bf16x8(acc[j], raw[r][j], ww[r]);
                        else add_bf16x8(acc[j], raw[r][j]);
                    }
        }
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const int v = v0 + 32 * j;
            if (v >= vec_per_row) continue;
            const int64_t off = static_cast<int64_t>(t) * p.row_bytes + v * 16;
            if (p.bias0 != nullptr || p.bias1 != nullptr) {
                if (p.round_partial) {
                    // a rank's partial sum is rounded once before it leaves the rank, then the biases are added
#pragma unroll
                    for (int i = 0; i < 8; ++i) acc[j][i] = __bfloat162float(__float2bfloat16_rn(acc[j][i]));
                }
                if (p.bias0 != nullptr) add_bf16x8(acc[j], ld_nc_int4(p.bias0 + off));
                if (p.bias1 != nullptr) add_bf16x8(acc[j], ld_nc_int4(p.bias1 + off));
            }
            int4 out;
            __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&out);
#pragma unroll
            for (int i = 0; i < 4; ++i) o2[i] = __floats2bfloat162_rn(acc[j][2 * i], acc[j][2 * i + 1]);
            st_na_int4(p.combined_x + off, out);
        }
    }
    if (threadIdx.x == 0 && (blockIdx.x == 0 || blockIdx.x == gridDim.x - 1))
        atomicMax(reinterpret_cast<unsigned long long*>(p.timeline + 1), static_cast<unsigned long long>(globaltimer_ns()));
}

template <typename Kernel, typename Params>
cudaError_t launch_plain(Kernel kernel, const Params& p, int grid, int block, cudaStream_t stream, bool programmatic) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = programmatic ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, p);
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
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ctas;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, local_plan_kernel, p);
}

cudaError_t launch_local_move(const LocalMoveParams& params, bool quant, int num_sms, bool programmatic, cudaStream_t stream) {
    LocalMoveParams p = params;
    static PreparedKernel prepared[2];
    cudaError_t err = quant ? prepared[1].prepare(local_move_kernel<true>, 0) : prepared[0].prepare(local_move_kernel<false>, 0);
    if (err != cudaSuccess) return err;
    const uint64_t in_bits = reinterpret_cast<uintptr_t>(p.x) | static_cast<uint64_t>(p.x_stride_bytes);
    const uint64_t out_bits = reinterpret_cast<uintptr_t>(p.recv_x) | static_cast<uint64_t>(p.recv_x_pitch);
    p.wide_in = in_bits % 32 == 0;
    p.wide_out = out_bits % 32 == 0;
    const int64_t items = static_cast<int64_t>(p.num_tokens) * ceil_div(p.src_row_bytes, kMoveSlice * kMoveUnroll) +
                          (p.do_expand && p.do_zero_padding ? static_cast<int64_t>(p.num_experts) * ceil_div(p.expert_alignment, kPadRows) : 0);
    const int64_t want = ceil_div<int64_t>(items, kMoveThreads / 32), most = static_cast<int64_t>(num_sms) * 8;
    const int grid = static_cast<int>(want < 1 ? 1 : (want > most ? most : want));
    return quant ? launch_plain(local_move_kernel<true>, p, grid, kMoveThreads, stream, programmatic)
                 : launch_plain(local_move_kernel<false>, p, grid, kMoveThreads, stream, programmatic);
}

template <int NV, int NR, bool kWeighted>
static cudaError_t launch_combine_cfg(const LocalCombineParams& p, int num_sms, cudaStream_t stream) {
    static PreparedKernel prepared;
    static int per_sm = 0;
    cudaError_t err = prepared.prepare(local_combine_kernel<NV, NR, kWeighted>, 0);
    if (err != cudaSuccess) return err;
    if (per_sm == 0) {
        int n = 0;
        err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, local_combine_kernel<NV, NR, kWeighted>, kCombineThreads, 0);
        if (err != cudaSuccess) return err;
        per_sm = n < 1 ? 1 : n;
    }
    const int64_t items = static_cast<int64_t>(p.num_tokens) * ceil_div(p.row_bytes / 16, 32 * NV);
    const int64_t want = ceil_div<int64_t>(items, kCombineThreads / 32), most = static_cast<int64_t>(num_sms) * per_sm;
    return launch_plain(local_combine_kernel<NV, NR, kWeighted>, p, static_cast<int>(want > most ? most : want), kCombineThreads, stream, false);
}

cudaError_t launch_local_combine(const LocalCombineParams& p, int num_sms, cudaStream_t stream) {
    if (p.num_tokens == 0) return cudaSuccess;
    // one row per token: four columns of it; up to four rows: two columns; more: eight rows of one column (128 bytes per lane or less)
    if (!p.do_expand) return launch_combine_cfg<4, 1, false>(p, num_sms, stream);
    if (p.num_topk <= 4) return p.weighted ? launch_combine_cfg<2, 4, true>(p, num_sms, stream) : launch_combine_cfg<2, 4, false>(p, num_sms, stream);
    return p.weighted ? launch_combine_cfg<1, 8, true>(p, num_sms, stream) : launch_combine_cfg<1, 8, false>(p, num_sms, stream);
}

}  // namespace ep
