// Plain and grouped GEMM on the tcgen05 core (see gemm_sm100.cuh): bf16 inputs, or e4m3 inputs
// with 1x128 (activations) and 128x128 (weights) fp32 block scales applied in the epilogue warps.
// The grouped form consumes the expanded (expert-major) output of the dispatch directly:
// `group_end` is the device-resident prefix array of the dispatch handle, so no host
// synchronisation sits between dispatch and the expert GEMM.
//
// The reference library contains no GEMM; this is the compute half of the fused MoE layer and of
// the all-gather -> GEMM / GEMM -> reduce-scatter operators (tp_fused.cu).
#include <algorithm>
#include <atomic>
#include <cstdlib>

#include "api.hpp"
#include "gemm_api.hpp"
#include "gemm_sm100.cuh"
#include "../common/launch.hpp"

namespace ep {
namespace gemm {

__device__ int pipe_status;         // see status_word

namespace {

// How the MMA issuers work: the whole warp walks the pipeline and one elected lane issues, the next barriers are tested before
// this k-block's instructions go out, and with an accumulator pass per k-block (software-scaled e4m3) one commit frees the
// stage and announces the pass. With one lane walking, testing and committing twice, a k-block cost the issuer 950 cycles,
// twice what the tensor pipe needs for it. (The bf16 pair kernel, whose k-block is longer, keeps the plain form: 1 % faster.)
struct Tile {
    int g, m0, m_end, n0;
    int kb0, kb1;       // k-blocks [kb0, kb1) of this tile (all of K unless the problem is grouped along K)
};

// Walks the tiles of a (grouped) problem in a fixed order: group, then bands of kBandM m-blocks, inside a band
// n-block then m-block.
struct Scheduler {
    static constexpr int kBandM = 8;
    const GemmParams& p;
    int tiles_n, BN, BM, BK;
    int g = 0, base = 0, start = 0, end = 0;
    __device__ Scheduler(const GemmParams& p_, int bn, int bm = gemm::BM, int bk = 64) : p(p_), tiles_n(p_.N / bn), BN(bn), BM(bm), BK(bk) {
        end = (p.group_end != nullptr && !p.k_grouped) ? p.group_end[0] : p.M;
    }
    __device__ bool get(int t, Tile& out) {
        if (p.k_grouped) {
            // groups along K: every group is a full M x N problem over its own range of k (the rows of one expert)
            const int tiles_m = ceil_div(p.M, BM);
            const int tiles = tiles_m * tiles_n;
            if (t >= p.num_groups * tiles) return false;
            const int gk = t / tiles, local = t % tiles;
            const int band = local / (kBandM * tiles_n), rem = local % (kBandM * tiles_n);
            const int band_m = min(kBandM, tiles_m - band * kBandM);
            out.g = gk;
            out.m0 = (band * kBandM + rem % band_m) * BM;
            out.m_end = p.M;
            out.n0 = (rem / band_m) * BN;
            const int k_start = gk == 0 ? 0 : align_up(p.group_end[gk - 1], p.group_alignment);
            const int k_end = max(p.group_end[gk], k_start);
            out.kb0 = k_start / BK;
            out.kb1 = ceil_div(k_end, BK);
            return true;
        }
        out.kb0 = 0;
        out.kb1 = ceil_div(p.K, BK);      // (only an MN-major problem may end inside a k-block: its missing rows load as zeros)
        while (g < p.num_groups) {
            const int rows = max(end - start, 0);
            const int tiles_m = ceil_div(rows, BM);
            const int tiles = tiles_m * tiles_n;
            if (t < base + tiles) {
                const int local = t - base;
                // m-blocks run fastest, in bands of kBandM m-blocks: the tiles that are in flight at the same time
                // then share few A row-blocks AND few B row-blocks, which keeps both resident in L2
                const int band = local / (kBandM * tiles_n), rem = local % (kBandM * tiles_n);
                const int band_m = min(kBandM, tiles_m - band * kBandM);
                out.g = g;
                out.m0 = start + (band * kBandM + rem % band_m) * BM;
                out.m_end = end;
                out.n0 = (rem / band_m) * BN;
                return true;
            }
            base += tiles;
            ++g;
            if (g < p.num_groups) {
                start = align_up(end, p.group_alignment);
                end = p.group_end[g];
            }
        }
        return false;
    }
};

template <int BN, bool kFp8>
struct Cfg {
    static constexpr int kEpiWarps = kFp8 ? 16 : 4;     // FP8: 4 lane quarters x 4 column quarters, so that many passes overlap
    static constexpr int kThreads = (2 + kEpiWarps) * 32;
    static constexpr int BK = kFp8 ? 128 : 64;          // one 128-byte swizzle span per row
    static constexpr int UMMA_K = kFp8 ? 32 : 16;
    static constexpr int A_BYTES = BM * 128, B_BYTES = BN * 128, STAGE = A_BYTES + B_BYTES;
    static constexpr int kStages = (192 * 1024) / STAGE;
    // accumulators in tensor memory: two tiles for bf16; with FP8 every k-block is an accumulator pass and the
    // epilogue is the slower side, so four passes may be in flight
    static constexpr int kAccStages = kFp8 ? 4 : 2;
    static constexpr int kBarBytes = (2 * kStages + 2 * kAccStages) * 8 + 16;
    static constexpr int kSmem = kStages * STAGE + kBarBytes + 1024;   // + slack to align the ring to 1024 bytes
    static constexpr int kTmemCols = kAccStages * BN;
};

// Sums of accumulator passes, two per 64-bit register: fma.rn.f32x2 rounds each half like fmaf and takes half the issue slots,
// which is what the epilogue warps of the software-scaled kernels are short of.
__device__ __forceinline__ uint64_t pack2(uint32_t lo, uint32_t hi) {
    uint64_t v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(lo), "r"(hi));
    return v;
}
template <int N>
__device__ __forceinline__ void fold(uint64_t* sum, const uint32_t (&r)[N], float scale) {
    const uint64_t s2 = pack2(__float_as_uint(scale), __float_as_uint(scale));
#pragma unroll
    for (int i = 0; i < N; i += 2) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(sum[i / 2]) : "l"(pack2(r[i], r[i + 1])), "l"(s2));
}
__device__ __forceinline__ void unpack_sums(const uint64_t* sum, bool zero, uint32_t (&r)[32]) {
#pragma unroll
    for (int i = 0; i < 32; ++i) r[i] = zero ? 0u : static_cast<uint32_t>(sum[i / 2] >> (32 * (i & 1)));
}

// Rows of a K-major A tile that the problem has (rows past the group's end give outputs that nobody stores): a tile with few
// of them is loaded in boxes of 32 rows. A decode batch has a handful of rows per expert, and the full box doubled what its
// tiles pull out of L2 (32 experts of 16 rows, 4096 x 7168 e4m3: 185 us with full boxes).
constexpr int kSmallBox = 32, kMaxSmallRows = 96;
__device__ __forceinline__ int small_boxes(int rows) { return rows <= kMaxSmallRows ? ceil_div(rows, kSmallBox) : 0; }
__device__ __forceinline__ void load_rows(uint8_t* dst, const CUtensorMap* map, const CUtensorMap* map_small, int boxes, int k, int row, uint64_t* bar) {
    if (boxes == 0) tma_load_2d(dst, map, k, row, bar);
    else for (int i = 0; i < boxes; ++i) tma_load_2d(dst + i * (kSmallBox * 128), map_small, k, row + i * kSmallBox, bar);
}

// Loads one operand tile of `rows` rows (K-major: one box) or `rows` columns of a [K, MN] matrix (MN-major: boxes of 64 x 64).
template <bool kMN>
__device__ __forceinline__ void load_operand(uint8_t* dst, const CUtensorMap* map, int k, int mn, int rows, uint64_t* bar) {
    if constexpr (!kMN) {
        tma_load_2d(dst, map, k, mn, bar);
    } else {
        for (int i = 0; i < rows / 64; ++i) tma_load_2d(dst + i * 8192, map, mn + i * 64, k, bar);
    }
}
template <bool kMN>
__device__ __forceinline__ void load_operand_pair(uint8_t* dst, const CUtensorMap* map, int k, int mn, int rows, uint32_t bar) {
    if constexpr (!kMN) {
        tma_load_2d_pair(dst, map, k, mn, bar);
    } else {
        for (int i = 0; i < rows / 64; ++i) tma_load_2d_pair(dst + i * 8192, map, mn + i * 64, k, bar);
    }
}

template <int BN, bool kFp8, bool kAMN = false, bool kBMN = false>
__global__ void __launch_bounds__(Cfg<BN, kFp8>::kThreads, 1)
gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_a32,
            const GemmParams p) {
    using C = Cfg<BN, kFp8>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::kStages * C::STAGE);
    uint64_t* empty = full + C::kStages;
    uint64_t* tmem_full = empty + C::kStages;
    uint64_t* tmem_empty = tmem_full + C::kAccStages;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + C::kAccStages);

    const int warp = warp_id(), lane = lane_id();
    const int num_kb = p.K / C::BK;
    launch_dependents();

    if (warp == 0 && lane == 0) {
        prefetch_tensormap(&map_a);
        prefetch_tensormap(&map_b);
        for (int s = 0; s < C::kStages; ++s) {
            mbar_init(full + s, 1);
            mbar_init(empty + s, 1);
        }
        for (int a = 0; a < C::kAccStages; ++a) {
            mbar_init(tmem_full + a, 1);
            // bf16: every epilogue thread arrives once per tile; FP8: one arrival per warp and k-block (an accumulator
            // pass per k-block makes per-thread arrivals the bottleneck)
            mbar_init(tmem_empty + a, kFp8 ? C::kEpiWarps : C::kEpiWarps * 32);
        }
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, C::kTmemCols);
        tmem_relinquish();
    }
    dependency_wait();           // everything above may run while the kernel ahead of this one drains
    const PipeCtx pc{p.error, globaltimer_ns() + p.timeout_ns};
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        if (lane == 0) {
            Scheduler sched(p, BN, BM, C::BK);
            Tile t;
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int ti = blockIdx.x; ok && sched.get(ti, t); ti += gridDim.x) {
                // (an MN-major B of a plain problem; group g of a grouped one starts at row g * K of the stacked [K, N] matrices)
                const int b_row = (p.k_grouped || kBMN ? 0 : t.g * p.N) + t.n0;
                const int boxes = kAMN ? 0 : small_boxes(t.m_end - t.m0);
                const uint32_t bytes = boxes == 0 ? C::STAGE : boxes * (kSmallBox * 128) + C::B_BYTES;
                for (int kb = t.kb0; kb < t.kb1; ++kb) {
                    if (!(ok = pipe_wait(pc, empty + s, ph ^ 1))) break;
                    uint8_t* sa = smem + s * C::STAGE;
                    mbar_arrive_expect_tx(full + s, bytes);
                    if constexpr (kAMN) load_operand<kAMN>(sa, &map_a, kb * C::BK, t.m0, BM, full + s);
                    else load_rows(sa, &map_a, &map_a32, boxes, kb * C::BK, t.m0, full + s);
                    load_operand<kBMN>(sa + C::A_BYTES, &map_b, kb * C::BK, b_row, BN, full + s);
                    if (++s == C::kStages) { s = 0; ph ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (see the note at the top)
        Scheduler sched(p, BN, BM, C::BK);
        Tile t;
        constexpr uint32_t idesc = make_idesc<kFp8>(BM, BN, kAMN, kBMN);
        const uint64_t da0 = kAMN ? make_smem_desc_mn(smem) : make_smem_desc(smem);
        const uint64_t db0 = kBMN ? make_smem_desc_mn(smem + C::A_BYTES) : make_smem_desc(smem + C::A_BYTES);
        int s = 0, acc = 0;
        uint32_t ph = 0, acc_ph = 0;
        bool ok = true, full_seen = false, empty_seen = false;
        for (int ti = blockIdx.x; ok && sched.get(ti, t); ti += gridDim.x) {
            if constexpr (!kFp8) pipe_wait_lane(pc, false, tmem_empty + acc, acc_ph ^ 1, ok);
            for (int kb = t.kb0; kb < t.kb1; ++kb) {
                if constexpr (kFp8) {
                    if (!(ok = pipe_wait_warp(pc, empty_seen, tmem_empty + acc, acc_ph ^ 1))) break;
                    if (!(ok = pipe_wait_warp(pc, full_seen, full + s, ph))) break;
                } else {
                    pipe_wait_lane(pc, full_seen, full + s, ph, ok);
                }
                tc_fence_after();
                const int s1 = s + 1 == C::kStages ? 0 : s + 1;
                const uint32_t ph1 = s1 == 0 ? ph ^ 1 : ph;
                full_seen = kFp8 ? pipe_test_warp(full + s1, ph1) : mbar_test_wait(full + s1, ph1);
                int acc1 = acc;
                uint32_t acc_ph1 = acc_ph;
                if constexpr (kFp8) {
                    acc1 = acc + 1 == C::kAccStages ? 0 : acc + 1;
                    acc_ph1 = acc1 == 0 ? acc_ph ^ 1 : acc_ph;
                    empty_seen = pipe_test_warp(tmem_empty + acc1, acc_ph1 ^ 1);
                }
                const uint64_t da = da0 + s * (C::STAGE >> 4), db = db0 + s * (C::STAGE >> 4);
                const uint32_t d_addr = tmem_base + acc * BN;
                if (elect_one() && ok) {
#pragma unroll
                    for (int k = 0; k < C::BK / C::UMMA_K; ++k) {
                        const uint32_t accumulate = kFp8 ? (k != 0) : (kb != t.kb0 || k != 0);
                        umma<kFp8>(d_addr, da + (kAMN ? 128 : 2) * k, db + (kBMN ? 128 : 2) * k, idesc, accumulate);
                    }
                    umma_commit(empty + s);         // (FP8: also tells the epilogue that this pass is complete)
                }
                s = s1;
                ph = ph1;
                acc = acc1;
                acc_ph = acc_ph1;
            }
            if constexpr (!kFp8) {
                if (elect_one() && ok) {
                    if (t.kb1 > t.kb0) umma_commit(tmem_full + acc);
                    else mbar_arrive(tmem_full + acc);        // an empty k range: nothing was issued, the epilogue writes zeros
                }
                if (++acc == C::kAccStages) { acc = 0; acc_ph ^= 1; }
            }
            if constexpr (!kFp8) ok = pipe_alive_warp(ok);
        }
    } else {
        // ------------------------------------------------------------ epilogue warps
        const int quarter = warp & 3;                  // the TMEM lanes this warp may read: [32 * quarter, +32)
        const int part = (warp - 2) / 4;               // fp8: which quarter of the columns
        constexpr int kCols = kFp8 ? BN / 4 : BN;      // columns per thread
        Scheduler sched(p, BN, BM, C::BK);
        Tile t;
        int acc = 0, s = 0;
        uint32_t acc_ph = 0, ph = 0;
        bool ok = true, seen = false;
        for (int ti = blockIdx.x; ok && sched.get(ti, t); ti += gridDim.x) {
            const int row = t.m0 + quarter * 32 + lane;
            const bool row_ok = row < t.m_end && row < p.M;
            const bool zero_row = !row_ok && p.zero_gap && row < p.M;   // alignment gap of the expanded layout
            const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
            __nv_bfloat16* c_row = p.C + (p.k_grouped ? static_cast<int64_t>(t.g) * p.c_group_stride : 0) +
                                   static_cast<int64_t>(row) * p.ldc + t.n0 + part * kCols;
            if constexpr (!kFp8) {
                pipe_wait_lane(pc, false, tmem_full + acc, acc_ph, ok);
                if (!(ok = pipe_alive_warp(ok))) break;
                tc_fence_after();
                const bool empty_k = t.kb1 <= t.kb0;
#pragma unroll 1
                for (int c = 0; c < BN / 32; ++c) {
                    uint32_t r[32];
                    tmem_ld_32x32(lane_addr + acc * BN + c * 32, r);
                    tmem_ld_wait();
                    if (empty_k) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) r[i] = 0u;
                    }
                    if (zero_row) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) r[i] = 0u;
                    }
                    if (row_ok || zero_row) store_row32(c_row + c * 32, r, p.c_wide != 0);
                }
                tc_fence_before();
                mbar_arrive(tmem_empty + acc);
                if (++acc == C::kAccStages) { acc = 0; acc_ph ^= 1; }
            } else {
                static_assert(kCols == 32, "the FP8 epilogue is written for 32 columns per thread");
                uint64_t sum[kCols / 2];
#pragma unroll
                for (int i = 0; i < kCols / 2; ++i) sum[i] = 0ull;
                const float* sfb = p.sfb + (static_cast<int64_t>(t.g) * (p.N / 128) + t.n0 / 128) * num_kb;
                const float* sfa = p.sfa + static_cast<int64_t>(row_ok ? row : 0) * p.sfa_row_stride;
                float next_scale = sfa[0] * sfb[0];
                for (int kb = 0; kb < num_kb; ++kb) {
                    const float scale = next_scale;
                    if (kb + 1 < num_kb) next_scale = sfa[static_cast<int64_t>(kb + 1) * p.sfa_k_stride] * sfb[kb + 1];
                    // The commit that frees stage s of the ring. (At most kAccStages <= kStages passes are ahead of this warp: the
                    // barrier cannot have completed another phase meanwhile.)
                    static_assert(C::kAccStages <= C::kStages, "the stage barrier would lap the epilogue");
                    if (!(ok = pipe_wait_warp(pc, seen, empty + s, ph))) break;
                    if (++s == C::kStages) { s = 0; ph ^= 1; }
                    tc_fence_after();
                    uint32_t r0[32];
                    tmem_ld_32x32(lane_addr + acc * BN + part * kCols, r0);
                    tmem_ld_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(tmem_empty + acc);      // the values are in registers: the accumulator can be reused
                    if (++acc == C::kAccStages) { acc = 0; acc_ph ^= 1; }
                    seen = pipe_test_warp(empty + s, ph);              // (asked before the sums, needed after them)
                    fold(sum, r0, scale);
                }
                if (ok && (row_ok || zero_row)) {
                    uint32_t r[32];
                    unpack_sums(sum, zero_row, r);
                    store_row32(c_row, r, p.c_wide != 0);
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, C::kTmemCols);
    }
}

// ==================================================================== CTA-pair kernel (bf16, 256 x 256 tiles)
// A cluster of two CTAs owns a 256 x 256 tile: CTA r loads rows [128 r, 128 r + 128) of the A tile and of the B tile
// (32 KB per stage instead of 48 KB for a lone CTA, so six stages fit and a third less shared-memory fill traffic
// per flop), the leader's MMA warp issues tcgen05.mma.cta_group::2 (M = 256), each CTA's epilogue warps drain the
// 128 accumulator rows in their own tensor memory. Barriers: `full` lives in the leader and counts the bytes of both
// CTAs; `empty` and `tmem_full` are signalled in both CTAs by one multicast commit; the leader's `tmem_empty`
// collects the epilogue warps of both CTAs.
struct PairCfg {
    static constexpr int BN = 256, BK = 64, UMMA_K = 16;
    static constexpr int A_BYTES = BM * 128, B_BYTES = (BN / 2) * 128, STAGE = A_BYTES + B_BYTES;
    static constexpr int kStages = 6;
    static constexpr int kAccStages = 2;
    static constexpr int kEpiWarps = 4;
    static constexpr int kThreads = (2 + kEpiWarps) * 32;
    static constexpr int kBarBytes = (2 * kStages + 2 * kAccStages) * 8 + 16;
    static constexpr int kSmem = kStages * STAGE + kBarBytes + 1024;
    static constexpr int kTmemCols = kAccStages * BN;
};

template <bool kAMN, bool kBMN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PairCfg::kThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const GemmParams p) {
    using C = PairCfg;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::kStages * C::STAGE);
    uint64_t* empty = full + C::kStages;
    uint64_t* tmem_full = empty + C::kStages;
    uint64_t* tmem_empty = tmem_full + C::kAccStages;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + C::kAccStages);

    const int warp = warp_id(), lane = lane_id();
    const uint32_t cta = cluster_ctarank();
    const bool leader = cta == 0;
    const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
    launch_dependents();

    if (warp == 0 && lane == 0) {
        prefetch_tensormap(&map_a);
        prefetch_tensormap(&map_b);
        for (int s = 0; s < C::kStages; ++s) {
            mbar_init(full + s, 1);
            mbar_init(empty + s, 1);
        }
        for (int a = 0; a < C::kAccStages; ++a) {
            mbar_init(tmem_full + a, 1);
            mbar_init(tmem_empty + a, 2 * C::kEpiWarps);
        }
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc_pair(tmem_slot, C::kTmemCols);
        tmem_relinquish_pair();
    }
    dependency_wait();
    const PipeCtx pc{p.error, globaltimer_ns() + p.timeout_ns};
    tc_fence_before();
    cluster_sync_all();          // barriers of both CTAs are initialised before anything arrives on them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer (both CTAs)
        if (lane == 0) {
            Scheduler sched(p, C::BN, 2 * BM, C::BK);
            Tile t;
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int ti = pair; ok && sched.get(ti, t); ti += num_pairs) {
                const int b_row = (p.k_grouped || kBMN ? 0 : t.g * p.N) + t.n0 + static_cast<int>(cta) * (C::BN / 2);
                for (int kb = t.kb0; kb < t.kb1; ++kb) {
                    if (!(ok = pipe_wait(pc, empty + s, ph ^ 1))) break;
                    uint8_t* sa = smem + s * C::STAGE;
                    if (leader) mbar_arrive_expect_tx(full + s, 2 * C::STAGE);
                    const uint32_t bar = map_to_cta(smem_u32(full + s), 0);
                    load_operand_pair<kAMN>(sa, &map_a, kb * C::BK, t.m0 + static_cast<int>(cta) * BM, BM, bar);
                    load_operand_pair<kBMN>(sa + C::A_BYTES, &map_b, kb * C::BK, b_row, C::BN / 2, bar);
                    if (++s == C::kStages) { s = 0; ph ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (leader only)
        if (leader && lane == 0) {
            Scheduler sched(p, C::BN, 2 * BM, C::BK);
            Tile t;
            constexpr uint32_t idesc = make_idesc<false>(2 * BM, C::BN, kAMN, kBMN);
            int s = 0, acc = 0;
            uint32_t ph = 0, acc_ph = 0;
            bool ok = true;
            for (int ti = pair; ok && sched.get(ti, t); ti += num_pairs) {
                if (!(ok = pipe_wait(pc, tmem_empty + acc, acc_ph ^ 1))) break;
                tc_fence_after();
                for (int kb = t.kb0; kb < t.kb1; ++kb) {
                    if (!(ok = pipe_wait(pc, full + s, ph))) break;
                    tc_fence_after();
                    const uint8_t* sa = smem + s * C::STAGE;
                    const uint64_t da = kAMN ? make_smem_desc_mn(sa) : make_smem_desc(sa);
                    const uint64_t db = kBMN ? make_smem_desc_mn(sa + C::A_BYTES) : make_smem_desc(sa + C::A_BYTES);
                    const uint32_t d_addr = tmem_base + acc * C::BN;
#pragma unroll
                    for (int k = 0; k < C::BK / C::UMMA_K; ++k)
                        umma_pair_bf16(d_addr, da + (kAMN ? 128 : 2) * k, db + (kBMN ? 128 : 2) * k, idesc, kb != t.kb0 || k != 0);
                    umma_commit_pair(empty + s);
                    if (++s == C::kStages) { s = 0; ph ^= 1; }
                }
                if (!ok) break;
                if (t.kb1 > t.kb0) {
                    umma_commit_pair(tmem_full + acc);
                } else {                                     // an empty k range: nothing was issued, the epilogues write zeros
                    mbar_arrive_cluster(map_to_cta(smem_u32(tmem_full + acc), 0));
                    mbar_arrive_cluster(map_to_cta(smem_u32(tmem_full + acc), 1));
                }
                if (++acc == C::kAccStages) { acc = 0; acc_ph ^= 1; }
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue warps (both CTAs, own 128 rows)
        const int quarter = warp & 3;
        Scheduler sched(p, C::BN, 2 * BM, C::BK);
        Tile t;
        int acc = 0;
        uint32_t acc_ph = 0;
        bool ok = true;
        for (int ti = pair; ok && sched.get(ti, t); ti += num_pairs) {
            const int row = t.m0 + static_cast<int>(cta) * BM + quarter * 32 + lane;
            const bool row_ok = row < t.m_end && row < p.M;
            const bool zero_row = !row_ok && p.zero_gap && row < p.M && row < align_up(t.m_end, p.group_alignment);
            const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
            __nv_bfloat16* c_row = p.C + (p.k_grouped ? static_cast<int64_t>(t.g) * p.c_group_stride : 0) + static_cast<int64_t>(row) * p.ldc + t.n0;
            pipe_wait_lane(pc, false, tmem_full + acc, acc_ph, ok);
            if (!(ok = pipe_alive_warp(ok))) break;
            tc_fence_after();
            const bool empty_k = t.kb1 <= t.kb0;
#pragma unroll 1
            for (int c = 0; c < C::BN / 32; ++c) {
                uint32_t r[32];
                tmem_ld_32x32(lane_addr + acc * C::BN + c * 32, r);
                tmem_ld_wait();
                if (empty_k) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) r[i] = 0u;
                }
                if (zero_row) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) r[i] = 0u;
                }
                if (row_ok || zero_row) store_row32(c_row + c * 32, r, p.c_wide != 0);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster_relaxed(map_to_cta(smem_u32(tmem_empty + acc), 0));     // (the loads have completed: tcgen05.wait::ld)
            if (++acc == C::kAccStages) { acc = 0; acc_ph ^= 1; }
        }
    }

    tc_fence_before();
    cluster_sync_all();          // nobody frees tensor memory, or leaves, while the peer may still signal or read
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, C::kTmemCols);
    }
}

// ==================================================================== CTA-pair kernel, e4m3 with software block scaling (256 x 256 tiles)
// Same division of labour as gemm_pair_kernel; a stage holds a 128-wide k-block (128 bytes per row), and every k-block is an
// accumulator pass of its own (two passes fit into the 512 columns of tensor memory): the leader commits the pass, the
// sixteen epilogue warps of each CTA -- four lane quarters x four column quarters of 64 -- take it into registers sixteen
// columns at a time and add it, times the product of the 1x128 scale of the row and the 128x128 scale of the weight block,
// to fp32 sums.
// What bounds it: the chain of one epilogue warp per pass (wait, four tensor-memory loads, the sums), 1300 cycles against 512
// of the tensor pipe at first. Hence: paired FMAs; the next barrier and scale asked for before the sums that precede their
// use; loads and sums alternate; scales come through a shared-memory ring that two warps of their own fill (read by the
// epilogue warps, one row per lane, they took 512 L1 cycles per pass); the second CTA's sixteen arrivals per pass travel as
// one. Passes of 128 columns, four in flight, were slower (619 against 525 us for 8 x 2048 x 4096 x 7168): the chain has the
// same length and there are twice as many.
struct PairFp8Cfg {
    static constexpr int BN = 256, BK = 128, UMMA_K = 32;
    static constexpr int A_BYTES = BM * 128, B_BYTES = (BN / 2) * 128, STAGE = A_BYTES + B_BYTES;
    static constexpr int kStages = 6;
    static constexpr int kAccStages = 2;
    static constexpr int kEpiWarps = 16, kSfWarps = 2;
    static constexpr int kThreads = (2 + kEpiWarps + kSfWarps) * 32;
    static constexpr int kSfChunk = 8, kSfStages = 4;                       // k-blocks per ring slot, slots
    static constexpr int kSfPitch = BM + 4;                                 // floats per k-block: 128 rows of A, 2 blocks of B
    static constexpr int kSfBytes = kSfStages * kSfChunk * kSfPitch * 4;
    static constexpr int kBarBytes = (2 * kStages + 2 * kAccStages + 2 * kSfStages) * 8 + 16;
    static constexpr int kSmem = kStages * STAGE + kSfBytes + kBarBytes + 1024;
    static constexpr int kTmemCols = kAccStages * BN;
    // 640 threads are launched with 96 registers each (61440); the epilogue's four warpgroups take 104, the fifth keeps 64:
    // 512 x 104 + 128 x 64 = 61440
    static constexpr int kEpiRegs = 104, kOtherRegs = 64;
    static constexpr int kTmaWarp = kEpiWarps, kMmaWarp = kEpiWarps + 1, kSfWarp = kEpiWarps + 2;
};

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PairFp8Cfg::kThreads, 1)
gemm_pair_fp8_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const GemmParams p) {
    using C = PairFp8Cfg;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    float* sf_ring = reinterpret_cast<float*>(smem + C::kStages * C::STAGE);          // [slots][k-blocks][rows of A, 2 of B]
    uint64_t* full = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(sf_ring) + C::kSfBytes);
    uint64_t* empty = full + C::kStages;
    uint64_t* tmem_empty = empty + C::kStages;
    uint64_t* tmem_drained = tmem_empty + C::kAccStages;       // the second CTA's own count of its epilogue warps
    uint64_t* sf_full = tmem_drained + C::kAccStages;
    uint64_t* sf_empty = sf_full + C::kSfStages;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sf_empty + C::kSfStages);

    const int warp = warp_id(), lane = lane_id();
    const uint32_t cta = cluster_ctarank();
    const bool leader = cta == 0;
    const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
    const int num_kb = p.K / C::BK;
    launch_dependents();

    if (warp == C::kTmaWarp && lane == 0) {
        prefetch_tensormap(&map_a);
        prefetch_tensormap(&map_b);
        for (int s = 0; s < C::kStages; ++s) {
            mbar_init(full + s, 1);
            mbar_init(empty + s, 1);
        }
        for (int a = 0; a < C::kAccStages; ++a) {
            mbar_init(tmem_empty + a, C::kEpiWarps + 1);      // the leader's epilogue warps and the second CTA's relay
            mbar_init(tmem_drained + a, C::kEpiWarps);
        }
        for (int i = 0; i < C::kSfStages; ++i) {
            mbar_init(sf_full + i, C::kSfWarps);
            mbar_init(sf_empty + i, C::kEpiWarps);
        }
        fence_mbar_init();
    }
    if (warp == C::kMmaWarp) {
        tmem_alloc_pair(tmem_slot, C::kTmemCols);
        tmem_relinquish_pair();
    }
    dependency_wait();
    const PipeCtx pc{p.error, globaltimer_ns() + p.timeout_ns};
    tc_fence_before();
    cluster_sync_all();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp < C::kEpiWarps) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(C::kEpiRegs));
        // ------------------------------------------------------------ epilogue warps (both CTAs, own 128 rows)
        const int quarter = warp & 3;                  // the TMEM lanes this warp may read: [32 * quarter, +32)
        const int part = warp >> 2;                    // which 64 of the 256 columns
        Scheduler sched(p, C::BN, 2 * BM, C::BK);
        Tile t;
        int acc = 0, slot = 0, s = 0;
        uint32_t sf_ph = 0, ph = 0;
        bool ok = true, seen = false;
        const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + part * 64;
        uint64_t* my_empty = leader ? tmem_empty : tmem_drained;
        static_assert(C::kAccStages <= C::kStages, "the stage barrier would lap the epilogue");
        for (int ti = pair; ok && sched.get(ti, t); ti += num_pairs) {
            uint64_t sum[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) sum[i] = 0ull;
            for (int kb0 = 0; kb0 < num_kb; kb0 += C::kSfChunk) {
                pipe_wait_lane(pc, false, sf_full + slot, sf_ph, ok);
                const float* sf = sf_ring + slot * C::kSfChunk * C::kSfPitch;
                const int n = min(C::kSfChunk, num_kb - kb0);
                float scale = sf[quarter * 32 + lane] * sf[BM + (part >> 1)];
                for (int j = 0; j < n; ++j) {
                    pipe_wait_lane(pc, seen, empty + s, ph, ok);      // the commit that frees stage s
                    tc_fence_after();
                    if (++s == C::kStages) { s = 0; ph ^= 1; }
                    const uint32_t addr = lane_addr + acc * C::BN;
                    uint32_t ra[16], rb[16];
                    tmem_ld_32x16(addr, ra);
                    tmem_ld_wait();
                    tmem_ld_32x16(addr + 16, rb);
                    fold(sum, ra, scale);
                    tmem_ld_wait();
                    tmem_ld_32x16(addr + 32, ra);
                    fold(sum + 8, rb, scale);
                    tmem_ld_wait();
                    tmem_ld_32x16(addr + 48, rb);
                    fold(sum + 16, ra, scale);
                    tmem_ld_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(my_empty + acc);      // the values are in registers: the accumulator can be reused
                    acc ^= 1;
                    seen = mbar_test_wait(empty + s, ph);
                    sf += C::kSfPitch;
                    float next = 0.f;
                    if (j + 1 < n) next = sf[quarter * 32 + lane] * sf[BM + (part >> 1)];
                    fold(sum + 24, rb, scale);
                    scale = next;
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(sf_empty + slot);       // (the last scale of the slot has been used)
                if (++slot == C::kSfStages) { slot = 0; sf_ph ^= 1; }
            }
            ok = pipe_alive_warp(ok);
            const int row = t.m0 + static_cast<int>(cta) * BM + quarter * 32 + lane;
            const bool row_ok = row < t.m_end && row < p.M;
            const bool zero_row = !row_ok && p.zero_gap && row < p.M && row < align_up(t.m_end, p.group_alignment);
            if (ok && (row_ok || zero_row)) {
                __nv_bfloat16* c_row = p.C + static_cast<int64_t>(row) * p.ldc + t.n0 + part * 64;
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    uint32_t r[32];
                    unpack_sums(sum + 16 * c, zero_row, r);
                    store_row32(c_row + c * 32, r, p.c_wide != 0);
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::kOtherRegs));
        if (warp == C::kTmaWarp) {
            // ------------------------------------------------------------ TMA producer (both CTAs)
            if (lane == 0) {
                Scheduler sched(p, C::BN, 2 * BM, C::BK);
                Tile t;
                int s = 0;
                uint32_t ph = 0;
                bool ok = true;
                for (int ti = pair; ok && sched.get(ti, t); ti += num_pairs) {
                    for (int kb = 0; kb < num_kb; ++kb) {
                        if (!(ok = pipe_wait(pc, empty + s, ph ^ 1))) break;
                        uint8_t* sa = smem + s * C::STAGE;
                        if (leader) mbar_arrive_expect_tx(full + s, 2 * C::STAGE);
                        const uint32_t bar = map_to_cta(smem_u32(full + s), 0);
                        tma_load_2d_pair(sa, &map_a, kb * C::BK, t.m0 + static_cast<int>(cta) * BM, bar);
                        tma_load_2d_pair(sa + C::A_BYTES, &map_b, kb * C::BK, t.g * p.N + t.n0 + static_cast<int>(cta) * (C::BN / 2), bar);
                        if (++s == C::kStages) { s = 0; ph ^= 1; }
                    }
                }
            }
        } else if (warp == C::kMmaWarp) {
            // ------------------------------------------------------------ MMA issuer (leader only)
            if (leader) {
                Scheduler sched(p, C::BN, 2 * BM, C::BK);
                Tile t;
                constexpr uint32_t idesc = make_idesc<true>(2 * BM, C::BN);
                const uint64_t da0 = make_smem_desc(smem), db0 = make_smem_desc(smem + C::A_BYTES);
                int s = 0, acc = 0;
                uint32_t ph = 0, acc_ph = 0;
                bool ok = true, full_seen = false, empty_seen = false;
                for (int ti = pair; ok && sched.get(ti, t); ti += num_pairs) {
                    for (int kb = 0; kb < num_kb; ++kb) {
                        pipe_wait_lane(pc, full_seen, full + s, ph, ok);
                        pipe_wait_lane(pc, empty_seen, tmem_empty + acc, acc_ph ^ 1, ok);
                        tc_fence_after();
                        const int s1 = s + 1 == C::kStages ? 0 : s + 1, acc1 = acc ^ 1;
                        const uint32_t ph1 = s1 == 0 ? ph ^ 1 : ph, acc_ph1 = acc1 == 0 ? acc_ph ^ 1 : acc_ph;
                        full_seen = mbar_test_wait(full + s1, ph1);
                        empty_seen = mbar_test_wait(tmem_empty + acc1, acc_ph1 ^ 1);
                        const uint64_t da = da0 + s * (C::STAGE >> 4), db = db0 + s * (C::STAGE >> 4);
                        const uint32_t d_addr = tmem_base + acc * C::BN;
                        if (elect_one() && ok) {
#pragma unroll
                            for (int k = 0; k < C::BK / C::UMMA_K; ++k) umma_pair_fp8(d_addr, da + 2 * k, db + 2 * k, idesc, k != 0);
                            umma_commit_pair(empty + s);           // frees the stage and tells the epilogues that this pass is complete
                        }
                        s = s1;
                        ph = ph1;
                        acc = acc1;
                        acc_ph = acc_ph1;
                    }
                    ok = pipe_alive_warp(ok);
                }
            } else if (!leader && lane == 0) {
                // relay: sixteen arrivals of this CTA's warps become one across the cluster, where each costs tens of cycles
                Scheduler sched(p, C::BN, 2 * BM, C::BK);
                Tile t;
                int acc = 0;
                uint32_t acc_ph = 0;
                bool ok = true;
                const uint32_t empty_bar = map_to_cta(smem_u32(tmem_empty), 0);
                for (int ti = pair; ok && sched.get(ti, t); ti += num_pairs)
                    for (int kb = 0; kb < num_kb; ++kb) {
                        if (!(ok = pipe_wait(pc, tmem_drained + acc, acc_ph))) break;
                        mbar_arrive_cluster_relaxed(empty_bar + acc * 8);
                        if (++acc == C::kAccStages) { acc = 0; acc_ph ^= 1; }
                    }
            }
        } else {
            // ------------------------------------------------------------ scale warps (both CTAs, own 128 rows)
            const int tid = (warp - C::kSfWarp) * 32 + lane;
            const bool vec = p.sfa_k_stride == 1 && p.sfa_row_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(p.sfa) & 15) == 0;
            Scheduler sched(p, C::BN, 2 * BM, C::BK);
            Tile t;
            int slot = 0;
            uint32_t sf_ph = 0;
            bool ok = true;
            for (int ti = pair; ok && sched.get(ti, t); ti += num_pairs) {
                const int last = min(t.m_end, p.M) - 1;
                const float* src[2];
#pragma unroll
                for (int i = 0; i < 2; ++i)      // (rows past the end repeat the last one: their sums are dropped)
                    src[i] = p.sfa + static_cast<int64_t>(min(t.m0 + static_cast<int>(cta) * BM + tid + i * 64, last)) * p.sfa_row_stride;
                const float* sfb = p.sfb + (static_cast<int64_t>(t.g) * (p.N / 128) + t.n0 / 128) * num_kb;
                for (int kb0 = 0; kb0 < num_kb; kb0 += C::kSfChunk) {
                    const int n = min(C::kSfChunk, num_kb - kb0);
                    float v[2][C::kSfChunk];
                    float vb = 0.f;
                    if (vec && n == C::kSfChunk) {
#pragma unroll
                        for (int i = 0; i < 2; ++i)
#pragma unroll
                            for (int j = 0; j < C::kSfChunk; j += 4) {
                                const float4 f = *reinterpret_cast<const float4*>(src[i] + kb0 + j);
                                v[i][j] = f.x;
                                v[i][j + 1] = f.y;
                                v[i][j + 2] = f.z;
                                v[i][j + 3] = f.w;
                            }
                    } else {
#pragma unroll
                        for (int i = 0; i < 2; ++i)
#pragma unroll
                            for (int j = 0; j < C::kSfChunk; ++j) v[i][j] = j < n ? src[i][static_cast<int64_t>(kb0 + j) * p.sfa_k_stride] : 0.f;
                    }
                    if (tid < 2 * C::kSfChunk && tid / 2 < n) vb = sfb[static_cast<int64_t>(tid & 1) * num_kb + kb0 + tid / 2];
                    pipe_wait_lane(pc, false, sf_empty + slot, sf_ph ^ 1, ok);
                    float* dst = sf_ring + slot * C::kSfChunk * C::kSfPitch;
#pragma unroll
                    for (int j = 0; j < C::kSfChunk; ++j) {
                        dst[j * C::kSfPitch + tid] = v[0][j];
                        dst[j * C::kSfPitch + tid + 64] = v[1][j];
                    }
                    if (tid < 2 * C::kSfChunk) dst[(tid / 2) * C::kSfPitch + BM + (tid & 1)] = vb;
                    __syncwarp();
                    if (lane == 0) mbar_arrive(sf_full + slot);
                    if (++slot == C::kSfStages) { slot = 0; sf_ph ^= 1; }
                }
                ok = pipe_alive_warp(ok);
            }
        }
    }

    tc_fence_before();
    cluster_sync_all();
    if (warp == C::kMmaWarp) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, C::kTmemCols);
    }
}

// ==================================================================== e4m3 with hardware block scaling (128 x 256 tiles)
// For scales that are exact powers of two the tensor core applies them itself (tcgen05.mma kind::mxf8f6f4.block_scale,
// UE8M0 scale factors in tensor memory), so a tile accumulates over ALL of K in tensor memory and the epilogue runs once
// per tile instead of once per k-block. Roles: TMA producer, MMA issuer, sixteen epilogue warps (four per lane quarter, 64
// columns each), four scale warps (one per lane quarter). Per k-block of 128 a scale warp writes the slot of that
// pipeline stage in tensor memory: 4 columns for the rows of A (1x128 scales: all four 32-wide slices share the byte)
// and 8 columns for the 256 columns of B (128x128 scales: two bytes per k-block, replicated); `full[s]` collects the
// producer's bytes and the four scale warps, `empty[s]` (an MMA commit) frees both the shared-memory stage and its
// scale slot. The scale bytes of a tile are staged in shared memory one tile ahead, so the feed never waits for memory.
// The accumulator (256 columns) is single-buffered: tensor memory has 512 columns and the scale slots need their own.
// (128 x 128 tiles with two accumulators were slower at every size, 1594 against 2200 TFLOP/s for long experts: 32 KB from L2
// per k-block at the 45 to 55 bytes per cycle that an SM gets.)
struct MxCfg {
    static constexpr int BN = 256, BK = 128, UMMA_K = 32;
    static constexpr int kEpiWarps = 16, kSfWarps = 4;
    static constexpr int kThreads = (2 + kEpiWarps + kSfWarps) * 32;
    static constexpr int A_BYTES = BM * 128, B_BYTES = BN * 128, STAGE = A_BYTES + B_BYTES;
    static constexpr int kStages = 192 * 1024 / STAGE;
    static constexpr int kSfCols = 16;                 // columns per scale slot: 4 (A) + 8 (B), padded to a store of 16
    static constexpr int kSfBase = 256;                // first scale column behind the accumulator
    static constexpr int kTmemCols = 512;
    static constexpr int kMaxKb = 64;                  // k-blocks whose scale bytes fit the staging area (K <= 8192)
    static constexpr int kSfPitch = BM + 16;           // per k-block: 128 bytes for the rows of A, 2 for B
    static constexpr int kSfStage = kMaxKb * kSfPitch;
    static constexpr int kBarBytes = (2 * kStages + 2) * 8 + 16;
    static constexpr int kSmem = kStages * STAGE + 2 * kSfStage + kBarBytes + 1024;
};

// Barrier of the scale warps of a CTA: true where all of them are `up`.
__device__ __forceinline__ bool scale_warps_meet(bool up, int threads) {
    uint32_t all;
    asm volatile(
        "{\n"
        ".reg .pred p, q;\n"
        "setp.ne.u32 p, %1, 0;\n"
        "barrier.cta.red.and.aligned.pred q, 3, %2, p;\n"
        "selp.u32 %0, 1, 0, q;\n"
        "}\n"
        : "=r"(all) : "r"(up ? 1u : 0u), "r"(threads) : "memory");
    return all != 0;
}

__device__ __forceinline__ uint32_t ue8m0_of(float scale) { return (__float_as_uint(scale) >> 23) & 0xffu; }

__global__ void __launch_bounds__(MxCfg::kThreads, 1)
gemm_mx_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_a32,
               const GemmParams p) {
    using C = MxCfg;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint8_t* sf_stage = smem + C::kStages * C::STAGE;                       // [2][kMaxKb][kSfPitch]
    uint64_t* full = reinterpret_cast<uint64_t*>(sf_stage + 2 * C::kSfStage);
    uint64_t* empty = full + C::kStages;
    uint64_t* tmem_full = empty + C::kStages;
    uint64_t* tmem_empty = tmem_full + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 1);

    const int warp = warp_id(), lane = lane_id();
    launch_dependents();

    if (warp == 0 && lane == 0) {
        prefetch_tensormap(&map_a);
        prefetch_tensormap(&map_b);
        for (int s = 0; s < C::kStages; ++s) {
            mbar_init(full + s, 1 + C::kSfWarps);      // the producer's arrival (+ bytes) and one arrival per scale warp
            mbar_init(empty + s, 1);
        }
        mbar_init(tmem_full, 1);
        mbar_init(tmem_empty, C::kEpiWarps);
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, C::kTmemCols);
        tmem_relinquish();
    }
    dependency_wait();           // everything above may run while the kernel ahead of this one drains
    const PipeCtx pc{p.error, globaltimer_ns() + p.timeout_ns};
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        if (lane == 0) {
            Scheduler sched(p, C::BN, BM, C::BK);
            Tile t;
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int ti = blockIdx.x; ok && sched.get(ti, t); ti += gridDim.x) {
                const int b_row = t.g * p.N + t.n0;
                const int boxes = small_boxes(t.m_end - t.m0);
                const uint32_t bytes = boxes == 0 ? C::STAGE : boxes * (kSmallBox * 128) + C::B_BYTES;
                for (int kb = t.kb0; kb < t.kb1; ++kb) {
                    if (!(ok = pipe_wait(pc, empty + s, ph ^ 1))) break;
                    uint8_t* sa = smem + s * C::STAGE;
                    mbar_arrive_expect_tx(full + s, bytes);
                    load_rows(sa, &map_a, &map_a32, boxes, kb * C::BK, t.m0, full + s);
                    tma_load_2d(sa + C::A_BYTES, &map_b, kb * C::BK, b_row, full + s);
                    if (++s == C::kStages) { s = 0; ph ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        Scheduler sched(p, C::BN, BM, C::BK);
        Tile t;
        const uint64_t da0 = make_smem_desc(smem), db0 = make_smem_desc(smem + C::A_BYTES);
        int s = 0;
        uint32_t ph = 0, acc_ph = 0;
        bool ok = true, full_seen = false;
        for (int ti = blockIdx.x; ok && sched.get(ti, t); ti += gridDim.x) {
            pipe_wait_lane(pc, false, tmem_empty, acc_ph ^ 1, ok);
            for (int kb = t.kb0; kb < t.kb1; ++kb) {
                pipe_wait_lane(pc, full_seen, full + s, ph, ok);
                tc_fence_after();
                const int s1 = s + 1 == C::kStages ? 0 : s + 1;
                const uint32_t ph1 = s1 == 0 ? ph ^ 1 : ph;
                full_seen = mbar_test_wait(full + s1, ph1);
                const uint64_t da = da0 + s * (C::STAGE >> 4), db = db0 + s * (C::STAGE >> 4);
                const uint32_t sfa = tmem_base + C::kSfBase + s * C::kSfCols, sfb = sfa + 4;
                if (elect_one() && ok) {
#pragma unroll
                    for (int k = 0; k < C::BK / C::UMMA_K; ++k)
                        umma_mx(tmem_base, da + 2 * k, db + 2 * k, make_idesc_mx(BM, C::BN, static_cast<uint32_t>(k)), (kb != t.kb0 || k != 0) ? 1u : 0u, sfa, sfb);
                    umma_commit(empty + s);
                }
                s = s1;
                ph = ph1;
            }
            if (elect_one() && ok) umma_commit(tmem_full);
            acc_ph ^= 1;
            ok = pipe_alive_warp(ok);
        }
    } else if (warp < 2 + C::kEpiWarps) {
        // ------------------------------------------------------------ epilogue warps: once per tile
        const int quarter = warp & 3;
        constexpr int kCols = C::BN / 4;               // columns per warp
        const int part = (warp - 2) / 4;
        Scheduler sched(p, C::BN, BM, C::BK);
        Tile t;
        uint32_t acc_ph = 0;
        bool ok = true;
        for (int ti = blockIdx.x; ok && sched.get(ti, t); ti += gridDim.x) {
            const int row = t.m0 + quarter * 32 + lane;
            const bool row_ok = row < t.m_end && row < p.M;
            const bool zero_row = !row_ok && p.zero_gap && row < p.M;
            const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + part * kCols;
            __nv_bfloat16* c_row = p.C + static_cast<int64_t>(row) * p.ldc + t.n0 + part * kCols;
            pipe_wait_lane(pc, false, tmem_full, acc_ph, ok);
            if (!(ok = pipe_alive_warp(ok))) break;
            tc_fence_after();
            // All of this warp's columns first: the accumulator is free for the next tile before anything is converted or
            // stored, which costs as much as several k-blocks.
            uint32_t r[kCols / 32][32];
#pragma unroll
            for (int c = 0; c < kCols / 32; ++c) tmem_ld_32x32(lane_addr + c * 32, r[c]);
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tmem_empty);
            if (row_ok || zero_row) {
#pragma unroll
                for (int c = 0; c < kCols / 32; ++c) {
                    if (zero_row) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) r[c][i] = 0u;
                    }
                    store_row32(c_row + c * 32, r[c], p.c_wide != 0);
                }
            }
            acc_ph ^= 1;
        }
    } else {
        // ------------------------------------------------------------ scale warps
        const int quarter = warp & 3;
        const int sf_tid = (warp - 2 - C::kEpiWarps) * 32 + lane;      // 0..127 = the row of the tile this thread stages
        const int kblocks = p.K / 128;
        const bool vec = p.sfa_k_stride == 1 && kblocks % 4 == 0 && p.sfa_row_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(p.sfa) & 15) == 0;
        Scheduler sched(p, C::BN, BM, C::BK);
        Tile t, nxt;
        auto stage_tile = [&](const Tile& tt, uint8_t* dst) {
            const int row = tt.m0 + sf_tid;
            const bool valid = row < tt.m_end && row < p.M;
            const float* src = p.sfa + static_cast<int64_t>(valid ? row : 0) * p.sfa_row_stride;
            // (sixteen bytes at a time where they are contiguous: a lane has a row of its own, 32 lines per load)
            if (vec) {
#pragma unroll 4
                for (int kb = 0; kb < kblocks; kb += 4) {
                    const float4 f = *reinterpret_cast<const float4*>(src + kb);
                    dst[kb * C::kSfPitch + sf_tid] = static_cast<uint8_t>(valid ? ue8m0_of(f.x) : 127u);
                    dst[(kb + 1) * C::kSfPitch + sf_tid] = static_cast<uint8_t>(valid ? ue8m0_of(f.y) : 127u);
                    dst[(kb + 2) * C::kSfPitch + sf_tid] = static_cast<uint8_t>(valid ? ue8m0_of(f.z) : 127u);
                    dst[(kb + 3) * C::kSfPitch + sf_tid] = static_cast<uint8_t>(valid ? ue8m0_of(f.w) : 127u);
                }
            } else {
                for (int kb = tt.kb0; kb < tt.kb1; ++kb)
                    dst[(kb - tt.kb0) * C::kSfPitch + sf_tid] = static_cast<uint8_t>(valid ? ue8m0_of(src[static_cast<int64_t>(kb) * p.sfa_k_stride]) : 127u);
            }
            const float* srcb = p.sfb + (static_cast<int64_t>(tt.g) * (p.N / 128) + tt.n0 / 128) * kblocks;
            for (int i = sf_tid; i < 2 * (tt.kb1 - tt.kb0); i += C::kSfWarps * 32) {
                const int h = i & 1, kb = tt.kb0 + (i >> 1);
                dst[(kb - tt.kb0) * C::kSfPitch + BM + h] = static_cast<uint8_t>(ue8m0_of(srcb[static_cast<int64_t>(h) * kblocks + kb]));
            }
        };
        // (a warp that has given up still comes to the barrier and takes the other scale warps with it)
        auto sf_barrier = [&](bool up) { return scale_warps_meet(up, C::kSfWarps * 32); };
        int s = 0, buf = 0;
        uint32_t ph = 0;
        bool ok = true;
        bool have = sched.get(blockIdx.x, t);
        if (have) stage_tile(t, sf_stage);
        sf_barrier(true);
        for (int ti = blockIdx.x; ok && have; ti += gridDim.x) {
            const bool have_next = sched.get(ti + gridDim.x, nxt);
            if (have_next) stage_tile(nxt, sf_stage + (buf ^ 1) * C::kSfStage);      // one tile ahead
            const uint8_t* mine = sf_stage + buf * C::kSfStage;
            // two k-blocks per round: the wait for the tensor-memory stores (a few hundred cycles) is paid once per round,
            // otherwise a scale warp, which sees every k-block, could not keep up with the tensor pipe
            for (int kb = t.kb0; kb < t.kb1; kb += 2) {
                const int n = min(2, t.kb1 - kb);
                int sj[2];
                for (int j = 0; j < n; ++j) {
                    sj[j] = s;
                    pipe_wait_lane(pc, false, empty + s, ph ^ 1, ok);
                    if (++s == C::kStages) { s = 0; ph ^= 1; }
                }
                tc_fence_after();
                for (int j = 0; j < n; ++j) {
                    const uint8_t* src = mine + (kb + j - t.kb0) * C::kSfPitch;
                    uint32_t v[16];
#pragma unroll
                    for (int i = 0; i < 4; ++i) v[i] = static_cast<uint32_t>(src[lane + 32 * i]) * 0x01010101u;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint32_t b = static_cast<uint32_t>(src[BM + h]) * 0x01010101u;
#pragma unroll
                        for (int i = 0; i < 4; ++i) v[4 + 4 * h + i] = b;
                    }
#pragma unroll
                    for (int i = 12; i < 16; ++i) v[i] = 0u;
                    tmem_st_32x16(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + C::kSfBase + sj[j] * C::kSfCols, v);
                }
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    for (int j = 0; j < n; ++j) {
                        mbar_arrive(full + sj[j]);
                    }
                }
            }
            ok = sf_barrier(ok);       // the next tile's bytes are complete; nobody reads this tile's any more
            buf ^= 1;
            t = nxt;
            have = have_next;
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, C::kTmemCols);
    }
}

// ==================================================================== e4m3 with hardware block scaling on CTA pairs (256 x 256 tiles)
// gemm_mx_kernel's scheme on the CTA-pair division of labour of gemm_pair_kernel: CTA r of the pair loads rows
// [128 r, 128 r + 128) of the A tile and of the B tile (32 KB per k-block and CTA instead of 48 KB: the block-scaled
// kernel on lone CTAs is bound by exactly this traffic), the leader issues tcgen05.mma.cta_group::2 with M = 256, each
// CTA's scale warps write the factors of its own 128 rows of A and of all 256 columns of B into its own tensor memory,
// each CTA's epilogue warps drain its 128 accumulator rows once per tile. `full` lives in the leader and collects the
// bytes of both CTAs and the eight scale warps of the pair; one multicast commit frees a stage (and its scale slot) in
// both CTAs; the leader's `tmem_empty` collects the epilogue warps of both.
struct MxPairCfg {
    static constexpr int BN = 256, BK = 128, UMMA_K = 32;
    static constexpr int kEpiWarps = 16, kSfWarps = 4;
    static constexpr int kThreads = (2 + kEpiWarps + kSfWarps) * 32;
    static constexpr int A_BYTES = BM * 128, B_BYTES = (BN / 2) * 128, STAGE = A_BYTES + B_BYTES;
    static constexpr int kStages = 6;
    static constexpr int kSfCols = 16, kSfBase = BN, kTmemCols = 512;
    static constexpr int kMaxKb = 64;
    static constexpr int kSfPitch = BM + 16;
    static constexpr int kSfStage = kMaxKb * kSfPitch;
    static constexpr int kBarBytes = (3 * kStages + 3) * 8 + 16;
    static constexpr int kSmem = kStages * STAGE + 2 * kSfStage + kBarBytes + 1024;
};

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(MxPairCfg::kThreads, 1)
gemm_mx_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const GemmParams p) {
    using C = MxPairCfg;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint8_t* sf_stage = smem + C::kStages * C::STAGE;
    uint64_t* full = reinterpret_cast<uint64_t*>(sf_stage + 2 * C::kSfStage);
    uint64_t* empty = full + C::kStages;
    uint64_t* tmem_full = empty + C::kStages;
    uint64_t* tmem_empty = tmem_full + 1;
    uint64_t* sf_done = tmem_empty + 1;                  // the second CTA's own count of its scale warps
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sf_done + C::kStages);

    const int warp = warp_id(), lane = lane_id();
    const uint32_t cta = cluster_ctarank();
    const bool leader = cta == 0;
    const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
    launch_dependents();

    if (warp == 0 && lane == 0) {
        prefetch_tensormap(&map_a);
        prefetch_tensormap(&map_b);
        for (int s = 0; s < C::kStages; ++s) {
            mbar_init(full + s, 1 + C::kSfWarps + 1);      // producer (+ bytes), the leader's scale warps, the second CTA's relay
            mbar_init(sf_done + s, C::kSfWarps);
            mbar_init(empty + s, 1);
        }
        mbar_init(tmem_full, 1);
        mbar_init(tmem_empty, 2 * C::kEpiWarps);
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc_pair(tmem_slot, C::kTmemCols);
        tmem_relinquish_pair();
    }
    dependency_wait();
    const PipeCtx pc{p.error, globaltimer_ns() + p.timeout_ns};
    tc_fence_before();
    cluster_sync_all();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer (both CTAs)
        if (lane == 0) {
            Scheduler sched(p, C::BN, 2 * BM, C::BK);
            Tile t;
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int ti = pair; ok && sched.get(ti, t); ti += num_pairs) {
                const int b_row = t.g * p.N + t.n0 + static_cast<int>(cta) * (C::BN / 2);
                for (int kb = t.kb0; kb < t.kb1; ++kb) {
                    if (!(ok = pipe_wait(pc, empty + s, ph ^ 1))) break;
                    uint8_t* sa = smem + s * C::STAGE;
                    if (leader) mbar_arrive_expect_tx(full + s, 2 * C::STAGE);
                    const uint32_t bar = map_to_cta(smem_u32(full + s), 0);
                    tma_load_2d_pair(sa, &map_a, kb * C::BK, t.m0 + static_cast<int>(cta) * BM, bar);
                    tma_load_2d_pair(sa + C::A_BYTES, &map_b, kb * C::BK, b_row, bar);
                    if (++s == C::kStages) { s = 0; ph ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (leader only)
        if (leader) {
            Scheduler sched(p, C::BN, 2 * BM, C::BK);
            Tile t;
            const uint64_t da0 = make_smem_desc(smem), db0 = make_smem_desc(smem + C::A_BYTES);
            int s = 0;
            uint32_t ph = 0, acc_ph = 0;
            bool ok = true, full_seen = false;
            for (int ti = pair; ok && sched.get(ti, t); ti += num_pairs) {
                pipe_wait_lane(pc, false, tmem_empty, acc_ph ^ 1, ok);
                for (int kb = t.kb0; kb < t.kb1; ++kb) {
                    pipe_wait_lane(pc, full_seen, full + s, ph, ok);
                    tc_fence_after();
                    const int s1 = s + 1 == C::kStages ? 0 : s + 1;
                    const uint32_t ph1 = s1 == 0 ? ph ^ 1 : ph;
                    full_seen = mbar_test_wait(full + s1, ph1);
                    const uint64_t da = da0 + s * (C::STAGE >> 4), db = db0 + s * (C::STAGE >> 4);
                    const uint32_t sfa = tmem_base + C::kSfBase + s * C::kSfCols, sfb = sfa + 4;
                    if (elect_one() && ok) {
#pragma unroll
                        for (int k = 0; k < C::BK / C::UMMA_K; ++k)
                            umma_mx_pair(tmem_base, da + 2 * k, db + 2 * k, make_idesc_mx(2 * BM, C::BN, static_cast<uint32_t>(k)),
                                         (kb != t.kb0 || k != 0) ? 1u : 0u, sfa, sfb);
                        umma_commit_pair(empty + s);
                    }
                    s = s1;
                    ph = ph1;
                }
                if (elect_one() && ok) umma_commit_pair(tmem_full);
                acc_ph ^= 1;
                ok = pipe_alive_warp(ok);
            }
        } else if (!leader && lane == 0) {
            // relay: the four arrivals of this CTA's scale warps become one across the cluster
            Scheduler sched(p, C::BN, 2 * BM, C::BK);
            Tile t;
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int ti = pair; ok && sched.get(ti, t); ti += num_pairs)
                for (int kb = t.kb0; kb < t.kb1; ++kb) {
                    if (!(ok = pipe_wait(pc, sf_done + s, ph))) break;
                    mbar_arrive_cluster_relaxed(map_to_cta(smem_u32(full + s), 0));
                    if (++s == C::kStages) { s = 0; ph ^= 1; }
                }
        }
    } else if (warp < 2 + C::kEpiWarps) {
        // ------------------------------------------------------------ epilogue warps (both CTAs, own 128 rows), once per tile
        const int quarter = warp & 3;
        const int part = (warp - 2) / 4;               // which 64 of the 256 columns
        Scheduler sched(p, C::BN, 2 * BM, C::BK);
        Tile t;
        uint32_t acc_ph = 0;
        bool ok = true;
        for (int ti = pair; ok && sched.get(ti, t); ti += num_pairs) {
            const int row = t.m0 + static_cast<int>(cta) * BM + quarter * 32 + lane;
            const bool row_ok = row < t.m_end && row < p.M;
            const bool zero_row = !row_ok && p.zero_gap && row < p.M && row < align_up(t.m_end, p.group_alignment);
            const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + part * 64;
            __nv_bfloat16* c_row = p.C + static_cast<int64_t>(row) * p.ldc + t.n0 + part * 64;
            pipe_wait_lane(pc, false, tmem_full, acc_ph, ok);
            if (!(ok = pipe_alive_warp(ok))) break;
            tc_fence_after();
            // All of this warp's columns first: the (only) accumulator is free for the next tile before anything is converted
            // or stored, which costs as much as several k-blocks.
            uint32_t r[2][32];
            tmem_ld_32x32(lane_addr, r[0]);
            tmem_ld_32x32(lane_addr + 32, r[1]);
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster_relaxed(map_to_cta(smem_u32(tmem_empty), 0));
            if (row_ok || zero_row) {
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    if (zero_row) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) r[c][i] = 0u;
                    }
                    store_row32(c_row + c * 32, r[c], p.c_wide != 0);
                }
            }
            acc_ph ^= 1;
        }
    } else {
        // ------------------------------------------------------------ scale warps (both CTAs)
        const int quarter = warp & 3;
        const int sf_tid = (warp - 2 - C::kEpiWarps) * 32 + lane;
        const int kblocks = p.K / 128;
        Scheduler sched(p, C::BN, 2 * BM, C::BK);
        Tile t, nxt;
        auto stage_tile = [&](const Tile& tt, uint8_t* dst) {
            const int row = tt.m0 + static_cast<int>(cta) * BM + sf_tid;
            const bool valid = row < tt.m_end && row < p.M;
            const float* src = p.sfa + static_cast<int64_t>(valid ? row : 0) * p.sfa_row_stride;
            for (int kb = tt.kb0; kb < tt.kb1; ++kb)
                dst[(kb - tt.kb0) * C::kSfPitch + sf_tid] = static_cast<uint8_t>(valid ? ue8m0_of(src[static_cast<int64_t>(kb) * p.sfa_k_stride]) : 127u);
            const float* srcb = p.sfb + (static_cast<int64_t>(tt.g) * (p.N / 128) + tt.n0 / 128) * kblocks;
            for (int i = sf_tid; i < 2 * (tt.kb1 - tt.kb0); i += C::kSfWarps * 32) {
                const int h = i & 1, kb = tt.kb0 + (i >> 1);
                dst[(kb - tt.kb0) * C::kSfPitch + BM + h] = static_cast<uint8_t>(ue8m0_of(srcb[static_cast<int64_t>(h) * kblocks + kb]));
            }
        };
        // (a warp that has given up still comes to the barrier and takes the other scale warps with it)
        auto sf_barrier = [&](bool up) { return scale_warps_meet(up, C::kSfWarps * 32); };
        int s = 0, buf = 0;
        uint32_t ph = 0;
        bool ok = true;
        bool have = sched.get(pair, t);
        if (have) stage_tile(t, sf_stage);
        sf_barrier(true);
        for (int ti = pair; ok && have; ti += num_pairs) {
            const bool have_next = sched.get(ti + num_pairs, nxt);
            if (have_next) stage_tile(nxt, sf_stage + (buf ^ 1) * C::kSfStage);
            const uint8_t* mine = sf_stage + buf * C::kSfStage;
            // two k-blocks per round: the wait for the tensor-memory stores (a few hundred cycles) is paid once per round,
            // otherwise a scale warp, which sees every k-block, could not keep up with the tensor pipe
            for (int kb = t.kb0; kb < t.kb1; kb += 2) {
                const int n = min(2, t.kb1 - kb);
                int sj[2];
                for (int j = 0; j < n; ++j) {
                    sj[j] = s;
                    pipe_wait_lane(pc, false, empty + s, ph ^ 1, ok);
                    if (++s == C::kStages) { s = 0; ph ^= 1; }
                }
                tc_fence_after();
                for (int j = 0; j < n; ++j) {
                    const uint8_t* src = mine + (kb + j - t.kb0) * C::kSfPitch;
                    uint32_t v[16];
#pragma unroll
                    for (int i = 0; i < 4; ++i) v[i] = static_cast<uint32_t>(src[lane + 32 * i]) * 0x01010101u;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint32_t b = static_cast<uint32_t>(src[BM + h]) * 0x01010101u;
#pragma unroll
                        for (int i = 0; i < 4; ++i) v[4 + 4 * h + i] = b;
                    }
#pragma unroll
                    for (int i = 12; i < 16; ++i) v[i] = 0u;
                    tmem_st_32x16(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + C::kSfBase + sj[j] * C::kSfCols, v);
                }
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    // (the stores are complete: tcgen05.wait::st above; the second CTA's relay passes its four arrivals on as one)
                    for (int j = 0; j < n; ++j) mbar_arrive(leader ? full + sj[j] : sf_done + sj[j]);
                }
            }
            ok = sf_barrier(ok);
            buf ^= 1;
            t = nxt;
            have = have_next;
        }
    }

    tc_fence_before();
    cluster_sync_all();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, C::kTmemCols);
    }
}

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                              const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn get_encode_fn() {
    static const EncodeFn fn = [] {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult res;
        const bool found = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &res) == cudaSuccess && res == cudaDriverEntryPointSuccess;
        return found ? reinterpret_cast<EncodeFn>(ptr) : nullptr;
    }();
    return fn;
}

}  // namespace

cudaError_t status_word(int** word) {
    constexpr int kDevices = 64;
    static std::atomic<int*> known[kDevices] = {};
    int device = 0;
    cudaError_t err = cudaGetDevice(&device);
    if (err != cudaSuccess) return err;
    const bool cached = device >= 0 && device < kDevices;
    if (cached && (*word = known[device].load(std::memory_order_relaxed)) != nullptr) return cudaSuccess;
    err = cudaGetSymbolAddress(reinterpret_cast<void**>(word), pipe_status);
    if (err == cudaSuccess && cached) known[device].store(*word, std::memory_order_relaxed);
    return err;
}

// 2-D K-major tensor map: `rows` x `cols` elements of `elem_bytes`, row pitch `row_stride_bytes`,
// box = `box_rows` x (128 / elem_bytes) elements, 128-byte swizzle.
bool make_kmajor_map(CUtensorMap* map, const void* base, int elem_bytes, uint64_t rows, uint64_t cols, uint64_t row_stride_bytes,
                     uint32_t box_rows) {
    EncodeFn encode = get_encode_fn();
    if (encode == nullptr) return false;
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {row_stride_bytes};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(128 / elem_bytes), box_rows};
    const cuuint32_t elem_strides[2] = {1, 1};
    const CUtensorMapDataType dtype = elem_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8;
    return encode(map, dtype, 2, const_cast<void*>(base), dims, strides, box, elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

namespace {

template <auto kKernel, typename C, typename... Args>
cudaError_t launch_tiles(int grid, cudaStream_t stream, const Args&... args) {
    static PreparedKernel prepared;
    const cudaError_t err = prepared.prepare(kKernel, C::kSmem);
    if (err != cudaSuccess) return err;
    return launch_early(kKernel, dim3(grid), dim3(C::kThreads), C::kSmem, stream, args...);
}

bool env_is(const char* name, char value) {
    const char* v = std::getenv(name);
    return v != nullptr && v[0] == value;
}

}  // namespace

// Which tiles a problem gets. What is known on the host: M rows in all (alignment gaps included), the number of groups, N, K.
enum class Tiles { kPair256, kLone256, kLone128 };

// Tiles of `bm` x `bn` over `units` at a time; about half of every group's last tile and of its alignment gap is padding.
int num_waves(const GemmParams& p, int bm, int bn, int units) {
    int64_t tiles_m;
    if (p.k_grouped) tiles_m = static_cast<int64_t>(p.num_groups) * ceil_div(p.M, bm);
    else if (p.group_end == nullptr) tiles_m = ceil_div(p.M, bm);
    else {
        const int64_t rows = std::max<int64_t>(p.M - static_cast<int64_t>(p.num_groups) * (std::min(p.group_alignment, 128) / 2), p.num_groups);
        tiles_m = std::max<int64_t>(p.num_groups, rows / bm + p.num_groups / 2);
    }
    return static_cast<int>(ceil_div<int64_t>(tiles_m * (p.N / bn), units));
}

cudaError_t launch_gemm(const GemmParams& params, const void* a, int64_t a_row_stride_bytes, const void* b, int64_t b_row_stride_bytes,
                        bool fp8, int num_sms, cudaStream_t stream) {
    GemmParams p = params;
    const int elem = fp8 ? 1 : 2, bk = fp8 ? 128 : 64;
    p.c_wide = (reinterpret_cast<uintptr_t>(p.C) | static_cast<uint64_t>(p.ldc) * 2 | static_cast<uint64_t>(p.c_group_stride) * 2) % 32 == 0;
    const bool k_tail_ok = p.a_mn && p.b_mn && !p.k_grouped && p.num_groups == 1;     // rows past the end load as zeros
    if (p.N % 128 != 0 || (p.K % bk != 0 && !k_tail_ok) || p.M <= 0) return cudaErrorInvalidValue;
    if (p.k_grouped && (fp8 || p.group_end == nullptr || p.group_alignment % bk != 0)) return cudaErrorInvalidValue;
    if ((p.a_mn || p.b_mn) && (fp8 || (p.a_mn && !p.b_mn) || (!p.k_grouped && p.num_groups != 1))) return cudaErrorInvalidValue;
    const uint64_t K = static_cast<uint64_t>(p.K), a_stride = static_cast<uint64_t>(a_row_stride_bytes), b_stride = static_cast<uint64_t>(b_row_stride_bytes);
    const uint64_t b_mats = p.k_grouped ? 1 : static_cast<uint64_t>(p.num_groups);
    // operand maps: K-major [rows, K] in boxes of `box` rows, or MN-major [K, columns] in boxes of 64 x 64
    auto map_of = [&](CUtensorMap* map, const void* base, bool mn, uint64_t rows, uint64_t mats, uint64_t stride, uint32_t box) {
        return mn ? make_kmajor_map(map, base, elem, mats * K, rows, stride, 64) : make_kmajor_map(map, base, elem, mats * rows, K, stride, box);
    };
    CUtensorMap map_a, map_a32 = {}, map_b;
    if (!map_of(&map_a, a, p.a_mn != 0, static_cast<uint64_t>(p.M), 1, a_stride, BM)) return cudaErrorInvalidValue;
    // (encoded on the host for every call: only the kernels of lone CTAs read it, and only for K-major rows)
    auto small_a_map = [&]() { return p.a_mn != 0 || map_of(&map_a32, a, false, static_cast<uint64_t>(p.M), 1, a_stride, kSmallBox); };
    auto map_b_of = [&](uint32_t box) { return map_of(&map_b, b, p.b_mn != 0, static_cast<uint64_t>(p.N), b_mats, b_stride, box); };
    const bool wide = p.N % 256 == 0, pairs = wide && num_sms >= 2;
    const int pair_grid = num_sms & ~1;

    // e4m3 with power-of-two scales: the block-scaled instruction kind (EP_GEMM_FP8_MX=0 keeps the software scaling)
    if (fp8 && p.scales_pow2 && !env_is("EP_GEMM_FP8_MX", '0') && !env_is("EP_GEMM_FP8_PAIR", '1') && wide && p.K / 128 <= MxCfg::kMaxKb) {
        // CTA pairs (EP_GEMM_FP8_MX_PAIR=1): 256 x 256 tiles, each CTA loads 128 rows of A and 128 of B. Opt-in: measured
        // no faster than lone CTAs (2.21 against 2.16 PFLOP/s), so the fill of shared memory from L2 is not what limits
        // the lone-CTA kernel; per k-block a CTA's shared memory takes 48 KB from TMA and hands 48 KB to the tensor
        // core in 541 tensor-pipe cycles either way, more than its 128 bytes per cycle.
        if (env_is("EP_GEMM_FP8_MX_PAIR", '1') && pairs) {
            if (!map_b_of(128)) return cudaErrorInvalidValue;
            return launch_tiles<gemm_mx_pair_kernel, MxPairCfg>(pair_grid, stream, map_a, map_b, p);
        }
        if (!map_b_of(256) || !small_a_map()) return cudaErrorInvalidValue;
        return launch_tiles<gemm_mx_kernel, MxCfg>(num_sms, stream, map_a, map_b, map_a32, p);
    }
    if (fp8) {
        // Software scaling (EP_GEMM_FP8_PAIR=1 / 0 forces / forbids pairs): a pass takes about 1160 cycles on a pair (256 x 256)
        // and 760 on a lone CTA (128 x 128), so pairs win unless their tiles are mostly padding or their last wave mostly
        // empty (8 experts of 700 rows, 4096 x 4096: 143 against 168 us; 16 of 20 rows: 100 against 66 us).
        const bool forced = env_is("EP_GEMM_FP8_PAIR", '1'), forbidden = env_is("EP_GEMM_FP8_PAIR", '0');
        const bool use_pair = pairs && !forbidden && (forced || num_waves(p, 256, 256, num_sms / 2) * 1.5f < num_waves(p, 128, 128, num_sms));
        if (!map_b_of(128) || (!use_pair && !small_a_map())) return cudaErrorInvalidValue;
        return use_pair ? launch_tiles<gemm_pair_fp8_kernel, PairFp8Cfg>(pair_grid, stream, map_a, map_b, p)
                        : launch_tiles<gemm_kernel<128, true>, Cfg<128, true>>(num_sms, stream, map_a, map_b, map_a32, p);
    }
    // bf16: CTA pairs with 256 x 256 tiles (EP_GEMM_CTA_PAIR=0: never), or one CTA per 128 x 256 tile, which takes 1.13 times
    // as long for its half but wastes less on ragged groups and in the last wave, and skips rows that do not exist (32 experts
    // of 16 rows, 4096 x 7168: 302 against 390 us; 8 of 2000 rows: 345 against 310 us).
    Tiles tiles = Tiles::kLone128;
    if (wide) tiles = pairs && !env_is("EP_GEMM_CTA_PAIR", '0') && num_waves(p, 256, 256, num_sms / 2) <= num_waves(p, 128, 256, num_sms) * 1.13f
                          ? Tiles::kPair256 : Tiles::kLone256;
    if (!map_b_of(tiles == Tiles::kLone256 ? 256 : 128)) return cudaErrorInvalidValue;
    if (tiles == Tiles::kPair256) {
        if (p.a_mn) return launch_tiles<gemm_pair_kernel<true, true>, PairCfg>(pair_grid, stream, map_a, map_b, p);
        return p.b_mn ? launch_tiles<gemm_pair_kernel<false, true>, PairCfg>(pair_grid, stream, map_a, map_b, p)
                      : launch_tiles<gemm_pair_kernel<false, false>, PairCfg>(pair_grid, stream, map_a, map_b, p);
    }
    if (!small_a_map()) return cudaErrorInvalidValue;
    if (tiles == Tiles::kLone256) {
        if (p.a_mn) return launch_tiles<gemm_kernel<256, false, true, true>, Cfg<256, false>>(num_sms, stream, map_a, map_b, map_a32, p);
        return p.b_mn ? launch_tiles<gemm_kernel<256, false, false, true>, Cfg<256, false>>(num_sms, stream, map_a, map_b, map_a32, p)
                      : launch_tiles<gemm_kernel<256, false>, Cfg<256, false>>(num_sms, stream, map_a, map_b, map_a32, p);
    }
    if (p.a_mn) return launch_tiles<gemm_kernel<128, false, true, true>, Cfg<128, false>>(num_sms, stream, map_a, map_b, map_a32, p);
    return p.b_mn ? launch_tiles<gemm_kernel<128, false, false, true>, Cfg<128, false>>(num_sms, stream, map_a, map_b, map_a32, p)
                  : launch_tiles<gemm_kernel<128, false>, Cfg<128, false>>(num_sms, stream, map_a, map_b, map_a32, p);
}

}  // namespace gemm
}  // namespace ep
