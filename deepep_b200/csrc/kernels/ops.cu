// Small memory-bound operators of the MoE layer (sm_100a): router top-k + softmax, SwiGLU (with an
// optional fused 1x128 e4m3 cast for the second expert GEMM), 1x128 block quantisation and
// dequantisation, and a 2-D bf16 transpose for weight-gradient GEMMs.
// All of them stream each byte once (32-byte accesses, no shared-memory staging except the
// transpose) and are bound by HBM bandwidth.
//
// The reference has none of these as kernels; its test helpers (deep_ep/utils/math.py:30-56) are
// the arithmetic these follow.
#include <algorithm>
#include <initializer_list>

#include "ops_api.hpp"
#include "../common/device_utils.cuh"
#include "../common/launch.hpp"

namespace ep {
namespace ops {

namespace {

// ---------------------------------------------------------------- router: top-k over experts, softmax over the selection
// one warp per token; the warp keeps the row in registers (experts <= 2048 -> 64 values per lane)
__device__ __forceinline__ float to_float(float v) { return v; }
__device__ __forceinline__ float to_float(__nv_bfloat16 v) { return __bfloat162float(v); }

template <int kPerLane, typename Logit>
__global__ void __launch_bounds__(256) router_topk_kernel(const Logit* __restrict__ logits, int64_t row_stride, int num_tokens, int num_experts, int num_topk,
                                                          int64_t* __restrict__ topk_idx, float* __restrict__ topk_weights) {
    launch_dependents();
    dependency_wait();
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = lane_id();
    if (warp >= num_tokens) return;
    const Logit* row = logits + static_cast<int64_t>(warp) * row_stride;
    float v[kPerLane];
#pragma unroll
    for (int i = 0; i < kPerLane; ++i) {
        const int e = i * 32 + lane;
        v[i] = e < num_experts ? to_float(row[e]) : -INFINITY;
    }
    float sel_val = 0.f;
    int sel_idx = -1;
    float vmax = -INFINITY;
    for (int k = 0; k < num_topk; ++k) {
        float best = -INFINITY;
        int best_e = 0x7fffffff;
#pragma unroll
        for (int i = 0; i < kPerLane; ++i) {
            const int e = i * 32 + lane;
            if (v[i] > best) { best = v[i]; best_e = e; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oe = __shfl_xor_sync(0xffffffffu, best_e, o);
            if (ob > best || (ob == best && oe < best_e)) { best = ob; best_e = oe; }   // ties: lowest expert id
        }
        if (k == 0) vmax = best;
        if ((best_e & 31) == lane) {
#pragma unroll
            for (int i = 0; i < kPerLane; ++i)
                if (i == (best_e >> 5)) v[i] = -INFINITY;
        }
        if (lane == k) { sel_val = best; sel_idx = best_e; }
    }
    float ex = (lane < num_topk) ? __expf(sel_val - vmax) : 0.f;
    float sum = ex;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane < num_topk) {
        topk_idx[static_cast<int64_t>(warp) * num_topk + lane] = sel_idx;
        topk_weights[static_cast<int64_t>(warp) * num_topk + lane] = ex / sum;
    }
}

// Router weights fp32 [experts, hidden] -> bf16 [padded experts, hidden], zero rows behind the last expert (the GEMM tiles
// its columns in multiples of 128).
__global__ void __launch_bounds__(256) router_weights_kernel(const float* __restrict__ w, int num_experts, int padded, int hidden, __nv_bfloat16* __restrict__ out) {
    launch_dependents();
    dependency_wait();
    const int64_t n = static_cast<int64_t>(padded) * hidden / 8, real = static_cast<int64_t>(num_experts) * hidden / 8;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        int4 v = make_int4(0, 0, 0, 0);
        if (i < real) {
            const float4 a = reinterpret_cast<const float4*>(w)[2 * i], b = reinterpret_cast<const float4*>(w)[2 * i + 1];
            __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v);
            h[0] = __floats2bfloat162_rn(a.x, a.y);
            h[1] = __floats2bfloat162_rn(a.z, a.w);
            h[2] = __floats2bfloat162_rn(b.x, b.y);
            h[3] = __floats2bfloat162_rn(b.z, b.w);
        }
        reinterpret_cast<int4*>(out)[i] = v;
    }
}

// ---------------------------------------------------------------- streaming kernels
// One piece of sixteen channels per lane and nothing else: neighbouring lanes have neighbouring pieces, and a grid of many
// short blocks streams faster than a resident grid that loops over the same work (cast of 8192 x 7168: 29 against 31-34 us).
// All of them are bound by HBM once the arithmetic per channel is short enough to hide. The pieces are numbered through the
// whole tensor: with a warp per (row, 512 channels) narrow rows left most lanes without work (SwiGLU of 200000 x 8 took 66
// us, the cast of 300000 x 128 58). Widths of casts are multiples of 128, so the eight lanes of a scale group are one row's.
constexpr int kPiece = 16, kSpan = 512;

struct RowCol {
    int row, ch;        // first channel of this lane
};
__device__ __forceinline__ RowCol row_piece(int pieces) {       // pieces of a row; the last rows' warps may reach past the tensor
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, row = i / static_cast<uint32_t>(pieces);
    return {static_cast<int>(row), static_cast<int>(i - row * static_cast<uint32_t>(pieces)) * kPiece};
}
// A warp per (row, 512 channels), for kernels whose lanes work on a row together.
__device__ __forceinline__ RowCol row_col(int columns) {
    const uint32_t w = blockIdx.x * (blockDim.x >> 5) + warp_id();
    const uint32_t row = w / static_cast<uint32_t>(columns);
    return {static_cast<int>(row), static_cast<int>(w - row * static_cast<uint32_t>(columns)) * kSpan + lane_id() * 16};
}

// Gradient of the router from the gradient of the top-k weights, one warp per (token, 512 channels): the softmax Jacobian
// over the selected experts, d logit_k = w_k (dw_k - sum_j w_j dw_j), as the bf16 row that the weight gradient contracts
// (zeros elsewhere), and dx += sum_k d logit_k * router[expert k] in fp32. Only the selected rows of the router weights are
// read, from L1 and L2, and the sum is rounded once (a GEMM over all padded experts and an elementwise addition took 14 us
// for 1000 x 2048 where this takes 4).
__global__ void __launch_bounds__(256) router_backward_kernel(const int64_t* __restrict__ topk_idx, const float* __restrict__ w, const float* __restrict__ dw,
                                                              int num_tokens, int num_topk, int num_experts, int padded, int hidden, int columns,
                                                              const __nv_bfloat16* __restrict__ router, __nv_bfloat16* dx, __nv_bfloat16* __restrict__ dlogits) {
    launch_dependents();
    dependency_wait();
    const RowCol rc = row_col(columns);
    const int t = rc.row, lane = lane_id();
    if (t >= num_tokens) return;
    const int64_t o = static_cast<int64_t>(t) * num_topk + lane;
    const float wv = lane < num_topk ? w[o] : 0.f, dv = lane < num_topk ? dw[o] : 0.f;
    const int64_t sel = lane < num_topk ? topk_idx[o] : -1;
    const int e = sel >= 0 && sel < num_experts ? static_cast<int>(sel) : -1;
    float inner = wv * dv;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) inner += __shfl_xor_sync(0xffffffffu, inner, s);
    const float g = wv * (dv - inner);
    if (rc.ch == lane * 16) {       // the first column writes the row of the logits' gradient
        __nv_bfloat16* row = dlogits + static_cast<int64_t>(t) * padded;
        for (int i = lane * 8; i < padded; i += 256) *reinterpret_cast<int4*>(row + i) = make_int4(0, 0, 0, 0);
        __syncwarp();               // the zeros of all lanes are in place
        if (e >= 0) row[e] = __float2bfloat16_rn(g);
    }
    const int halves = min(2, (hidden - rc.ch) / 8);       // 16-byte pieces of this lane (hidden is a multiple of 8)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const bool in = h < halves;
        __nv_bfloat16* at = dx + static_cast<int64_t>(t) * hidden + rc.ch + h * 8;
        int4 v = in ? *reinterpret_cast<const int4*>(at) : make_int4(0, 0, 0, 0);
        __nv_bfloat162* v2 = reinterpret_cast<__nv_bfloat162*>(&v);
        float2 acc[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i] = __bfloat1622float2(v2[i]);
        for (int k = 0; k < num_topk; ++k) {
            const int ek = __shfl_sync(0xffffffffu, e, k);
            const float gk = __shfl_sync(0xffffffffu, g, k);
            if (ek < 0 || !in) continue;
            const int4 r = *reinterpret_cast<const int4*>(router + static_cast<int64_t>(ek) * hidden + rc.ch + h * 8);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 f = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(&r)[i]);
                acc[i].x = fmaf(gk, f.x, acc[i].x);
                acc[i].y = fmaf(gk, f.y, acc[i].y);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) v2[i] = __floats2bfloat162_rn(acc[i].x, acc[i].y);
        if (in) *reinterpret_cast<int4*>(at) = v;
    }
}

// Is the row in an alignment gap of the expanded layout (behind the rows of its expert)? The row belongs to the first group
// whose aligned end lies behind it. Warp-collective, the same row on every lane:
__device__ __forceinline__ bool in_gap(const RowGroups& g, int row) {
    if (g.ends == nullptr) return false;
    for (int base = 0; base < g.num; base += 32) {
        const int i = base + lane_id();
        const int end = i < g.num ? g.ends[i] : 0x3fffffff;
        const uint32_t behind = __ballot_sync(0xffffffffu, align_up(end, g.alignment) > row);
        if (behind != 0) {
            const int src = __ffs(behind) - 1;
            return base + src >= g.num || row >= __shfl_sync(0xffffffffu, end, src);
        }
    }
    return true;
}
// ... and any row on any lane of a whole warp.
__device__ __forceinline__ bool in_gap_of_lane(const RowGroups& g, int row) {
    if (g.ends == nullptr) return false;
    if (__all_sync(0xffffffffu, row == __shfl_sync(0xffffffffu, row, 0))) return in_gap(g, row);
    int lo = 0, hi = g.num;
    while (lo < hi) {
        const int mid = (lo + hi) / 2;
        if (align_up(g.ends[mid], g.alignment) > row) hi = mid;
        else lo = mid + 1;
    }
    return lo == g.num || row >= g.ends[lo];
}

// 1 / (1 + e^-x) with the hardware's exponential and reciprocal (with a correctly rounded division the forward kernel issued 40
// instructions per value and ran at 45 % of the memory rate). The exponential is taken of -|x|, so that the denominator lies
// in [1, 2]: the fast division gives 0 for denominators above 2^126, for x below -87.3, where the sigmoid is 1e-38 and its
// products need not be that small. (That costs the cast forward kernel 6 %, 62 to 66 us for 32768 x 2048, the others 1 %; a
// branch for such values alone cost the backward kernel 17 %.) Against 64 bits the bf16 results are off by 1.6594e-3 of their
// norm for N(0, 1) inputs, as with the rounded division.
__device__ __forceinline__ float sigmoid(float x) {
    const float t = __expf(-fabsf(x)), r = __fdividef(1.f, 1.f + t);
    return x >= 0.f ? r : t * r;
}

__device__ __forceinline__ void unpack16(const int4& lo, const int4& hi, float (&f)[16]) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(h == 0 ? &lo : &hi);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 t = __bfloat1622float2(h2[j]);
            f[8 * h + 2 * j] = t.x;
            f[8 * h + 2 * j + 1] = t.y;
        }
    }
}
__device__ __forceinline__ void pack16(const float (&f)[16], int4& lo, int4& hi) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        __nv_bfloat162* h2 = reinterpret_cast<__nv_bfloat162*>(h == 0 ? &lo : &hi);
#pragma unroll
        for (int j = 0; j < 4; ++j) h2[j] = __floats2bfloat162_rn(f[8 * h + 2 * j], f[8 * h + 2 * j + 1]);
    }
}

// ---------------------------------------------------------------- 128x128 weight quantisation: one block per weight block
// The arithmetic is that of the elementwise definition (scale = max(amax, 1e-4) / 448, correctly rounded divisions); the block
// is read once and held in registers between the two passes, instead of five passes over fp32 copies of the weights. A NaN
// anywhere in the block is its maximum, so that the whole block becomes NaN: weights that have gone wrong stay visible.
__device__ __forceinline__ uint32_t magnitude_bits(const int4& raw) {      // of the largest magnitude; NaN above infinity
    auto mag = [](int w) { return static_cast<uint32_t>(w) & 0x7fff7fffu; };
    const uint32_t m = __vmaxu2(__vmaxu2(mag(raw.x), mag(raw.y)), __vmaxu2(mag(raw.z), mag(raw.w)));
    return max(m >> 16, m & 0xffffu);
}
__global__ void __launch_bounds__(256) weight_quant_kernel(const __nv_bfloat16* __restrict__ w, int rows, int cols, int pow2, uint8_t* __restrict__ q,
                                                           float* __restrict__ scales) {
    launch_dependents();
    dependency_wait();
    __shared__ uint32_t s_max[8];
    const int64_t base = (static_cast<int64_t>(blockIdx.z) * rows + blockIdx.y * 128) * cols + blockIdx.x * 128;
    const int r0 = threadIdx.x >> 3, c = (threadIdx.x & 7) * 16;        // 32 rows per pass, 16 channels per thread
    int4 lo[4], hi[4];
    uint32_t bits = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint8_t* src = reinterpret_cast<const uint8_t*>(w + base + static_cast<int64_t>(r0 + 32 * i) * cols + c);
        lo[i] = ld_nc_int4(src);
        hi[i] = ld_nc_int4(src + 16);
        bits = max(bits, max(magnitude_bits(lo[i]), magnitude_bits(hi[i])));
    }
    bits = __reduce_max_sync(0xffffffffu, bits);
    if (lane_id() == 0) s_max[warp_id()] = bits;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i) bits = max(bits, s_max[i]);
    const float amax = __uint_as_float(bits << 16);
    float scale = __fdiv_rn(amax < 1e-4f ? 1e-4f : amax, 448.f);
    if (pow2) scale = exp2f(ceilf(log2f(scale)));
    if (threadIdx.x == 0) scales[(static_cast<int64_t>(blockIdx.z) * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = scale;
    const float inv = pow2 ? 1.f / scale : 0.f;                         // exact for a power of two
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float f[16];
        unpack16(lo[i], hi[i], f);
#pragma unroll
        for (int j = 0; j < 16; ++j) f[j] = pow2 ? f[j] * inv : __fdiv_rn(f[j], scale);
        int4 o;
        uint32_t* ow = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
        for (int j = 0; j < 4; ++j) ow[j] = pack4_e4m3(f[4 * j], f[4 * j + 1], f[4 * j + 2], f[4 * j + 3]);
        st_na_int4(q + base + static_cast<int64_t>(r0 + 32 * i) * cols + c, o);
    }
}

// ---------------------------------------------------------------- 1x128 quantisation
__global__ void __launch_bounds__(256) quant_kernel(const uint8_t* __restrict__ x, int64_t x_stride_bytes, int rows, int hidden, int wide, int pow2,
                                                    uint8_t* __restrict__ out, float* __restrict__ scales, int64_t sf_row_stride,
                                                    int64_t sf_col_stride) {
    launch_dependents();
    dependency_wait();
    const RowCol rc = row_piece(hidden / kPiece);
    const bool in = rc.row < rows;
    int4 lo, hi;
    load_32(x + rc.row * x_stride_bytes + rc.ch * 2, in ? kPiece * 2 : 0, wide != 0, lo, hi);
    float scale;
    const int4 q = cast16_e4m3(lo, hi, pow2 != 0, scale);       // hidden % 128 == 0: a scale group is all in or all out
    if (in) {
        st_na_int4(out + static_cast<int64_t>(rc.row) * hidden + rc.ch, q);
        if ((lane_id() & 7) == 0) scales[rc.row * sf_row_stride + (rc.ch >> 7) * sf_col_stride] = scale;
    }
}

__global__ void __launch_bounds__(256) dequant_kernel(const uint8_t* __restrict__ q, const float* __restrict__ scales, int64_t sf_row_stride,
                                                      int64_t sf_col_stride, int rows, int hidden, int wide, const RowGroups groups, uint8_t* __restrict__ out) {
    launch_dependents();
    dependency_wait();
    const RowCol rc = row_piece(hidden / kPiece);
    const bool in = rc.row < rows;
    int4 raw = make_int4(0, 0, 0, 0);
    float s = 0.f;
    if (in) {
        raw = ld_nc_int4(q + static_cast<int64_t>(rc.row) * hidden + rc.ch);
        s = scales[rc.row * sf_row_stride + (rc.ch >> 7) * sf_col_stride];
    }
    const bool gap = in_gap_of_lane(groups, rc.row);
    const __nv_fp8x2_storage_t* p2 = reinterpret_cast<const __nv_fp8x2_storage_t*>(&raw);
    float f[16];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const __half2_raw h = __nv_cvt_fp8x2_to_halfraw2(p2[j], __NV_E4M3);
        const float2 t = __half22float2(*reinterpret_cast<const __half2*>(&h));
        f[2 * j] = gap ? 0.f : t.x * s;
        f[2 * j + 1] = gap ? 0.f : t.y * s;
    }
    int4 lo, hi;
    pack16(f, lo, hi);
    store_32(out + (static_cast<int64_t>(rc.row) * hidden + rc.ch) * 2, in ? kPiece * 2 : 0, wide != 0, lo, hi);
}

// ---------------------------------------------------------------- SwiGLU: out = silu(gate) * up (* row weight), optional fused 1x128 cast
// Rows in alignment gaps are left alone (a decode batch over 32 experts has 4096 rows, of which 512 mean something).
template <bool kQuant>
__global__ void __launch_bounds__(256) swiglu_kernel(const uint8_t* __restrict__ x, int rows, int inter, int wide, const float* __restrict__ row_weight,
                                                     const int* __restrict__ num_valid_rows, const RowGroups groups, uint8_t* __restrict__ out,
                                                     float* __restrict__ scales, int64_t sf_row_stride, int64_t sf_col_stride, int pow2) {
    launch_dependents();
    dependency_wait();
    const RowCol rc = row_piece(ceil_div(inter, kPiece));
    const bool gap = in_gap_of_lane(groups, rc.row);
    const bool in = !gap && rc.row < (num_valid_rows != nullptr ? min(*num_valid_rows, rows) : rows);
    if (!__any_sync(0xffffffffu, in)) return;
    const int left = in ? (inter - rc.ch) * 2 : 0;
    const uint8_t* src = x + (static_cast<int64_t>(rc.row) * 2 * inter + rc.ch) * 2;
    int4 glo, ghi, ulo, uhi;
    load_32(src, left, wide != 0, glo, ghi);
    load_32(src + static_cast<int64_t>(inter) * 2, left, wide != 0, ulo, uhi);
    const float wr = row_weight != nullptr && in ? row_weight[rc.row] : 1.f;
    float g[16], u[16];
    unpack16(glo, ghi, g);
    unpack16(ulo, uhi, u);
#pragma unroll
    for (int j = 0; j < 16; ++j) g[j] = g[j] * sigmoid(g[j]) * u[j] * wr;
    int4 lo, hi;
    pack16(g, lo, hi);
    if constexpr (!kQuant) {
        store_32(out + (static_cast<int64_t>(rc.row) * inter + rc.ch) * 2, left, wide != 0, lo, hi);
    } else {
        // the cast sees the bf16 values, so fused and unfused paths agree bit for bit
        float scale;
        const int4 q = cast16_e4m3(lo, hi, pow2 != 0, scale);
        if (left > 0) {
            st_na_int4(out + static_cast<int64_t>(rc.row) * inter + rc.ch, q);
            if ((lane_id() & 7) == 0) scales[rc.row * sf_row_stride + (rc.ch >> 7) * sf_col_stride] = scale;
        }
    }
}

// d(gate|up) from d(out): dgate = dout * up * sig * (1 + gate * (1 - sig)), dup = dout * silu(gate), both times the
// row's gate weight. One block per row, so that the two by-products of the MoE backward pass come out of the same read of
// (gate, up, dout): the weighted activation silu(gate) * up * w (the operand of the W2 weight gradient) and the gradient
// of the gate weight, sum_i dout_i * silu(gate_i) * up_i (a row dot product). Rows in alignment gaps give zeros.
__global__ void __launch_bounds__(256) swiglu_bwd_kernel(const uint8_t* __restrict__ x, const uint8_t* __restrict__ dout, int inter, int wide,
                                                         const float* __restrict__ row_weight, const RowGroups groups, uint8_t* __restrict__ dx,
                                                         uint8_t* __restrict__ act_out, float* __restrict__ dweight) {
    launch_dependents();
    dependency_wait();
    __shared__ float s_part[8];
    const int row = blockIdx.x;
    const bool gap = in_gap(groups, row);
    const float wr = row_weight != nullptr && !gap ? row_weight[row] : 1.f;
    float dot = 0.f;
    for (int ch = threadIdx.x * 16; ch < inter; ch += blockDim.x * 16) {
        const int left = (inter - ch) * 2;
        const uint8_t* src = x + (static_cast<int64_t>(row) * 2 * inter + ch) * 2;
        int4 lo = make_int4(0, 0, 0, 0), hi = lo;
        float g[16], u[16], d[16];
        if (!gap) {
            int4 ulo, uhi, dlo, dhi;
            load_32(src, left, wide != 0, lo, hi);
            load_32(src + static_cast<int64_t>(inter) * 2, left, wide != 0, ulo, uhi);
            load_32(dout + (static_cast<int64_t>(row) * inter + ch) * 2, left, wide != 0, dlo, dhi);
            unpack16(lo, hi, g);
            unpack16(ulo, uhi, u);
            unpack16(dlo, dhi, d);
        } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) g[j] = u[j] = d[j] = 0.f;
        }
        float a[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const float s = sigmoid(g[j]);
            const float silu = g[j] * s;
            // the activation as the forward pass rounded it (bf16), before the weight
            const float act = __bfloat162float(__float2bfloat16_rn(silu * u[j]));
            dot = fmaf(d[j], act, dot);
            a[j] = act * wr;
            const float dw = d[j] * wr;
            g[j] = dw * u[j] * s * (1.f + g[j] * (1.f - s));
            u[j] = dw * silu;
        }
        uint8_t* dst = dx + (static_cast<int64_t>(row) * 2 * inter + ch) * 2;
        pack16(g, lo, hi);
        store_32(dst, left, wide != 0, lo, hi);
        pack16(u, lo, hi);
        store_32(dst + static_cast<int64_t>(inter) * 2, left, wide != 0, lo, hi);
        if (act_out != nullptr) {
            pack16(a, lo, hi);
            store_32(act_out + (static_cast<int64_t>(row) * inter + ch) * 2, left, wide != 0, lo, hi);
        }
    }
    if (dweight != nullptr) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
        if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = dot;
        __syncthreads();
        if (threadIdx.x == 0) {
            float acc = 0.f;
            for (int i = 0; i < (static_cast<int>(blockDim.x) >> 5); ++i) acc += s_part[i];      // fixed order: the result does not depend on timing
            dweight[row] = acc;
        }
    }
}

// ---------------------------------------------------------------- bf16 transpose [rows, cols] -> [cols, rows], 64 x 64 tiles
// Interior tiles of aligned tensors move 16 bytes per thread on both sides: a thread loads eight columns of two
// consecutive rows, pairs them up column by column (one 32-bit word = the same column of both rows) and stores the
// words transposed into shared memory (pitch 33 words); the write side reads four words = eight rows of one column
// and stores them as one 16-byte vector. Edge tiles and unaligned tensors take the element-wise path.
__global__ void __launch_bounds__(256) transpose_kernel(const __nv_bfloat16* __restrict__ in, int64_t in_stride, int64_t in_batch, int rows, int cols,
                                                        __nv_bfloat16* __restrict__ out, int64_t out_stride, int64_t out_batch, int aligned) {
    launch_dependents();
    dependency_wait();
    __shared__ uint32_t tile_t[64 * 33];      // [column][row pair]
    const int r0 = blockIdx.y * 64, c0 = blockIdx.x * 64;
    in += blockIdx.z * in_batch;
    out += blockIdx.z * out_batch;
    if (aligned && r0 + 64 <= rows && c0 + 64 <= cols) {
        const int rp = threadIdx.x >> 3, cv = threadIdx.x & 7;
        const int4 a = ld_nc_int4(reinterpret_cast<const uint8_t*>(in + (r0 + 2 * rp) * in_stride + c0 + cv * 8));
        const int4 b = ld_nc_int4(reinterpret_cast<const uint8_t*>(in + (r0 + 2 * rp + 1) * in_stride + c0 + cv * 8));
        const uint32_t aw[4] = {static_cast<uint32_t>(a.x), static_cast<uint32_t>(a.y), static_cast<uint32_t>(a.z), static_cast<uint32_t>(a.w)};
        const uint32_t bw[4] = {static_cast<uint32_t>(b.x), static_cast<uint32_t>(b.y), static_cast<uint32_t>(b.z), static_cast<uint32_t>(b.w)};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            // columns 2j and 2j + 1 of this thread's eight: low halves of both rows, then high halves
            tile_t[(cv * 8 + 2 * j) * 33 + rp] = __byte_perm(aw[j], bw[j], 0x5410);
            tile_t[(cv * 8 + 2 * j + 1) * 33 + rp] = __byte_perm(aw[j], bw[j], 0x7632);
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int i = threadIdx.x + u * 256;
            const int c = i >> 3, rv = i & 7;
            int4 v;
            v.x = static_cast<int>(tile_t[c * 33 + 4 * rv]);
            v.y = static_cast<int>(tile_t[c * 33 + 4 * rv + 1]);
            v.z = static_cast<int>(tile_t[c * 33 + 4 * rv + 2]);
            v.w = static_cast<int>(tile_t[c * 33 + 4 * rv + 3]);
            st_na_int4(reinterpret_cast<uint8_t*>(out + (c0 + c) * out_stride + r0 + rv * 8), v);
        }
        return;
    }
    __nv_bfloat16* tile = reinterpret_cast<__nv_bfloat16*>(tile_t);     // [64][66]
    for (int i = threadIdx.x; i < 64 * 64; i += 256) {
        const int r = i / 64, c = i % 64;
        tile[r * 66 + c] = (r0 + r < rows && c0 + c < cols) ? in[(r0 + r) * in_stride + c0 + c] : __float2bfloat16(0.f);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 64 * 64; i += 256) {
        const int c = i / 64, r = i % 64;
        if (c0 + c < cols && r0 + r < rows) out[(c0 + c) * out_stride + r0 + r] = tile[r * 66 + c];
    }
}

// blocks of 256 threads for one thread per piece; 0 = too many to be numbered
int piece_blocks(int rows, int width) {
    const int64_t pieces = static_cast<int64_t>(rows) * ceil_div(width, kPiece);
    return pieces < (1ll << 32) - 256 ? static_cast<int>((pieces + 255) / 256) : 0;
}
int is_wide(std::initializer_list<uint64_t> parts) {
    uint64_t bits = 0;
    for (uint64_t v : parts) bits |= v;
    return bits % 32 == 0 ? 1 : 0;
}
uint64_t addr(const void* p) { return reinterpret_cast<uintptr_t>(p); }

}  // namespace

template <typename Logit>
static cudaError_t router_topk_any(const Logit* logits, int64_t row_stride, int num_tokens, int num_experts, int num_topk, int64_t* topk_idx,
                                   float* topk_weights, cudaStream_t stream) {
    if (num_tokens == 0) return cudaSuccess;
    if (num_experts > 2048 || num_topk > 32 || num_topk > num_experts) return cudaErrorInvalidValue;
    const int blocks = (num_tokens * 32 + 255) / 256;
    const int per_lane = (num_experts + 31) / 32;
    if (per_lane <= 2) return launch_early(router_topk_kernel<2, Logit>, dim3(blocks), dim3(256), 0, stream, logits, row_stride, num_tokens, num_experts, num_topk, topk_idx, topk_weights);
    if (per_lane <= 8) return launch_early(router_topk_kernel<8, Logit>, dim3(blocks), dim3(256), 0, stream, logits, row_stride, num_tokens, num_experts, num_topk, topk_idx, topk_weights);
    if (per_lane <= 16) return launch_early(router_topk_kernel<16, Logit>, dim3(blocks), dim3(256), 0, stream, logits, row_stride, num_tokens, num_experts, num_topk, topk_idx, topk_weights);
    return launch_early(router_topk_kernel<64, Logit>, dim3(blocks), dim3(256), 0, stream, logits, row_stride, num_tokens, num_experts, num_topk, topk_idx, topk_weights);
}

cudaError_t router_topk(const void* logits, bool bf16, int64_t row_stride, int num_tokens, int num_experts, int num_topk, int64_t* topk_idx,
                        float* topk_weights, cudaStream_t stream) {
    return bf16 ? router_topk_any(static_cast<const __nv_bfloat16*>(logits), row_stride, num_tokens, num_experts, num_topk, topk_idx, topk_weights, stream)
                : router_topk_any(static_cast<const float*>(logits), row_stride, num_tokens, num_experts, num_topk, topk_idx, topk_weights, stream);
}

cudaError_t router_weights(const float* w, int num_experts, int padded_experts, int hidden, void* out, cudaStream_t stream) {
    if (hidden % 8 != 0) return cudaErrorInvalidValue;
    const int64_t want = (static_cast<int64_t>(padded_experts) * hidden / 8 + 255) / 256;
    return launch_early(router_weights_kernel, dim3(static_cast<int>(std::min<int64_t>(std::max<int64_t>(want, 1), 148 * 16))), dim3(256), 0, stream, w, num_experts, padded_experts, hidden, static_cast<__nv_bfloat16*>(out));
}

cudaError_t router_backward(const int64_t* topk_idx, const float* w, const float* dw, int num_tokens, int num_topk, int num_experts, int padded_experts,
                            int hidden, const void* router, void* dx, void* dlogits, cudaStream_t stream) {
    if (num_tokens == 0) return cudaSuccess;
    const int columns = (hidden + kSpan - 1) / kSpan;
    const int64_t warps = static_cast<int64_t>(num_tokens) * columns;
    if (num_topk > 32 || padded_experts % 8 != 0 || hidden % 8 != 0 || warps >= (1ll << 31)) return cudaErrorInvalidValue;
    return launch_early(router_backward_kernel, dim3(static_cast<int>((warps + 7) / 8)), dim3(256), 0, stream, topk_idx, w, dw, num_tokens, num_topk, num_experts, padded_experts, hidden, columns, static_cast<const __nv_bfloat16*>(router),
        static_cast<__nv_bfloat16*>(dx), static_cast<__nv_bfloat16*>(dlogits));
}

cudaError_t quant_weights_128x128(const void* w, int groups, int rows, int cols, bool pow2, void* q, float* scales, cudaStream_t stream) {
    if (groups == 0 || rows == 0 || cols == 0) return cudaSuccess;
    if (rows % 128 != 0 || cols % 128 != 0 || groups > 65535 || rows / 128 > 65535) return cudaErrorInvalidValue;
    return launch_early(weight_quant_kernel, dim3(cols / 128, rows / 128, groups), dim3(256), 0, stream, static_cast<const __nv_bfloat16*>(w), rows, cols, pow2 ? 1 : 0,
                                                                                  static_cast<uint8_t*>(q), scales);
}

cudaError_t quant_1x128(const void* x, int64_t x_stride_bytes, int rows, int hidden, bool pow2, void* out, float* scales,
                        int64_t sf_row_stride, int64_t sf_col_stride, cudaStream_t stream) {
    if (rows == 0) return cudaSuccess;
    const int blocks = piece_blocks(rows, hidden);
    if (hidden % 128 != 0 || blocks == 0) return cudaErrorInvalidValue;
    return launch_early(quant_kernel, dim3(blocks), dim3(256), 0, stream, static_cast<const uint8_t*>(x), x_stride_bytes, rows, hidden,
                                             is_wide({addr(x), static_cast<uint64_t>(x_stride_bytes)}), pow2, static_cast<uint8_t*>(out), scales,
                                             sf_row_stride, sf_col_stride);
}

cudaError_t dequant_1x128(const void* q, const float* scales, int64_t sf_row_stride, int64_t sf_col_stride, int rows, int hidden,
                          const RowGroups& groups, void* out, cudaStream_t stream) {
    if (rows == 0) return cudaSuccess;
    const int blocks = piece_blocks(rows, hidden);
    if (hidden % 128 != 0 || blocks == 0) return cudaErrorInvalidValue;
    return launch_early(dequant_kernel, dim3(blocks), dim3(256), 0, stream, static_cast<const uint8_t*>(q), scales, sf_row_stride, sf_col_stride, rows, hidden,
                                               is_wide({addr(out)}), groups, static_cast<uint8_t*>(out));
}

cudaError_t swiglu(const void* x, int rows, int inter, const float* row_weight, const int* num_valid_rows, const RowGroups& groups, void* out, bool quant,
                   float* scales, int64_t sf_row_stride, int64_t sf_col_stride, bool pow2, cudaStream_t stream) {
    if (rows == 0) return cudaSuccess;
    const int blocks = piece_blocks(rows, inter);
    if (inter % 8 != 0 || (quant && inter % 128 != 0) || blocks == 0) return cudaErrorInvalidValue;
    const int wide = is_wide({addr(x), addr(out), static_cast<uint64_t>(inter) * 2});
    if (quant)
        return launch_early(swiglu_kernel<true>, dim3(blocks), dim3(256), 0, stream, static_cast<const uint8_t*>(x), rows, inter, wide, row_weight, num_valid_rows, groups,
                                                        static_cast<uint8_t*>(out), scales, sf_row_stride, sf_col_stride, pow2 ? 1 : 0);
    else
        return launch_early(swiglu_kernel<false>, dim3(blocks), dim3(256), 0, stream, static_cast<const uint8_t*>(x), rows, inter, wide, row_weight, num_valid_rows, groups,
                                                         static_cast<uint8_t*>(out), nullptr, 0, 0, 0);
}

cudaError_t swiglu_backward(const void* x, const void* dout, int rows, int inter, const float* row_weight, const RowGroups& groups, void* dx, void* act_out,
                            float* dweight, cudaStream_t stream) {
    if (rows == 0) return cudaSuccess;
    if (inter % 8 != 0) return cudaErrorInvalidValue;
    // (more than 128 threads lengthen the blocks' ends; where the rows alone do not fill the GPU they shorten the rows: 8 x 16384
    // 11.4 us with 128)
    const int threads = std::min(rows < 296 ? 256 : 128, align_up(ceil_div(inter, 16), 32));
    const int wide = is_wide({addr(x), addr(dout), addr(dx), addr(act_out), static_cast<uint64_t>(inter) * 2});
    return launch_early(swiglu_bwd_kernel, dim3(rows), dim3(threads), 0, stream, static_cast<const uint8_t*>(x), static_cast<const uint8_t*>(dout), inter, wide, row_weight, groups,
                                                    static_cast<uint8_t*>(dx), static_cast<uint8_t*>(act_out), dweight);
}

cudaError_t transpose_bf16(const void* in, int64_t in_stride, int64_t in_batch, int batch, int rows, int cols, void* out, int64_t out_stride,
                           int64_t out_batch, cudaStream_t stream) {
    if (rows == 0 || cols == 0 || batch == 0) return cudaSuccess;
    dim3 grid((cols + 63) / 64, (rows + 63) / 64, batch);
    const int aligned = in_stride % 8 == 0 && out_stride % 8 == 0 && in_batch % 8 == 0 && out_batch % 8 == 0 && addr(in) % 16 == 0 && addr(out) % 16 == 0;
    return launch_early(transpose_kernel, grid, dim3(256), 0, stream, static_cast<const __nv_bfloat16*>(in), in_stride, in_batch, rows, cols, static_cast<__nv_bfloat16*>(out),
                                               out_stride, out_batch, aligned);
}

}  // namespace ops
}  // namespace ep
