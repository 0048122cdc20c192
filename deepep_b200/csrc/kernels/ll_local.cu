// Low-latency dispatch and combine of a group of ONE rank (sm_100a): a decode batch goes straight from the caller's rows
// into the packed expert-major layout and back, without messages, arrival flags, fences or call counters that gate
// anything -- the multi-rank kernels (ll.cu) spend their time on exactly that chain (17 us for a kernel that moves four
// tokens, 26 + 22 us for 128 tokens of hidden 7168, against about 4 us that the bytes of 128 tokens take).
// Row order, src_info, layout_range, scales and the fp32 summation order are those of the multi-rank kernels.
#include "api.hpp"
#include "../common/device_utils.cuh"

namespace ep {

namespace {

constexpr int kLLLocalThreads = 512, kLLLocalWarps = kLLLocalThreads / 32;

__device__ __forceinline__ int* ll_mask_words(uint64_t* local_ws) {
    return reinterpret_cast<int*>(reinterpret_cast<uint8_t*>(local_ws) + kWsLLOffsetBytes) + 2 * kMaxExperts;
}

// One block per token (grid-stride): warp k looks up the position of the token's k-th pair among the earlier tokens of its
// expert, then every warp streams 1 KB slices of the row, cast on the way, to the K packed rows. The per-expert counts are
// a histogram that every block builds for itself (at most 2048 entries, one or two shared-memory adds per thread), which
// is cheaper than any hand-over between blocks; a block writes the counts of its share of the experts.
__global__ void __launch_bounds__(kLLLocalThreads) ll_local_dispatch_kernel(const __grid_constant__ LLDispatchParams p) {
    extern __shared__ int s_ll[];
    const int T = p.num_tokens, H = p.hidden, K = p.num_topk, E = p.num_experts, Tm = p.num_max_tokens;
    int* s_idx = s_ll;                  // [T * K]
    int* s_hist = s_idx + T * K;        // [E]
    __shared__ int s_slot[kMaxLLTopk], s_exp[kMaxLLTopk];
    const int tid = threadIdx.x, lane = lane_id(), warp = warp_id();
    const int bid = blockIdx.x, nb = gridDim.x;
    dependency_wait();
    launch_dependents();
    const int row_bytes = H * 2, slices = ceil_div(row_bytes, 1024);
    // The chain of dependent loads is what these few microseconds are made of: the mask word, the routing and the first
    // slices of the block's first row are requested together.
    const int mask_word = *reinterpret_cast<volatile int*>(ll_mask_words(p.c.local_ws));
    int4 lo = make_int4(0, 0, 0, 0), hi = lo;
    auto load = [&](int t, int s) {
        const int off = s * 1024 + lane * 32;
        lo = hi = make_int4(0, 0, 0, 0);
        if (t < T && off < row_bytes) {                             // rows are multiples of 256 bytes: 32 bytes are in or out
            const uint8_t* src = p.x + static_cast<int64_t>(t) * row_bytes + off;
            lo = *reinterpret_cast<const int4*>(src);
            hi = *reinterpret_cast<const int4*>(src + 16);
        }
    };
    load(bid, warp);
    for (int e = tid; e < E; e += kLLLocalThreads) s_hist[e] = 0;
    for (int i = tid; i < T * K; i += kLLLocalThreads) {
        const int e = load_topk_idx(p.topk_idx, p.idx32 != 0, i, E);
        s_idx[i] = mask_word != 0 ? -1 : e;                         // this rank has masked itself
    }
    __syncthreads();
    for (int i = tid; i < T * K; i += kLLLocalThreads)
        if (s_idx[i] >= 0) atomicAdd(s_hist + s_idx[i], 1);
    const int sf_per_row = p.use_fp8 ? (p.use_ue8m0 ? H / 512 : H / 128) : 0;
    const int64_t out_row_bytes = p.use_fp8 ? H : row_bytes;
    for (int t = bid; t < T; t += nb) {
        if (t != bid) load(t, warp);        // (the first slice of every warp: before the positions are known)
        if (warp < K) {
            const int e = s_idx[t * K + warp];
            int before = 0;
            if (e >= 0) {
#pragma unroll 8
                for (int i = lane; i < t * K; i += 32) before += s_idx[i] == e;
            }
            before = warp_reduce_sum(before);
            if (lane == 0) {
                s_exp[warp] = e;
                s_slot[warp] = before;
                if (e >= 0) p.packed_recv_src_info[static_cast<int64_t>(e) * Tm + before] = t | (warp << 16);
            }
        }
        __syncthreads();
        for (int s = warp; s < slices; s += kLLLocalWarps) {
            if (s != warp) load(t, s);
            const int off = s * 1024 + lane * 32;
            if (!p.use_fp8) {
                if (off < row_bytes)
                    for (int k = 0; k < K; ++k)
                        if (s_exp[k] >= 0) {
                            uint8_t* dst = p.packed_recv_x + (static_cast<int64_t>(s_exp[k]) * Tm + s_slot[k]) * out_row_bytes + off;
                            st_na_int4(dst, lo);
                            st_na_int4(dst + 16, hi);
                        }
                continue;
            }
            // 16 channels per lane, eight lanes per scale group
            float scale;
            const int4 q = cast16_e4m3(lo, hi, p.round_scale != 0, scale);
            if (off < row_bytes) {
                const int g = off >> 8;
                for (int k = 0; k < K; ++k) {
                    if (s_exp[k] < 0) continue;
                    const int64_t row = static_cast<int64_t>(s_exp[k]) * Tm + s_slot[k];
                    st_na_int4(p.packed_recv_x + row * out_row_bytes + off / 2, q);
                    if ((lane & 7) == 0) {
                        // column-major scales: [expert][group][row]
                        if (p.use_ue8m0)
                            p.packed_recv_sf[((static_cast<int64_t>(s_exp[k]) * sf_per_row + (g >> 2)) * Tm + s_slot[k]) * 4 + (g & 3)] =
                                static_cast<uint8_t>(__float_as_uint(scale) >> 23);
                        else
                            reinterpret_cast<float*>(p.packed_recv_sf)[(static_cast<int64_t>(s_exp[k]) * sf_per_row + g) * Tm + s_slot[k]] = scale;
                    }
                }
            }
        }
        __syncthreads();        // the positions of this token have been used
    }
    if (bid >= T) __syncthreads();      // (blocks without a token: the histogram is complete)
    for (int e = bid + tid * nb; e < E; e += nb * kLLLocalThreads) {
        const int n = s_hist[e];
        p.packed_recv_count[e] = n;
        p.packed_recv_layout_range[e] = n;
        if (p.cumulative_stats != nullptr && n != 0) atomicAdd(p.cumulative_stats + e, n);
    }
    if (bid == 0 && tid < 2) p.c.local_ws[kWsLLCalls + tid] += 1;      // a later multi-rank style call (LogFMT) continues from here
}

constexpr int kLLCombineThreads = 128, kLLCombineCols = kLLCombineThreads * 8;

// Block = (token, 1024 channels). The warps first find the packed row of every top-k lane of the token (src_info names
// token and lane of each row; an expert holds at most T rows, one or two passes of a warp), then every thread sums eight
// channels over up to eight rows in flight, in ascending lane order.
__global__ void __launch_bounds__(kLLCombineThreads) ll_local_combine_kernel(const __grid_constant__ LLCombineParams p) {
    const int H = p.hidden, K = p.num_topk, E = p.num_experts, Tm = p.num_max_tokens, T = p.num_tokens;
    __shared__ int s_row[kMaxLLTopk];
    __shared__ float s_w[kMaxLLTopk];
    const int tid = threadIdx.x, lane = lane_id(), warp = warp_id();
    dependency_wait();
    launch_dependents();
    const int mask_word = *reinterpret_cast<volatile int*>(ll_mask_words(p.c.local_ws));
    const int parts = ceil_div(H, kLLCombineCols);
    for (int item = blockIdx.x; item < T * parts; item += gridDim.x) {
        const int t = item / parts, ch = (item % parts) * kLLCombineCols + tid * 8;
        for (int k = warp; k < K; k += kLLCombineThreads / 32) {
            const int e = load_topk_idx(p.topk_idx, p.idx32 != 0, static_cast<int64_t>(t) * K + k, E);
            const float weight = p.topk_weights[static_cast<int64_t>(t) * K + k];
            int row = -1;
            if (e >= 0 && mask_word == 0) {
                // the first rows are looked at before it is known how many there are (one step less in the chain of loads)
                const int* info = p.src_info + static_cast<int64_t>(e) * Tm;
                const int first = lane < Tm ? info[lane] : -1;
                const int n = min(static_cast<int>(p.layout_range[e] & 0xffffffff), Tm);
                const int want = t | (k << 16);
                if (lane < n && first == want) row = lane;
                for (int j = lane + 32; j < n; j += 32)
                    if (info[j] == want) row = j;
            }
            row = __reduce_max_sync(0xffffffffu, row);
            if (lane == 0) {
                s_row[k] = row < 0 ? -1 : e * Tm + row;
                s_w[k] = weight;
            }
        }
        __syncthreads();
        if (ch < H) {
            float acc[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[i] = 0.f;
            for (int k0 = 0; k0 < K; k0 += 8) {
                int4 raw[8];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (k0 + u < K && s_row[k0 + u] >= 0) raw[u] = ld_nc_int4(p.x + (static_cast<int64_t>(s_row[k0 + u]) * H + ch) * 2);
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (k0 + u < K && s_row[k0 + u] >= 0) {
                        const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&raw[u]);
                        const float wk = s_w[k0 + u];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float2 v = __bfloat1622float2(h2[i]);
                            acc[2 * i] = fmaf(wk, v.x, acc[2 * i]);
                            acc[2 * i + 1] = fmaf(wk, v.y, acc[2 * i + 1]);
                        }
                    }
            }
            int4 out;
            __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&out);
#pragma unroll
            for (int i = 0; i < 4; ++i) o2[i] = __floats2bfloat162_rn(acc[2 * i], acc[2 * i + 1]);
            st_na_int4(p.combined_x + (static_cast<int64_t>(t) * H + ch) * 2, out);
        }
        __syncthreads();
    }
    if (blockIdx.x == 0 && tid < 2) p.c.local_ws[kWsLLCalls + 2 + tid] += 1;
}

template <typename Params>
cudaError_t launch_dependent(void (*fn)(const Params), const Params& p, int grid, int block, int smem, cudaStream_t stream, bool programmatic) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = programmatic ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, fn, p);
}

}  // namespace

cudaError_t launch_ll_local_dispatch(const LLDispatchParams& p, int num_sms, bool programmatic, cudaStream_t stream) {
    static PreparedKernel prepared;
    const int smem_bytes = (p.num_tokens * p.num_topk + p.num_experts) * 4;
    cudaError_t err = prepared.prepare(ll_local_dispatch_kernel, smem_bytes);
    if (err != cudaSuccess) return err;
    // a block per token; a few more where there are few tokens, for the counts of the experts
    const int want = p.num_tokens > 16 ? p.num_tokens : 16;
    return launch_dependent(ll_local_dispatch_kernel, p, want < num_sms ? want : num_sms, kLLLocalThreads, smem_bytes, stream, programmatic);
}

cudaError_t launch_ll_local_combine(const LLCombineParams& p, int num_sms, bool limited, bool programmatic, cudaStream_t stream) {
    static PreparedKernel prepared;
    cudaError_t err = prepared.prepare(ll_local_combine_kernel, 0);
    if (err != cudaSuccess) return err;
    const int items = p.num_tokens * ceil_div(p.hidden, kLLCombineCols), most = limited ? num_sms : num_sms * 8;
    const int grid = items < 1 ? 1 : (items < most ? items : most);
    return launch_dependent(ll_local_combine_kernel, p, grid, kLLCombineThreads, 0, stream, programmatic);
}

}  // namespace ep
