// Mixture-of-experts routing and pointwise glue: top-k router, deterministic route plan,
// SwiGLU split, weighted reduce.
#include <cuda_bf16.h>

#include <algorithm>
#include <cfloat>
#include <climits>

#include "cuda_util.h"

namespace mfqb {

// Launch as a programmatic dependent: the kernel becomes resident while its predecessor drains and waits for it
// (griddepcontrol.wait) before it touches memory.
template <typename... KArgs, typename... Args>
static void launch_after(void (*kernel)(KArgs...), dim3 grid, dim3 block, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    MFQB_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...));
}
__device__ __forceinline__ void after_predecessor() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// ---- top-k router: one warp per token ---------------------------------------------------
// Selection is exact: score comparisons only, ties to the smaller expert id, NaN -> -FLT_MAX
// (mfq/kernels/cuda/moe.cu:124-263).
__device__ __forceinline__ bool score_before(float sa, int ea, float sb, int eb) { return sa > sb || (sa == sb && ea < eb); }

__global__ void __launch_bounds__(128) moe_topk_kernel(const float* __restrict__ logits, const float* __restrict__ bias,
                                                        int32_t* __restrict__ ids, float* __restrict__ weights, int tokens,
                                                        int experts, int k, int mode, int normalize, float norm_floor,
                                                        float scale) {
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= tokens) return;
    const float* z = logits + (size_t)row * experts;
    auto clean = [](float v) { return isnan(v) ? -FLT_MAX : v; };
    float smax = 0.f, ssum = 1.f;
    if (mode == MFQB_ROUTER_SOFTMAX) {
        smax = -INFINITY;
        for (int e = lane; e < experts; e += 32) smax = fmaxf(smax, clean(z[e]));
        for (int o = 16; o; o >>= 1) smax = fmaxf(smax, __shfl_xor_sync(0xffffffffu, smax, o));
        ssum = 0.f;
        for (int e = lane; e < experts; e += 32) ssum += expf(clean(z[e]) - smax);
        for (int o = 16; o; o >>= 1) ssum += __shfl_xor_sync(0xffffffffu, ssum, o);
    }
    auto weight_of = [&](float raw) {
        if (mode == MFQB_ROUTER_DELAYED_SOFTMAX) return raw;
        if (mode == MFQB_ROUTER_SIGMOID) return 1.0f / (1.0f + expf(-raw));
        if (mode == MFQB_ROUTER_SQRT_SOFTPLUS) return sqrtf(raw > 20.0f ? raw : log1pf(expf(raw)));
        return expf(raw - smax) / ssum;
    };
    int chosen[16];
    float my_weight = 0.f;   // lane r keeps the weight of rank r
    for (int r = 0; r < k; ++r) {
        float bs = -INFINITY, bw = -INFINITY;
        int be = INT_MAX;
        for (int e = lane; e < experts; e += 32) {
            bool taken = false;
            for (int p = 0; p < r; ++p) taken |= chosen[p] == e;
            if (taken) continue;
            const float wgt = weight_of(clean(z[e]));
            const float sc = wgt + (bias ? bias[e] : 0.0f);
            if (score_before(sc, e, bs, be)) { bs = sc; bw = wgt; be = e; }
        }
        for (int o = 16; o; o >>= 1) {
            const float os = __shfl_xor_sync(0xffffffffu, bs, o), ow = __shfl_xor_sync(0xffffffffu, bw, o);
            const int oe = __shfl_xor_sync(0xffffffffu, be, o);
            if (score_before(os, oe, bs, be)) { bs = os; bw = ow; be = oe; }
        }
        chosen[r] = be;
        if (lane == r) my_weight = bw;
        if (lane == 0) ids[(size_t)row * k + r] = be;
    }
    float v = lane < k ? my_weight : 0.f;
    if (mode == MFQB_ROUTER_DELAYED_SOFTMAX) {
        float m = lane < k ? v : -INFINITY;
        for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        v = lane < k ? expf(v - m) : 0.f;
        float d = v;
        for (int o = 16; o; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        v /= d;
    } else if (normalize) {
        float d = v;
        for (int o = 16; o; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        v /= fmaxf(d, norm_floor);
    }
    if (lane < k) weights[(size_t)row * k + lane] = v * scale;
}

// The same selection for up to 32 * EPL experts: a lane keeps its experts' weights and scores in
// registers (computed once), and a bit per expert marks the ones already chosen.  Same operations in
// the same order as moe_topk_kernel, so both give identical ids and weights.
template <int EPL>
__global__ void __launch_bounds__(128) moe_topk_regs_kernel(const float* __restrict__ logits, const float* __restrict__ bias,
                                                             int32_t* __restrict__ ids, float* __restrict__ weights, int tokens,
                                                             int experts, int k, int mode, int normalize, float norm_floor,
                                                             float scale) {
    after_predecessor();
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= tokens) return;
    const float* z = logits + (size_t)row * experts;
    float raw[EPL], bs_add[EPL];
    unsigned taken = 0u;   // bit j: expert lane + 32 j is out of range or already chosen
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
        const int e = lane + 32 * j;
        const bool ok = e < experts;
        const float v = ok ? z[e] : 0.f;
        raw[j] = isnan(v) ? -FLT_MAX : v;
        bs_add[j] = (ok && bias) ? bias[e] : 0.f;
        if (!ok) taken |= 1u << j;
    }
    float smax = 0.f, ssum = 1.f;
    if (mode == MFQB_ROUTER_SOFTMAX) {
        smax = -INFINITY;
#pragma unroll
        for (int j = 0; j < EPL; ++j)
            if (!((taken >> j) & 1u)) smax = fmaxf(smax, raw[j]);
        for (int o = 16; o; o >>= 1) smax = fmaxf(smax, __shfl_xor_sync(0xffffffffu, smax, o));
        ssum = 0.f;
#pragma unroll
        for (int j = 0; j < EPL; ++j)
            if (!((taken >> j) & 1u)) ssum += expf(raw[j] - smax);
        for (int o = 16; o; o >>= 1) ssum += __shfl_xor_sync(0xffffffffu, ssum, o);
    }
    float wg[EPL], sc[EPL];
#pragma unroll
    for (int j = 0; j < EPL; ++j) {
        float wv;
        if (mode == MFQB_ROUTER_DELAYED_SOFTMAX) wv = raw[j];
        else if (mode == MFQB_ROUTER_SIGMOID) wv = 1.0f / (1.0f + expf(-raw[j]));
        else if (mode == MFQB_ROUTER_SQRT_SOFTPLUS) wv = sqrtf(raw[j] > 20.0f ? raw[j] : log1pf(expf(raw[j])));
        else wv = expf(raw[j] - smax) / ssum;
        wg[j] = wv;
        sc[j] = wv + bs_add[j];
    }
    float my_weight = 0.f;   // lane r keeps the weight of rank r
    for (int r = 0; r < k; ++r) {
        float bs = -INFINITY, bw = -INFINITY;
        int be = INT_MAX;
#pragma unroll
        for (int j = 0; j < EPL; ++j)
            if (!((taken >> j) & 1u) && score_before(sc[j], lane + 32 * j, bs, be)) { bs = sc[j]; bw = wg[j]; be = lane + 32 * j; }
        for (int o = 16; o; o >>= 1) {
            const float os = __shfl_xor_sync(0xffffffffu, bs, o), ow = __shfl_xor_sync(0xffffffffu, bw, o);
            const int oe = __shfl_xor_sync(0xffffffffu, be, o);
            if (score_before(os, oe, bs, be)) { bs = os; bw = ow; be = oe; }
        }
        if (lane == (be & 31)) taken |= 1u << (be >> 5);
        if (lane == r) my_weight = bw;
        if (lane == 0) ids[(size_t)row * k + r] = be;
    }
    float v = lane < k ? my_weight : 0.f;
    if (mode == MFQB_ROUTER_DELAYED_SOFTMAX) {
        float m = lane < k ? v : -INFINITY;
        for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        v = lane < k ? expf(v - m) : 0.f;
        float d = v;
        for (int o = 16; o; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        v /= d;
    } else if (normalize) {
        float d = v;
        for (int o = 16; o; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        v /= fmaxf(d, norm_floor);
    }
    if (lane < k) weights[(size_t)row * k + lane] = v * scale;
}

// ---- route plan ------------------------------------------------------------------------------
// counts -> exclusive scan -> stable placement (one warp per expert walks the pairs in order),
// so every expert's segment lists its pairs in ascending order: the plan is deterministic.
__global__ void route_count_kernel(const int32_t* __restrict__ ids, int pairs, int experts, int32_t* __restrict__ counts) {
    const int e = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (e >= experts) return;
    int n = 0;
    for (int p = lane; p < pairs; p += 32) n += ids[p] == e;
    for (int o = 16; o; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    if (lane == 0) counts[e] = n;
}

__global__ void route_scan_kernel(int experts, int tile_m, int32_t* __restrict__ expert_bounds, int32_t* __restrict__ tile_bounds) {
    // expert_bounds[1..E] holds the counts on entry; one thread scans (E <= 4096, a few microseconds
    // at most, off the critical path of the expert matmuls of small batches which do not use the plan)
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        int run = 0, tiles = 0;
        expert_bounds[0] = 0;
        tile_bounds[0] = 0;
        for (int e = 0; e < experts; ++e) {
            const int c = expert_bounds[e + 1];
            run += c;
            tiles += (c + tile_m - 1) / tile_m;
            expert_bounds[e + 1] = run;
            tile_bounds[e + 1] = tiles;
        }
    }
}

__global__ void route_place_kernel(const int32_t* __restrict__ ids, int pairs, int experts,
                                   const int32_t* __restrict__ expert_bounds, int32_t* __restrict__ pair_order) {
    const int e = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (e >= experts) return;
    int at = expert_bounds[e];
    for (int base = 0; base < pairs; base += 32) {
        const int p = base + lane;
        const bool hit = p < pairs && ids[p] == e;
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (hit) pair_order[at + __popc(m & ((1u << lane) - 1u))] = p;
        at += __popc(m);
    }
}

// The same plan in one launch of one CTA, for up to 1024 experts and 65535 pairs.  Every warp owns a contiguous stretch of the
// pairs and counts it by expert (lanes with the same id find each other with match_any); the counts are scanned over warps and
// experts, and in a second pass over its stretch the warp places its pairs, in ascending order.  Nothing is serial over experts
// or walks all pairs per expert, as a first form with one scanning thread did (8 us for 2048 pairs and 128 experts; now 3).
constexpr int kRoutePlanExperts = 1024, kRoutePlanPairs = 65535, kRoutePlanWarps = 16;
__global__ void __launch_bounds__(32 * kRoutePlanWarps) route_plan_kernel(const int32_t* __restrict__ ids, int pairs, int experts, int tile_m,
                                                                          int32_t* __restrict__ expert_bounds, int32_t* __restrict__ tile_bounds,
                                                                          int32_t* __restrict__ pair_order) {
    __shared__ unsigned short hist[kRoutePlanWarps][kRoutePlanExperts];   // pairs of an expert in a warp's stretch, then those before it
    __shared__ int first[kRoutePlanExperts];
    __shared__ int2 warp_sum[kRoutePlanWarps];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    for (int e = lane; e < experts; e += 32) hist[warp][e] = 0;
    __syncwarp();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int per = ((pairs + kRoutePlanWarps - 1) / kRoutePlanWarps + 31) / 32 * 32, p0 = min(pairs, warp * per), p1 = min(pairs, p0 + per);
    auto id_at = [&](int p) {
        const int e = p < p1 ? __ldcg(ids + p) : -1;
        return e >= 0 && e < experts ? e : -1;   // an id out of range takes no place in the plan
    };
    for (int base = p0; base < p1; base += 32) {
        const int e = id_at(base + lane);
        const unsigned same = __match_any_sync(0xffffffffu, e);
        if (e >= 0 && lane == __ffs(same) - 1) hist[warp][e] += (unsigned short)__popc(same);
        __syncwarp();
    }
    __syncthreads();
    // thread t: experts 2t, 2t + 1
    int cnt[2] = {0, 0};
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int e = 2 * tid + j;
        if (e < experts)
            for (int w = 0; w < kRoutePlanWarps; ++w) {
                const int c = hist[w][e];
                hist[w][e] = (unsigned short)cnt[j];
                cnt[j] += c;
            }
    }
    const int t0 = (cnt[0] + tile_m - 1) / tile_m, t1 = (cnt[1] + tile_m - 1) / tile_m;
    int2 run = make_int2(cnt[0] + cnt[1], t0 + t1);   // inclusive over threads
    for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, run.x, o), b = __shfl_up_sync(0xffffffffu, run.y, o);
        if (lane >= o) { run.x += a; run.y += b; }
    }
    if (lane == 31) warp_sum[warp] = run;
    __syncthreads();
    for (int w = 0; w < warp; ++w) { run.x += warp_sum[w].x; run.y += warp_sum[w].y; }
    const int b0 = run.x - cnt[0] - cnt[1], q0 = run.y - t0 - t1;
    if (2 * tid < experts) { first[2 * tid] = b0; expert_bounds[2 * tid] = b0; tile_bounds[2 * tid] = q0; }
    if (2 * tid + 1 < experts) { first[2 * tid + 1] = b0 + cnt[0]; expert_bounds[2 * tid + 1] = b0 + cnt[0]; tile_bounds[2 * tid + 1] = q0 + t0; }
    if (tid == (experts - 1) / 2) { expert_bounds[experts] = run.x; tile_bounds[experts] = run.y; }
    __syncthreads();
    for (int base = p0; base < p1; base += 32) {
        const int e = id_at(base + lane);
        const unsigned same = __match_any_sync(0xffffffffu, e);
        if (e >= 0) pair_order[first[e] + hist[warp][e] + __popc(same & ((1u << lane) - 1u))] = base + lane;
        __syncwarp();
        if (e >= 0 && lane == __ffs(same) - 1) hist[warp][e] += (unsigned short)__popc(same);
        __syncwarp();
    }
}

// ---- pointwise glue -----------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ float to_f32(T v);
template <>
__device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T, typename O>
__global__ void swiglu_kernel(const T* __restrict__ gate_up, int rows, int f, O* __restrict__ hidden) {
    const size_t total = (size_t)rows * f;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const size_t r = i / f, j = i % f;
        const float g = to_f32(gate_up[r * 2 * f + j]), u = to_f32(gate_up[r * 2 * f + f + j]);
        const float v = u * g / (1.0f + expf(-g));
        if constexpr (sizeof(O) == 4) hidden[i] = v;
        else hidden[i] = __float2bfloat16_rn(v);
    }
}

template <typename T, typename O>
__global__ void weighted_reduce_kernel(const T* __restrict__ src, const float* __restrict__ weights, int tokens, int routes, int h,
                                       O* __restrict__ y) {
    after_predecessor();
    const size_t total = (size_t)tokens * h;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const size_t t = i / h, j = i % h;
        float acc = 0.f;
        for (int r = 0; r < routes; ++r) acc += weights[t * routes + r] * to_f32(src[(t * routes + r) * h + j]);
        if constexpr (sizeof(O) == 4) y[i] = acc;
        else y[i] = __float2bfloat16_rn(acc);
    }
}
// The same for float32 rows of whole quads: four columns a thread, four routes in flight.  Grid (column blocks, tokens).
template <typename O>
__global__ void __launch_bounds__(256) weighted_reduce4_kernel(const float* __restrict__ src, const float* __restrict__ weights, int routes, int h, O* __restrict__ y) {
    after_predecessor();
    const int j = blockIdx.x * 256 + threadIdx.x;
    const size_t t = blockIdx.y;
    if (4 * j >= h) return;
    const float* w = weights + t * routes;
    const float4* row = reinterpret_cast<const float4*>(src + t * routes * h) + j;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int r0 = 0; r0 < routes; r0 += 4) {
        float4 v[4];
        float wr[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const bool in = r0 + u < routes;
            v[u] = in ? __ldcg(row + (size_t)(r0 + u) * (h >> 2)) : make_float4(0.f, 0.f, 0.f, 0.f);
            wr[u] = in ? __ldcg(w + r0 + u) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (r0 + u < routes) { acc.x += wr[u] * v[u].x; acc.y += wr[u] * v[u].y; acc.z += wr[u] * v[u].z; acc.w += wr[u] * v[u].w; }
    }
    if constexpr (sizeof(O) == 4) {
        reinterpret_cast<float4*>(y + t * h)[j] = acc;
    } else {
        const __nv_bfloat162 a = __floats2bfloat162_rn(acc.x, acc.y), b = __floats2bfloat162_rn(acc.z, acc.w);
        reinterpret_cast<uint2*>(y + t * h)[j] = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
    }
}

void launch_swiglu(const void* gate_up, int in_dtype, int rows, int f, void* hidden, cudaStream_t s) {
    const size_t total = (size_t)rows * f;
    if (total == 0) return;
    const int block = 256, grid = (int)std::min<size_t>((total + block - 1) / block, 148 * 8);
    if (in_dtype == MFQB_F32) swiglu_kernel<float, __nv_bfloat16><<<grid, block, 0, s>>>(static_cast<const float*>(gate_up), rows, f, static_cast<__nv_bfloat16*>(hidden));
    else swiglu_kernel<__nv_bfloat16, __nv_bfloat16><<<grid, block, 0, s>>>(static_cast<const __nv_bfloat16*>(gate_up), rows, f, static_cast<__nv_bfloat16*>(hidden));
    MFQB_CUDA(cudaGetLastError());
}

// float32 gate|up -> float32 activation (the library's own intermediate: no rounding between the two expert matmuls)
void launch_swiglu_f32(const float* gate_up, int rows, int f, float* hidden, cudaStream_t s) {
    const size_t total = (size_t)rows * f;
    if (total == 0) return;
    const int block = 256, grid = (int)std::min<size_t>((total + block - 1) / block, 148 * 8);
    swiglu_kernel<float, float><<<grid, block, 0, s>>>(gate_up, rows, f, hidden);
    MFQB_CUDA(cudaGetLastError());
}

void launch_weighted_reduce(const void* src, int in_dtype, const float* weights, int tokens, int routes, int h, void* y, int y_dtype,
                            cudaStream_t s) {
    const size_t total = (size_t)tokens * h;
    if (total == 0) return;
    const bool quads = in_dtype == MFQB_F32 && h % 4 == 0 && tokens <= 65535 && ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(y)) & 15) == 0;
    if (quads) {
        const dim3 grid((unsigned)((h / 4 + 255) / 256), (unsigned)tokens), block(256);
        if (y_dtype == MFQB_F32) launch_after(weighted_reduce4_kernel<float>, grid, block, s, static_cast<const float*>(src), weights, routes, h, static_cast<float*>(y));
        else launch_after(weighted_reduce4_kernel<__nv_bfloat16>, grid, block, s, static_cast<const float*>(src), weights, routes, h, static_cast<__nv_bfloat16*>(y));
        return;
    }
    const dim3 block(256), grid((unsigned)std::min<size_t>((total + 255) / 256, 148 * 8));
    auto go = [&](auto in, auto out) {
        using T = decltype(in);
        using O = decltype(out);
        launch_after(weighted_reduce_kernel<T, O>, grid, block, s, static_cast<const T*>(src), weights, tokens, routes, h, static_cast<O*>(y));
    };
    if (in_dtype == MFQB_F32) {
        if (y_dtype == MFQB_F32) go(float{}, float{});
        else go(float{}, __nv_bfloat16{});
    } else {
        if (y_dtype == MFQB_F32) go(__nv_bfloat16{}, float{});
        else go(__nv_bfloat16{}, __nv_bfloat16{});
    }
}

void launch_route_plan(const int32_t* ids, int pairs, int experts, int tile_m, int32_t* expert_bounds, int32_t* tile_bounds,
                       int32_t* pair_order, cudaStream_t stream) {
    if (experts <= kRoutePlanExperts && pairs <= kRoutePlanPairs) {
        launch_after(route_plan_kernel, dim3(1), dim3(32 * kRoutePlanWarps), stream, ids, pairs, experts, tile_m, expert_bounds, tile_bounds, pair_order);
        return;
    }
    const int blocks = (experts + 3) / 4;
    route_count_kernel<<<blocks, 128, 0, stream>>>(ids, pairs, experts, expert_bounds + 1);
    route_scan_kernel<<<1, 32, 0, stream>>>(experts, tile_m, expert_bounds, tile_bounds);
    route_place_kernel<<<blocks, 128, 0, stream>>>(ids, pairs, experts, expert_bounds, pair_order);
    MFQB_CUDA(cudaGetLastError());
}

}  // namespace mfqb

using namespace mfqb;

extern "C" {
#pragma GCC visibility push(default)

int mfqb_moe_topk(const float* logits, int tokens, int experts, int k, int mode, const float* bias, int normalize,
                  float norm_floor, float scale, int32_t* ids, float* weights, mfqb_stream_t stream) {
    return guarded([&] {
        if (!logits || !ids || !weights) fail(MFQB_ERR_ARG, "mfqb_moe_topk: null argument");
        if (tokens < 0 || experts < 1 || experts > 4096) fail(MFQB_ERR_ARG, "mfqb_moe_topk: experts must be in [1, 4096]");
        if (k < 1 || k > 16 || k > experts) fail(MFQB_ERR_ARG, "mfqb_moe_topk: top_k must be in [1, min(16, experts)]");
        if (mode < 0 || mode > 3) fail(MFQB_ERR_ARG, "mfqb_moe_topk: unknown router mode %d", mode);
        if (tokens == 0) return;
        const dim3 grid((tokens + 3) / 4), block(128);
        if (experts <= 128) launch_after(moe_topk_regs_kernel<4>, grid, block, stream, logits, bias, ids, weights, tokens, experts, k, mode, normalize, norm_floor, scale);
        else if (experts <= 256) launch_after(moe_topk_regs_kernel<8>, grid, block, stream, logits, bias, ids, weights, tokens, experts, k, mode, normalize, norm_floor, scale);
        else if (experts <= 512) launch_after(moe_topk_regs_kernel<16>, grid, block, stream, logits, bias, ids, weights, tokens, experts, k, mode, normalize, norm_floor, scale);
        else moe_topk_kernel<<<grid, block, 0, stream>>>(logits, bias, ids, weights, tokens, experts, k, mode, normalize, norm_floor, scale);
        MFQB_CUDA(cudaGetLastError());
    });
}

int mfqb_moe_route_plan(const int32_t* ids, int tokens, int k, int experts, int tile_m, int32_t* expert_bounds,
                        int32_t* tile_bounds, int32_t* pair_order, mfqb_stream_t stream) {
    return guarded([&] {
        if (!ids || !expert_bounds || !tile_bounds || !pair_order) fail(MFQB_ERR_ARG, "mfqb_moe_route_plan: null argument");
        if (tokens < 0 || k < 1 || experts < 1 || tile_m < 1) fail(MFQB_ERR_ARG, "mfqb_moe_route_plan: bad sizes");
        launch_route_plan(ids, tokens * k, experts, tile_m, expert_bounds, tile_bounds, pair_order, stream);
    });
}

int mfqb_moe_swiglu(const void* gate_up, int in_dtype, int rows, int f, void* hidden_bf16, mfqb_stream_t stream) {
    return guarded([&] {
        if (!gate_up || !hidden_bf16 || rows < 0 || f < 1) fail(MFQB_ERR_ARG, "mfqb_moe_swiglu: bad argument");
        launch_swiglu(gate_up, in_dtype, rows, f, hidden_bf16, stream);
    });
}

int mfqb_moe_weighted_reduce(const void* expert_out, int in_dtype, const float* weights, int tokens, int routes, int h, void* y,
                             int y_dtype, mfqb_stream_t stream) {
    return guarded([&] {
        if (!expert_out || !weights || !y || tokens < 0 || routes < 1 || h < 1) fail(MFQB_ERR_ARG, "mfqb_moe_weighted_reduce: bad argument");
        launch_weighted_reduce(expert_out, in_dtype, weights, tokens, routes, h, y, y_dtype, stream);
    });
}

#pragma GCC visibility pop
}  // extern "C"
