// Host side of the tensor-memory tile kernel (tile_tc.cuh): activation tiles, shared-memory plan, launches.
#include <algorithm>
#include <cmath>
#include <mutex>

#include "cuda_util.h"
#include "tile_tc.h"
#include "tile_tc_launch.cuh"

namespace mfqb {

int* device_status_word(int device);

// ---- activations ---------------------------------------------------------------------------------------------------------
struct XTilesArgs {
    const void* x;
    int kind;              // TileX
    int k, x_rows;
    size_t row_bytes;
    unsigned char* out;
    float* down;
    // experts: a block row is a position of the route plan, its source row the pair (src_div = 1), the pair's token (src_div =
    // routes), or the position itself (src_div = 0)
    const int *expert_bounds, *tile_bounds, *pair_order, *expert_pool;
    int n_experts, src_div, m;
    int t8[kTileMaxPools], gs[kTileMaxPools], nchunks[kTileMaxPools];
    int staged;            // bf16 rows go through shared memory
    unsigned* counters;    // the product's arrival counts, cleared here: nothing is left over from a call that was cut short
    int n_counters;
};

// (2^e, 2^-e) with 2^e * max in [2^14, 2^15); (1, 1) for a zero, subnormal or non-finite maximum.
__device__ __forceinline__ float2 x_row_scale(uint32_t absmax_bits) {
    int eb = (int)(absmax_bits >> 23);
    if (eb == 0 || eb == 255) return make_float2(1.f, 1.f);
    eb = max(eb, 15);   // below 2^-112 rows keep fewer bits
    return make_float2(__uint_as_float((uint32_t)(268 - eb) << 23), __uint_as_float((uint32_t)(eb - 14) << 23));
}

template <int KIND>
__device__ __forceinline__ float x_value(const void* row, int k, int j) {
    if constexpr (KIND == kTileXShared) return __bfloat162float(static_cast<const __nv_bfloat16*>(row)[j]);
    if constexpr (KIND == kTileXBf16) return __bfloat162float(__ldcg(static_cast<const __nv_bfloat16*>(row) + j));
    const float v = __ldcg(static_cast<const float*>(row) + j);
    return __ldcg(static_cast<const float*>(row) + k + j) * v / (1.0f + expf(-v));
}
// Four consecutive values from column j on, zero past the row.
template <int KIND>
__device__ __forceinline__ float4 x_quad(const void* row, int k, int j, bool aligned) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (aligned && j + 3 < k) {
        if constexpr (KIND == kTileXBf16 || KIND == kTileXShared) {
            const uint2* at = reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(row) + j);
            const uint2 r = KIND == kTileXShared ? *at : __ldcg(at);
            v = make_float4(__uint_as_float(r.x << 16), __uint_as_float(r.x & 0xFFFF0000u), __uint_as_float(r.y << 16), __uint_as_float(r.y & 0xFFFF0000u));
        } else {
            v = __ldcg(reinterpret_cast<const float4*>(static_cast<const float*>(row) + j));
            const float4 u = __ldcg(reinterpret_cast<const float4*>(static_cast<const float*>(row) + k + j));
            v = make_float4(u.x * v.x / (1.0f + expf(-v.x)), u.y * v.y / (1.0f + expf(-v.y)), u.z * v.z / (1.0f + expf(-v.z)), u.w * v.w / (1.0f + expf(-v.w)));
        }
    } else {
        if (j < k) v.x = x_value<KIND>(row, k, j);
        if (j + 1 < k) v.y = x_value<KIND>(row, k, j + 1);
        if (j + 2 < k) v.z = x_value<KIND>(row, k, j + 2);
        if (j + 3 < k) v.w = x_value<KIND>(row, k, j + 3);
    }
    return v;
}
__device__ __forceinline__ uint32_t x_pack(float a, float b) {   // non-finite -> NaN, which poisons the token's outputs
    const __half ha = isfinite(a) ? __float2half_rn(a) : __ushort_as_half((unsigned short)0x7E00);
    const __half hb = isfinite(b) ? __float2half_rn(b) : __ushort_as_half((unsigned short)0x7E00);
    return (uint32_t)__half_as_ushort(ha) | ((uint32_t)__half_as_ushort(hb) << 16);
}

__device__ __forceinline__ uint32_t x_pack_rest(float a, float b, uint32_t packed) {   // what rounding cut off; 0 beside a NaN
    const float2 r = __half22float2(*reinterpret_cast<const __half2*>(&packed));
    const __half2 h = __floats2half2_rn(isfinite(a) ? a - r.x : 0.f, isfinite(b) ? b - r.y : 0.f);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// Slabs first, first + step, ... of a row's tile: see x_tiles_kernel.  r: row of the tile, pitch: bytes of a 64-column slab of it.
template <int KIND, int XTERMS = 1>
__device__ __forceinline__ void x_write_slabs(const void* row, bool row_al, int k, int gs, int T, int nslabs, float scale, unsigned char* dst, int r, int pitch, int first,
                                              int step) {
    const bool quad_al = row_al && (gs & 3) == 0;
    for (int js = first; js < nslabs; js += step) {
        const int ch = js / (4 * T), jj = js - ch * 4 * T, h = jj & 1, ft = jj >> 1, f = ft / T, t = ft - f * T;
        const int g = ch * kChunkGroupsB + 4 * f + 2 * h;
        uint32_t w[8], e[8];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int slot = 8 * t + 4 * (c & 1), k0 = (g + (c >> 1)) * gs + slot;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (slot + 3 < gs) {
                v = x_quad<KIND>(row, k, k0, quad_al);
            } else {
                if (slot < gs && k0 < k) v.x = x_value<KIND>(row, k, k0);
                if (slot + 1 < gs && k0 + 1 < k) v.y = x_value<KIND>(row, k, k0 + 1);
                if (slot + 2 < gs && k0 + 2 < k) v.z = x_value<KIND>(row, k, k0 + 2);
            }
            w[c] = x_pack(v.x * scale, v.z * scale);
            w[4 + c] = x_pack(v.y * scale, v.w * scale);
            if constexpr (XTERMS == 2) {
                e[c] = x_pack_rest(v.x * scale, v.z * scale, w[c]);
                e[4 + c] = x_pack_rest(v.y * scale, v.w * scale, w[4 + c]);
            }
        }
        const int slab = js & 3;
        unsigned char* at = dst + (size_t)(js >> 2) * XTERMS * pitch;
        *reinterpret_cast<uint4*>(at + (((2 * slab) ^ (r & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
        *reinterpret_cast<uint4*>(at + (((2 * slab + 1) ^ (r & 7)) << 4)) = make_uint4(w[4], w[5], w[6], w[7]);
        if constexpr (XTERMS == 2) {
            at += pitch;
            *reinterpret_cast<uint4*>(at + (((2 * slab) ^ (r & 7)) << 4)) = make_uint4(e[0], e[1], e[2], e[3]);
            *reinterpret_cast<uint4*>(at + (((2 * slab + 1) ^ (r & 7)) << 4)) = make_uint4(e[4], e[5], e[6], e[7]);
        }
    }
}

// Scales a row to the top of the f16 range and writes it as B operand: per 64-column slab the tile's rows of 128 bytes with
// the 128-byte swizzle, columns in the decoders' order (slab of 16 columns (f, t, h): octet t of groups 4f + 2h, + 1; quads
// c = 0..3 of these 16 slots, their slots 0 and 2 in columns 2c, 2c + 1, slots 1 and 3 in columns 8 + 2c, + 1).  Slots past
// the group size, groups and columns past the row are zero.  Grid (rows, splits), for a grid's other dimensions end at 65535:
// every CTA takes the row's maximum for itself (from L2; a second launch for the maxima costs more for the rows of a decoding
// batch) and writes its share.
template <int KIND, int XTERMS>
__global__ void __launch_bounds__(256) x_tiles_kernel(const __grid_constant__ XTilesArgs a) {
    extern __shared__ __align__(16) unsigned char x_row[];   // bf16 rows: kept between the two passes (a.staged)
    __shared__ uint32_t red[8];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int p = blockIdx.x;
    int pool = 0, src = p, tile_begin = p / a.x_rows * a.x_rows, ncols = min(a.x_rows, a.m - tile_begin), base = tile_begin;
    if (a.tile_bounds != nullptr) {
        if (p >= a.expert_bounds[a.n_experts]) return;
        int lo = 0, hi = a.n_experts - 1;   // expert with expert_bounds[e] <= p < expert_bounds[e + 1]
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (a.expert_bounds[mid] <= p) lo = mid;
            else hi = mid - 1;
        }
        pool = a.expert_pool[lo];
        if (pool < 0) return;
        const int eb = a.expert_bounds[lo], local = (p - eb) / a.x_rows * a.x_rows;
        tile_begin = eb + local;
        ncols = min(a.x_rows, a.expert_bounds[lo + 1] - tile_begin);
        base = tile_x_row(eb, lo, local);
        if (a.src_div > 0) src = a.pair_order[p] / a.src_div;
    }
    const int T = a.t8[pool], gs = a.gs[pool], nslabs = a.nchunks[pool] * 4 * T, k = a.k, tid = threadIdx.x;
    constexpr int ESZ = KIND == kTileXBf16 ? 2 : 4;
    const unsigned char* row = static_cast<const unsigned char*>(a.x) + (size_t)src * k * (KIND == kTileXSwiglu ? 2 : 1) * ESZ;
    const bool row_al = (reinterpret_cast<uintptr_t>(row) & (4 * ESZ - 1)) == 0 && (KIND != kTileXSwiglu || (k & 3) == 0);
    // largest magnitude as float bits (they order like the values, NaN and infinity largest).  Eight loads in flight per
    // thread, out-of-range ones predicated off: a plain unrolled loop runs its few iterations one after the other.
    uint32_t ab = 0u;
    if (KIND == kTileXBf16 && (reinterpret_cast<uintptr_t>(row) & 15) == 0 && (k & 7) == 0) {
        for (int j0 = tid; j0 < (k >> 3); j0 += 2048) {
            uint4 v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = j0 + 256 * u < (k >> 3) ? __ldcg(reinterpret_cast<const uint4*>(row) + j0 + 256 * u) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                if (a.staged && j0 + 256 * u < (k >> 3)) reinterpret_cast<uint4*>(x_row)[j0 + 256 * u] = v[u];
                const uint32_t w4[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
                for (int i = 0; i < 4; ++i) ab = max(ab, max(w4[i] & 0x7FFF0000u, (w4[i] << 16) & 0x7FFF0000u));
            }
        }
    } else {
        for (int j0 = 4 * tid; j0 < k; j0 += 4096) {
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = j0 + 1024 * u < k ? x_quad<KIND>(row, k, j0 + 1024 * u, row_al) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                ab = max(max(ab, __float_as_uint(fabsf(v[u].x))), max(__float_as_uint(fabsf(v[u].y)), max(__float_as_uint(fabsf(v[u].z)), __float_as_uint(fabsf(v[u].w)))));
        }
    }
    for (int o = 16; o > 0; o >>= 1) ab = max(ab, __shfl_xor_sync(0xffffffffu, ab, o));
    if ((tid & 31) == 0) red[tid >> 5] = ab;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i) ab = max(ab, red[i]);
    const float2 sc = x_row_scale(ab);
    if (blockIdx.y == 0 && tid == 0) a.down[p] = sc.y;
    if (p == 0 && blockIdx.y == 0)
        for (int i = tid; i < a.n_counters; i += 256) a.counters[i] = 0u;
    const int r = p - tile_begin, pitch = ((ncols + 7) & ~7) * 128;
    unsigned char* dst = a.out + (size_t)base * a.row_bytes + (size_t)r * 128;
    if (KIND == kTileXBf16 && a.staged && (reinterpret_cast<uintptr_t>(row) & 15) == 0 && (k & 7) == 0)
        x_write_slabs<kTileXShared>(x_row, true, k, gs, T, nslabs, sc.x, dst, r, pitch, blockIdx.y * 256 + tid, gridDim.y * 256);
    else
        x_write_slabs<KIND, XTERMS>(row, row_al, k, gs, T, nslabs, sc.x, dst, r, pitch, blockIdx.y * 256 + tid, gridDim.y * 256);
}

// The same behind a residual add and RMSNorm, one CTA per row: the row stays in registers between the sum of squares and the
// scaling, and in shared memory as bf16 between the scaling and the slabs.  In a decoder block this is one kernel (and one
// trip through memory) less before q|k|v and before gate|up.
__global__ void __launch_bounds__(1024) norm_tiles_kernel(const __grid_constant__ XTilesArgs a, const __grid_constant__ TileNorm nm) {
    constexpr int KEEP = 2;
    extern __shared__ __align__(16) unsigned char norm_row[];
    __shared__ float red[32];
    __shared__ uint32_t red_max[32];
    const int tid = threadIdx.x, nv = a.k >> 2, p = blockIdx.x;
    float4* row = reinterpret_cast<float4*>(nm.h + (size_t)p * a.k);
    const float4* drow = nm.delta ? reinterpret_cast<const float4*>(nm.delta + (size_t)p * a.k) : nullptr;
    const float4* g4 = reinterpret_cast<const float4*>(nm.gamma);
    uint2* xs = reinterpret_cast<uint2*>(norm_row);
    float4 v[KEEP], g[KEEP];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#pragma unroll
    for (int j = 0; j < KEEP; ++j)   // gamma is a constant of the model: fetched while the predecessor still runs
        if (tid + j * 1024 < nv) g[j] = __ldg(g4 + tid + j * 1024);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    float ss = 0.f;
    auto take = [&](int i) {
        float4 t = row[i];
        if (drow) {
            const float4 d = drow[i];
            t.x += d.x; t.y += d.y; t.z += d.z; t.w += d.w;
            row[i] = t;
        }
        ss += t.x * t.x + t.y * t.y + t.z * t.z + t.w * t.w;
        return t;
    };
#pragma unroll
    for (int j = 0; j < KEEP; ++j)
        if (tid + j * 1024 < nv) v[j] = take(tid + j * 1024);
    for (int i = tid + KEEP * 1024; i < nv; i += 1024) take(i);
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((tid & 31) == 0) red[tid >> 5] = ss;
    __syncthreads();
    float tot = red[tid & 31];
    for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
    const float inv = rsqrtf(tot / (float)a.k + nm.eps);
    uint32_t ab = 0u;
    auto put = [&](int i, const float4& t, const float4& gm) {
        const __nv_bfloat162 lo = __floats2bfloat162_rn(t.x * inv * gm.x, t.y * inv * gm.y), hi = __floats2bfloat162_rn(t.z * inv * gm.z, t.w * inv * gm.w);
        const uint32_t w0 = *reinterpret_cast<const uint32_t*>(&lo), w1 = *reinterpret_cast<const uint32_t*>(&hi);
        ab = max(max(ab, max(w0 & 0x7FFF0000u, (w0 << 16) & 0x7FFF0000u)), max(w1 & 0x7FFF0000u, (w1 << 16) & 0x7FFF0000u));
        xs[i] = make_uint2(w0, w1);
    };
#pragma unroll
    for (int j = 0; j < KEEP; ++j)
        if (tid + j * 1024 < nv) put(tid + j * 1024, v[j], g[j]);
    for (int i = tid + KEEP * 1024; i < nv; i += 1024) put(i, row[i], __ldg(g4 + i));
    for (int o = 16; o > 0; o >>= 1) ab = max(ab, __shfl_xor_sync(0xffffffffu, ab, o));
    if ((tid & 31) == 0) red_max[tid >> 5] = ab;
    __syncthreads();
    ab = red_max[tid & 31];
    for (int o = 16; o > 0; o >>= 1) ab = max(ab, __shfl_xor_sync(0xffffffffu, ab, o));
    const float2 sc = x_row_scale(ab);
    if (tid == 0) a.down[p] = sc.y;
    if (p == 0)
        for (int i = tid; i < a.n_counters; i += 1024) a.counters[i] = 0u;
    const int T = a.t8[0], tile_begin = p / a.x_rows * a.x_rows, r = p - tile_begin, pitch = ((min(a.x_rows, a.m - tile_begin) + 7) & ~7) * 128;
    x_write_slabs<kTileXShared>(norm_row, true, a.k, a.gs[0], T, a.nchunks[0] * 4 * T, sc.x, a.out + (size_t)tile_begin * a.row_bytes + (size_t)r * 128, r, pitch, tid, 1024);
}

// All of the SM's unified memory as shared memory.  Kernels of a chain that ask for different splits do not become resident
// beside one another: the activation kernels (up to 33 KB) would wait for the tile kernel's CTAs to leave, and these for them
// (16 rows through NINT6 4096 x 14336: 25.0 us instead of 20.9).
template <auto kernel>
static void whole_carveout() {
    static bool done[64] = {};
    int dev = 0;
    MFQB_CUDA(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && done[dev]) return;
    MFQB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    if (dev >= 0 && dev < 64) done[dev] = true;
}

static void launch_x_tiles(XTilesArgs a, int kind, int x_terms, int rows, int nslabs, int sms, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    // one CTA per row fills the chip from a few hundred rows on; fewer rows are shared out
    const int splits = std::max(1, std::min((nslabs + 255) / 256, 2 * sms / std::max(rows, 1)));
    // a second trip to L2 for the values costs a decoding batch 0.7 us of its chain; rows of up to 32 KB fit beside a tile CTA
    a.staged = kind == kTileXBf16 && a.k <= 16384 && rows <= 64;
    if (a.staged) cfg.dynamicSmemBytes = (size_t)(a.k + 7) / 8 * 16;
    cfg.gridDim = dim3((unsigned)rows, (unsigned)splits);
    cfg.blockDim = dim3(256);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    auto go = [&](auto kind_c, auto terms_c) {
        constexpr int KIND = decltype(kind_c)::value, XTERMS = decltype(terms_c)::value;
        whole_carveout<x_tiles_kernel<KIND, XTERMS>>();
        MFQB_CUDA(cudaLaunchKernelEx(&cfg, x_tiles_kernel<KIND, XTERMS>, a));
    };
    using std::integral_constant;
    if (kind == kTileXBf16) go(integral_constant<int, kTileXBf16>{}, integral_constant<int, 1>{});
    else if (x_terms == 1) go(integral_constant<int, kTileXSwiglu>{}, integral_constant<int, 1>{});
    else go(integral_constant<int, kTileXSwiglu>{}, integral_constant<int, 2>{});
}

// ---- plans ---------------------------------------------------------------------------------------------------------------
static size_t x_row_bytes(const NintDevB& w) { return (size_t)w.nchunks * w.t8 * 128; }

// Rings for token tiles of `n` columns: two stages of each, then records up to 144 KB (what a decoder step frees comes back from
// HBM 2 us later: with 64 KB the expert products waited for it, 128 experts and 32 tokens 183 us instead of 170) and activation
// slabs.  False when the codec's tables and two stages of each do not fit.
static bool tile_plan(TileArgs& a, TilePlan& p, int n, size_t rec_bytes, int t8, int terms, int x_terms, size_t ctx_bytes) {
    const size_t budget = kTileDynSmem - 1024, ctx = (ctx_bytes + 15) / 16 * 16;
    a.n_mma = n;
    a.d_cols = n <= 32 ? 32 : (n <= 64 ? 64 : (n <= 128 ? 128 : 256));
    // a second accumulator, unless two-term weights need its columns for two stages of either half
    a.d_bufs = n <= 128 && (terms == 1 || (512 - 2 * a.d_cols) / (16 * t8 * terms) >= 4) ? 2 : 1;
    const int a_total = 512 - a.d_bufs * a.d_cols;
    // Small N: every barrier round trip costs more than the tensor work between two of them, so a step takes two chunks and an
    // activation stage all of a step.  Large N: one chunk a step, activations in 64-column slabs.
    for (int step = 2; step >= 0; --step) {
        a.x_whole = step > 0;
        a.step = std::max(step, 1);
        a.a_cols = 16 * t8 * terms * a.step;
        a.a_stages = std::min(kTileAStages, a_total / a.a_cols);
        const size_t rec_stage = 8 * rec_bytes * a.step, x_stage = (size_t)n * 128 * x_terms * (a.x_whole ? a.step * t8 : 1);
        if (a.a_stages < 2 || ctx + (a.step > 1 ? 3 : 2) * rec_stage + 2 * x_stage > budget || (a.x_whole && x_stage > 24 * 1024)) continue;
        size_t left = budget - ctx - 2 * rec_stage - 2 * x_stage;
        int rs = 2, xs = 2;
        for (bool grown = true; grown;) {
            grown = false;
            if (xs < 4 && left >= x_stage) { ++xs; left -= x_stage; grown = true; }
            if (rs < kTileRecStages && (size_t)(rs + 1) * rec_stage <= 144 * 1024 && left >= rec_stage) { ++rs; left -= rec_stage; grown = true; }
        }
        while (xs < kTileXStages && !a.x_whole && left >= x_stage) { ++xs; left -= x_stage; }
        a.rec_stages = rs;
        a.rec_stage_bytes = (int)rec_stage;
        a.x_stages = xs;
        a.x_stage_bytes = (int)x_stage;
        p.smem = 1024 + std::max((size_t)xs * x_stage + (size_t)rs * rec_stage + ctx, std::max<size_t>(n, 32) * kTileRows * 4);   // a shared tile's parts are added there
        a.sum_bytes = (int)p.smem - 1024;
        return true;
    }
    return false;
}

static cudaError_t launch_one(const TileArgs& a, const TilePlan& p, int terms, cudaStream_t s) {
    switch (a.pools[0].table ? 0 : a.pools[0].bits) {
        case 0: return launch_tile_nvq(a, p, terms, s);
        case 2: return launch_tile_bits<2>(a, p, s);
        case 3: return launch_tile_bits<3>(a, p, s);
        case 4: return launch_tile_bits<4>(a, p, s);
        case 5: return launch_tile_bits<5>(a, p, s);
        case 6: return launch_tile_bits<6>(a, p, s);
        case 8: return launch_tile_bits<8>(a, p, s);
        default: return cudaErrorNotSupported;
    }
}

// Exponent that takes the state scales of a joint-codebook record to the top of what their products with the codes (up to 127)
// may reach in f16.
static int lattice_shift(const float* lut) {
    float top = 0.f;
    for (int i = 0; i < 16; ++i) top = std::max(top, std::fabs(lut[i]));
    int e = 0;
    if (top > 0.f && std::isfinite(top)) std::frexp(top, &e);   // top = m 2^e, m in [0.5, 1)
    return 8 - e;
}
// f16 state scales of a lattice record, normalised so that code x scale stays below 2^15.
void tile_lattice_scales(const NintDevB& w, uint16_t (&lut16)[16], float& undo) {
    const int shift = w.jsc ? lattice_shift(w.lut) : 0;
    for (int i = 0; i < 16; ++i) lut16[i] = __half_as_ushort(__float2half(std::ldexp(w.jsc ? w.lut[i] : (float)i, shift)));
    undo = std::ldexp(1.f, -shift);
}
int lattice_terms(const float* lut, const int8_t* codes, size_t n_codes) {
    bool used[128] = {};
    for (size_t i = 0; i < n_codes; ++i) used[codes[i] & 127] = true;
    const int shift = lattice_shift(lut);
    int terms = 1;
    for (int s = 0; s < 16; ++s) {
        const float scaled = std::ldexp(lut[s], shift);
        if (std::isfinite(lut[s]) && __half2float(__float2half(scaled)) != scaled) return 0;   // scales more than some 2^21 apart
        for (int c = 0; c < 128; ++c) {
            if (!used[c] || lut[s] == 0.f) continue;
            int e;
            const float m = std::frexp(lut[s] * (float)c, &e) * 2048.f;   // 11 significant bits are an f16
            if (c && m != std::floor(m)) terms = 2;
        }
    }
    return terms;
}

// y [m, n] = x [m, k] W^T.  False when this weight has no tile kernel.
bool launch_tile_product(const NintDevB& w, const void* x, int m, void* y, int y_dtype, int device, cudaStream_t s, bool glu, const TileNorm* norm) {
    if (norm && (w.k % 4 || w.k > 20480)) return false;   // the row as bf16 in a CTA's 48 KB
    TileArgs a{};
    TilePlan p;
    const int terms = w.tile_terms;
    if (terms == 0) return false;
    // token tiles: as few as 256 columns allow, or fewer columns where a codebook of 128 KB leaves no room for the rings of that many
    // (giving up there cost a product of 256 rows 32 passes of the single-row kernel), of equal size
    const size_t rec_bytes = (size_t)w.rec_words * 4, ctx_bytes = w.table ? (size_t)w.table_words * 4 + 64 : 0;
    auto equal_tiles = [m](int most) {
        const int ntok = (m + most - 1) / most;
        return std::max(16, ((m + ntok - 1) / ntok + 15) / 16 * 16);
    };
    int n = equal_tiles(256);
    for (int most = n; !tile_plan(a, p, n, rec_bytes, w.t8, terms, 1, ctx_bytes); n = equal_tiles(most))
        if ((most -= 16) < 16) return false;
    const int row_tiles = (w.n + kTileRows - 1) / kTileRows, sms = device_sm_count(device);
    const long long tiles = (long long)row_tiles * ((m + n - 1) / n), units = tiles * w.nchunks;
    if (units * (sms + 1) >= (1ll << 31) * 1ll * sms || units >= (1ll << 31)) return false;
    a.pools[0] = w;
    a.lut_undo = 1.f;
    if (w.table) tile_lattice_scales(w, a.lut16, a.lut_undo);
    a.m = m;
    a.ntok = (m + n - 1) / n;
    a.x_rows = n;
    a.x_row_bytes = x_row_bytes(w);
    a.y = y;
    a.y_dtype = y_dtype;
    a.ldy = glu ? w.n / 2 : w.n;
    a.glu = glu;
    a.units = (int)units;
    a.only_pool = -1;
    a.error = device_status_word(device);
    // Fewer tiles than SMs: either as many CTAs per tile as fit, each with one part of one tile, or equal ranges over all SMs.
    // The latter give a CTA less to do, but parts of two tiles, and two sums over CTAs that follow one another: each costs
    // about as much as three chunks (1.5 to 2.5 us against 0.6 for a chunk of 16 tokens; both grow with the tokens), and half of
    // the second one is hidden behind the CTA's other part: with six chunks instead of three for two sums, 16 rows through NINT6
    // 4096 x 14336 took 22.4 us instead of 21.1, with none 8 rows through NVQ3 17408 x 5120 31.4 instead of 23.8.
    // A chunk of groups of 16 is over sooner, in 0.4 us of 40 tokens and 0.8 of 250, beside 4.6 and 14 for two sums: they count six
    // chunks, more than 128 tokens ten.  Split and equal, us: NINT2-16 5000 x 2888, 20 rows 11.9 and 15.8, 512 rows 32.3 and 39.2
    // (three chunks chose the latter); 14336 x 4096, 60 rows 29.9 and 28.7; over 1400 shapes 4 % from one line to the other.
    // Without sharing there is no sum.  At most a dozen CTAs per tile (kTileGroup): the last one adds the others' parts.
    const long long sums = terms == 1 && w.t8 == 2 ? (n > 128 ? 10 : 6) : 3;
    const long long split = std::min({(long long)sms / tiles, (long long)std::max(1, w.nchunks / 2), (long long)kTileGroup});
    const long long chunks_split = split ? (w.nchunks + split - 1) / split + (split > 1 ? 3 : 0) : 0, chunks_equal = (units + sms - 1) / sms + sums;
    a.split = split && chunks_split <= chunks_equal ? (int)split : 0;
    p.grid = a.split ? (int)(tiles * split) : (int)std::max<long long>(1, std::min<long long>(sms, (units + 1) / 2));
    // The two launches below belong together: another thread's on the same stream would take the scratch between them.
    static std::mutex launches[64];
    std::lock_guard<std::mutex> lock(launches[device]);
    // One call with this weight makes room for every smaller batch of it: decoding batches keep a small block of their own beside
    // the prefill's, and the parts of shared tiles are as many as any plan may have.
    static GrowOnlyScratch xs[2], parts, counts;
    const char* what = "mfqb_mul_mat (f16 activation tiles)";
    auto x_bytes = [&](int rows) { return ((size_t)(rows + 7) / 8 * 8 * a.x_row_bytes + 255) / 256 * 256; };
    const size_t xb = x_bytes(m);
    if (m > 16) xs[0].reserve(device, x_bytes(16) + 64, s, what);
    unsigned char* buf = static_cast<unsigned char*>(xs[m > 16].get(device, xb + (size_t)m * 4, s, what));
    a.x = buf;
    a.x_down = reinterpret_cast<const float*>(buf + xb);
    a.partial = static_cast<float*>(parts.get(device, (size_t)sms * 2 * 256 * kTileRows * 4, s, "mfqb_mul_mat (parts of shared tiles)", true));
    a.counters = static_cast<unsigned*>(counts.get(device, (size_t)sms * 2 * 4, s, "mfqb_mul_mat (tile counters)", true));
    XTilesArgs xa{};
    xa.x = x;
    xa.kind = kTileXBf16;
    xa.k = w.k;
    xa.m = m;
    xa.x_rows = n;
    xa.row_bytes = a.x_row_bytes;
    xa.out = buf;
    xa.down = reinterpret_cast<float*>(buf + xb);
    xa.counters = a.counters;
    xa.n_counters = 2 * p.grid;
    xa.t8[0] = w.t8;
    xa.gs[0] = w.gs;
    xa.nchunks[0] = w.nchunks;
    if (norm) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)m);
        cfg.blockDim = dim3(1024);
        cfg.dynamicSmemBytes = (size_t)w.k * 2;
        cfg.stream = s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        whole_carveout<norm_tiles_kernel>();
        MFQB_CUDA(cudaLaunchKernelEx(&cfg, norm_tiles_kernel, xa, *norm));
    } else {
        launch_x_tiles(xa, kTileXBf16, 1, m, w.nchunks * 4 * w.t8, sms, s);
    }
    const cudaError_t e = launch_one(a, p, terms, s);
    if (e == cudaErrorNotSupported) return false;
    if (e != cudaSuccess)
        fail(MFQB_ERR_CUDA, "%s%d gs=%d tile product launch (m = %d, %zu bytes of shared memory): %s", w.table ? "NVQ index bits " : "NINT", w.table ? w.index_bits : w.bits,
             w.gs, m, p.smem, cudaGetErrorString(e));
    return true;
}

// ---- expert products -----------------------------------------------------------------------------------------------------
static bool experts_one_launch(const NintDevB* pools, const int* held, int npools) {   // the codecs of TileExperts
    for (int i = 0; i < npools; ++i) {
        const int c = pools[i].bits * 16 + pools[i].t8;
        if (held[i] && c != 2 * 16 + 2 && c != 3 * 16 + 3 && c != 4 * 16 + 3 && c != 5 * 16 + 4 && c != 6 * 16 + 3 && c != 8 * 16 + 3 && c != 8 * 16 + 6) return false;
    }
    return true;
}
// Two terms where a group size is no multiple of eight, or a codec outside the one-launch kernel below two dozen pairs per expert:
// these ran on the integer kernels before there was a tile kernel for them.
int tile_experts_terms(const NintDevB* pools, const int* held, int npools, int pairs, int experts) {
    for (int i = 0; i < npools; ++i)
        if (held[i] && pools[i].tile_terms == 2) return 2;
    return experts_one_launch(pools, held, npools) || pairs / 24 >= experts ? 1 : 2;
}
static int x_terms_of(int terms, bool float_x) { return terms == 2 && float_x ? 2 : 1; }   // bf16 values are f16 numbers
// Pairs per tile: one tile for nearly every expert, since each tile decodes the expert's weights once (three standard
// deviations above the mean of evenly routed pairs); a tile's unused columns cost tensor time only, which the decoding hides.
int tile_experts_rows(int pairs, int experts, int max_rows) {
    const double mean = (double)pairs / std::max(experts, 1);
    const int rows = (int)(mean + 3.0 * std::sqrt(mean) + 3.0);
    return std::max(16, std::min(max_rows, (rows + 15) / 16 * 16));
}
size_t tile_experts_x_bytes(const NintDevB* pools, const int* held, int npools, int pairs, int experts, int terms, bool float_x) {
    size_t row = 0;
    for (int i = 0; i < npools; ++i)
        if (held[i]) row = std::max(row, x_row_bytes(pools[i]) * x_terms_of(terms, float_x));
    const size_t rows = (size_t)(pairs + 7) / 8 * 8 + 8 * ((size_t)experts + 1);   // tile_x_row
    return (rows * row + 255) / 256 * 256 + ((size_t)pairs * 4 + 255) / 256 * 256;
}
int tile_experts_max_rows(const NintDevB* pools, const int* held, int npools, int terms, bool float_x) {
    if (npools > kTileMaxPools || (terms == 2 && !experts_one_launch(pools, held, npools))) return 0;
    TileArgs a{};
    TilePlan p;
    size_t rec = 0;
    int t8 = 0;
    for (int i = 0; i < npools; ++i) {
        if (!held[i]) continue;
        rec = std::max(rec, (size_t)pools[i].rec_words * 4);
        t8 = std::max(t8, pools[i].t8);
    }
    int n = 256;
    while (n > 0 && t8 && !tile_plan(a, p, n, rec, t8, terms, x_terms_of(terms, float_x), 0)) n -= 16;
    return n;
}

void launch_tile_experts_product(const NintDevB* pools, const int* held, int npools, const TileRoutes& r, int terms, const void* x, TileX kind, int src_div, void* xbuf, void* y,
                                 int y_dtype, bool scatter, int rows_per_expert, int rb_per_expert, int device, cudaStream_t s) {
    const int x_terms = x_terms_of(terms, kind != kTileXBf16);
    TileArgs a{};
    TilePlan p;
    XTilesArgs xa{};
    size_t rec = 0;
    int t8 = 0, nslabs = 0, k = 0;
    for (int i = 0; i < npools; ++i) {
        if (!held[i]) continue;
        const NintDevB& w = pools[i];
        a.pools[i] = w;
        a.pools[i].tile_terms = terms;
        rec = std::max(rec, (size_t)w.rec_words * 4);
        t8 = std::max(t8, w.t8);
        a.x_row_bytes = std::max(a.x_row_bytes, x_row_bytes(w) * x_terms);
        nslabs = std::max(nslabs, w.nchunks * 4 * w.t8);
        k = w.k;
        xa.t8[i] = w.t8;
        xa.gs[i] = w.gs;
        xa.nchunks[i] = w.nchunks;
    }
    if (t8 == 0) return;   // nothing held here
    const int n = std::max(16, r.tile_rows), sms = device_sm_count(device);
    if (!tile_plan(a, p, n, rec, t8, terms, x_terms, 0)) fail(MFQB_ERR_UNSUPPORTED, "expert tile product: tiles of %d pairs do not fit shared memory", n);
    unsigned char* buf = static_cast<unsigned char*>(xbuf);
    const size_t rows = (size_t)(r.pairs + 7) / 8 * 8 + 8 * ((size_t)r.n_experts + 1);
    float* down = reinterpret_cast<float*>(buf + (rows * a.x_row_bytes + 255) / 256 * 256);
    xa.x = x;
    xa.kind = kind;
    xa.k = k;
    xa.x_rows = r.tile_rows;
    xa.row_bytes = a.x_row_bytes;
    xa.out = buf;
    xa.down = down;
    xa.expert_bounds = r.expert_bounds;
    xa.tile_bounds = r.tile_bounds;
    xa.pair_order = r.pair_order;
    xa.expert_pool = r.expert_pool;
    xa.n_experts = r.n_experts;
    xa.src_div = src_div;
    launch_x_tiles(xa, kind, x_terms, r.pairs, nslabs, sms, s);
    a.x = buf;
    a.x_rows = r.tile_rows;
    a.x_down = down;
    a.y = y;
    a.y_dtype = y_dtype;
    a.ldy = rows_per_expert;
    a.expert_bounds = r.expert_bounds;
    a.tile_bounds = r.tile_bounds;
    a.pair_order = r.pair_order;
    a.expert_pool = r.expert_pool;
    a.expert_local = r.expert_local;
    a.n_experts = r.n_experts;
    a.rb_per_expert = rb_per_expert;
    a.rows_per_expert = rows_per_expert;
    a.scatter = scatter;
    a.error = device_status_word(device);
    const long long items = (long long)((rows_per_expert + kTileRows - 1) / kTileRows) * (r.pairs / r.tile_rows + std::min(r.pairs, r.n_experts));
    p.grid = (int)std::max<long long>(1, std::min<long long>(sms, items));
    a.only_pool = -1;
    a.lut_undo = 1.f;
    if (experts_one_launch(pools, held, npools)) {
        const cudaError_t e = launch_tile_experts(a, p, terms, x_terms, s);
        if (e != cudaSuccess) fail(MFQB_ERR_CUDA, "expert tile product launch (tiles of %d, %zu bytes of shared memory): %s", n, p.smem, cudaGetErrorString(e));
        return;
    }
    for (int i = 0; i < npools; ++i) {   // other profiles: cohort by cohort
        if (!held[i]) continue;
        TileArgs b = a;
        b.pools[0] = pools[i];
        b.only_pool = i;
        const cudaError_t e = launch_one(b, p, 1, s);
        if (e != cudaSuccess) fail(MFQB_ERR_CUDA, "NINT%d gs=%d expert tile product launch: %s", pools[i].bits, pools[i].gs, cudaGetErrorString(e));
    }
}

}  // namespace mfqb
