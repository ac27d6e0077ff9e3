// Dense decoder step around the packed-weight products: the QuantLinear / FFN-shaped runtime layer
// of the reference (cpp_runtime/mfq_decode.cpp:9116-9407 QuantLinear, 10456-10602 FFN,
// 12210-12400 FullBlock::forward, 13993-14145 Model::hidden_forward / next_token) reduced to what one
// decode step of a Llama-shaped model needs: RMSNorm, fused q|k|v projection, rotary embedding, bf16
// KV-cache write, grouped-query decode attention over the cache, output projection, SwiGLU FFN with a
// fused gate|up projection, final norm, lm_head and arg-max.  Every projection is a packed weight
// handle of this library (mfqb_mul_mat); the small kernels here are the glue between them.
//
// Tensor parallelism (Megatron style, as the reference's load_quant_linear assigns axes by tensor
// name, cpp_runtime/mfq_decode.cpp:9422-9443): q/k/v, gate/up and lm_head are split on the output
// axis (heads, FFN columns, vocabulary rows), o_proj and down_proj on the input axis; a rank holds
// n_q/world query heads and n_kv/world KV heads with their slice of the cache.  The two row-parallel
// products of a layer end in a sum over ranks (mfqb_mul_mat_allreduce for one row, product +
// mfqb_allreduce_f32 for a batch), the arg-max over the vocabulary shards in a small gather.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <memory>
#include <vector>

#include <cmath>

#include "cuda_util.h"
#include "rows_mma.h"
#include "tile_tc.h"

namespace mfqb {

const NintDevB& weight_device_layout(const mfqb_weight* w);
void reserve_fewer_rows(const mfqb_weight* w, int m, bool glu, cudaStream_t s);

constexpr int kHeadDim = 128;

// Every kernel of the step is launched with the programmatic-dependent-launch attribute: it becomes
// resident while its predecessor still runs, and waits here until that one has completed.
__device__ __forceinline__ void dep_wait() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <typename... KArgs, typename... Args>
static void launch_dep_smem(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    MFQB_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...));
}
template <typename... KArgs, typename... Args>
static void launch_dep(void (*kernel)(KArgs...), dim3 grid, dim3 block, cudaStream_t s, Args... args) {
    launch_dep_smem(kernel, grid, block, 0, s, args...);
}

// ---- glue kernels --------------------------------------------------------------------------------

// h [rows, H] (float32 residual stream) += delta [rows, H] (optional); xn = h / rms(h) * gamma as bf16.
// One CTA of 1024 threads per row, four columns per thread and pass: a row of up to 8192 columns is
// read once and stays in registers between the sum of squares and the scaling (H is a multiple of 4).
__global__ void __launch_bounds__(1024) add_rmsnorm_kernel(float* __restrict__ h, const float* __restrict__ delta, const float* __restrict__ gamma,
                                                            __nv_bfloat16* __restrict__ xn, int H, float eps) {
    constexpr int KEEP = 2;
    __shared__ float red[32];
    const int tid = threadIdx.x, nv = H >> 2;
    float4* row = reinterpret_cast<float4*>(h + (size_t)blockIdx.x * H);
    const float4* drow = delta ? reinterpret_cast<const float4*>(delta + (size_t)blockIdx.x * H) : nullptr;
    const float4* g4 = reinterpret_cast<const float4*>(gamma);
    uint2* out = reinterpret_cast<uint2*>(xn + (size_t)blockIdx.x * H);
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
    const float inv = rsqrtf(tot / (float)H + eps);
    auto put = [&](int i, const float4& t, const float4& gm) {
        const __nv_bfloat162 lo = __floats2bfloat162_rn(t.x * inv * gm.x, t.y * inv * gm.y), hi = __floats2bfloat162_rn(t.z * inv * gm.z, t.w * inv * gm.w);
        out[i] = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    };
#pragma unroll
    for (int j = 0; j < KEEP; ++j)
        if (tid + j * 1024 < nv) put(tid + j * 1024, v[j], g[j]);
    for (int i = tid + KEEP * 1024; i < nv; i += 1024) put(i, row[i], __ldg(g4 + i));
}

// cos and sin of position x frequency for the 64 rotation pairs, once per step and sequence:
// table [rows][64] (cos, sin).  The frequencies theta^(-2i/128) come from the host.
// It does not let its successors start early: what runs after it in the step finds the positions and the caches of all earlier
// steps complete even before its own wait (attn_decode_kernel relies on that).
__global__ void __launch_bounds__(64) rope_table_kernel(const int* __restrict__ pos, const float* __restrict__ inv_freq, float2* __restrict__ table) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    float sn, cs;
    sincosf((float)pos[blockIdx.x] * inv_freq[threadIdx.x], &sn, &cs);
    table[blockIdx.x * 64 + threadIdx.x] = make_float2(cs, sn);
}

// Rotary embedding (halves convention: pairs (i, i + 64)) of one 128-wide head at `src`: the lane's
// eight dimensions 8 * l16 .. 8 * l16 + 7, times `scale`; tab = the sequence's 64 (cos, sin) pairs.
__device__ __forceinline__ void rope8(const float* __restrict__ src, const float2* __restrict__ tab, int l16, float scale, float* out) {
    const int base = 8 * (l16 & 7);   // pair index i = base + j in [0, 64)
    const float4 lo0 = *reinterpret_cast<const float4*>(src + base), lo1 = *reinterpret_cast<const float4*>(src + base + 4);
    const float4 hi0 = *reinterpret_cast<const float4*>(src + 64 + base), hi1 = *reinterpret_cast<const float4*>(src + 64 + base + 4);
    const float lo[8] = {lo0.x, lo0.y, lo0.z, lo0.w, lo1.x, lo1.y, lo1.z, lo1.w};
    const float hi[8] = {hi0.x, hi0.y, hi0.z, hi0.w, hi1.x, hi1.y, hi1.z, hi1.w};
    const float4* t4 = reinterpret_cast<const float4*>(tab + base);   // two (cos, sin) pairs per load
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
        const float4 t = __ldg(t4 + (j >> 1));
        const float ra0 = lo[j] * t.x - hi[j] * t.y, rb0 = hi[j] * t.x + lo[j] * t.y;
        const float ra1 = lo[j + 1] * t.z - hi[j + 1] * t.w, rb1 = hi[j + 1] * t.z + lo[j + 1] * t.w;
        out[j] = (l16 < 8 ? ra0 : rb0) * scale;
        out[j + 1] = (l16 < 8 ? ra1 : rb1) * scale;
    }
}
__device__ __forceinline__ uint4 pack_bf16x8(const float* f) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(f[0], f[1]), b = __floats2bfloat162_rn(f[2], f[3]);
    const __nv_bfloat162 c = __floats2bfloat162_rn(f[4], f[5]), d = __floats2bfloat162_rn(f[6], f[7]);
    return make_uint4(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b), *reinterpret_cast<const uint32_t*>(&c),
                      *reinterpret_cast<const uint32_t*>(&d));
}
constexpr int kMaxSplits = 64;
constexpr int kAttnWarps = 4, kAttnStages = 3;   // rounds of 16 tokens in flight per warp
constexpr int kAttnStageBytes = 2 * 16 * kHeadDim * 2;   // K and V of 16 tokens
// Dynamic shared memory of the attention kernel: the warps' K/V rings (reused afterwards for their results), the rotated queries, the new key and value.
constexpr size_t attn_smem_bytes(int g) { return (size_t)kAttnWarps * kAttnStages * kAttnStageBytes + (size_t)g * kHeadDim * 4 + 2 * kHeadDim * 2; }
__device__ __forceinline__ void cp_async16_zfill(uint32_t smem_dst, const void* gsrc, bool valid) {   // zeros where not valid
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_dst), "l"(gsrc), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// A pair of float32 values as three bf16 pairs whose sum carries 24 bits: t[0] + t[1] + t[2].
__device__ __forceinline__ void split3(float x, float y, uint32_t (&t)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
        t[i] = *reinterpret_cast<const uint32_t*>(&h);
        x -= __low2float(h);
        y -= __high2float(h);
    }
}
constexpr int kPartStride = kHeadDim + 4;   // a split's record per head: 128 output values | max | sum | pad (528 bytes)

// Grouped-query decode attention for one new token per sequence, one launch: rotary embedding,
// cache write, scan and merge.  qkv [rows, (nq + 2 nkv) * 128] float32 is the fused projection;
// the caches are [rows][nkv][max_ctx][128] bf16 for K and for V.
//
// CTA (split, kv head, row) scans its slice of the context for the G = nq / nkv query heads that share
// the KV head; the CTA whose slice holds the new position rotates the new key, rounds key and value to bf16, writes
// them into the caches and puts them in their place in the ring (no other CTA reads that position in this step).
// What earlier steps left in the caches does not hang on the product ahead in the stream: every warp asks for its first rounds
// before the kernel waits for that product.  With the copies after the wait the first of them was the start of the kernel:
// 8 steps of one sequence over a 4096-token context took 16.69 ms in place of 16.45, of 16 sequences 36.84 in place of 36.52.
//
// The scan is bound by the cache bytes as long as the arithmetic stays off the float pipes: with a half-warp per token and
// scalar products it took 30 instructions per 16 bytes (84 us for 16 sequences at a 4096-token context, 3.2 TB/s).  Here a
// warp takes 16 tokens at a time through a private ring of asynchronous copies and multiplies on mma.m16n8k16: scores
// S^T = Q K^T with the query heads in the rows, then O += P V with the scores' accumulators as they are for the A operand.
// The caches are bf16; the float32 queries and probabilities enter as three bf16 terms each (exact to 24 bits), which are the
// spare rows of the 16-row operand: rows 0-3 first terms of up to four heads, 4-7 second, 8-11 third.  Eight heads take a
// second A operand for the third terms.
template <int G>
__global__ void __launch_bounds__(32 * kAttnWarps, 2) attn_decode_kernel(const float* __restrict__ qkv, __nv_bfloat16* kcache, __nv_bfloat16* vcache,
                                                             const int* __restrict__ pos, float* part, unsigned* counters,
                                                             __nv_bfloat16* __restrict__ out, int nq, int nkv, int max_ctx, int nsplit,
                                                             const float2* __restrict__ rope_table) {
    constexpr int SETS = G > 4 ? 2 : 1;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    extern __shared__ __align__(128) unsigned char attn_smem[];
    const int split = blockIdx.x, kvh = blockIdx.y, row = blockIdx.z;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, q = lane >> 2, c = lane & 3, l16 = lane & 15;
    const int p = __ldcg(pos + row), len = p + 1;   // the token written by this step takes part
    const int per = (len + nsplit - 1) / nsplit;
    const int t0 = split * per, t1 = min(len, t0 + per);
    const bool holds = t0 <= p && p < t1;   // this CTA's slice holds the new position (uniform over the CTA)
    __nv_bfloat16* kb = kcache + ((size_t)row * nkv + kvh) * max_ctx * kHeadDim;
    __nv_bfloat16* vb = vcache + ((size_t)row * nkv + kvh) * max_ctx * kHeadDim;
    // Ring of this warp: per stage 16 rows of K, then 16 rows of V, 256 bytes each, 16-byte pieces XORed with the row number.
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(attn_smem) + (uint32_t)(warp * kAttnStages * kAttnStageBytes);
    auto request = [&](int base, int stage) {   // one copy group per round; zeros past the end of the slice and for the new position
        const uint32_t dst = ring + (uint32_t)(stage * kAttnStageBytes);
        const int t = base + 16 * warp + (lane >> 4);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = 2 * i + (lane >> 4);
            const bool in = t + 2 * i < t1 && t + 2 * i < p;
            const size_t off = in ? (size_t)(t + 2 * i) * kHeadDim + 8 * l16 : 0;
            const uint32_t at = dst + (uint32_t)(r * 256 + ((l16 ^ (r & 7)) << 4));
            cp_async16_zfill(at, kb + off, in);
            cp_async16_zfill(at + 4096u, vb + off, in);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
#pragma unroll
    for (int i = 0; i < kAttnStages - 1; ++i) request(t0 + i * 16 * kAttnWarps, i);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const float* qkv_row = qkv + (size_t)row * (nq + 2 * nkv) * kHeadDim;
    const float2* tab = rope_table + (size_t)row * 64;
    // Rotation pair i of the group's queries: thread i, i + 128, ...
    constexpr int QPT = (G * 64 + 32 * kAttnWarps - 1) / (32 * kAttnWarps);
    float q_lo[QPT], q_hi[QPT];
    float2 q_cs[QPT];
#pragma unroll
    for (int j = 0; j < QPT; ++j) {
        const int i = tid + 32 * kAttnWarps * j, g = i >> 6, d = i & 63;
        if (g < G) {
            q_lo[j] = __ldcg(qkv_row + (size_t)(kvh * G + g) * kHeadDim + d);
            q_hi[j] = __ldcg(qkv_row + (size_t)(kvh * G + g) * kHeadDim + 64 + d);
            q_cs[j] = __ldcg(tab + d);
        }
    }
    uint4* fresh = reinterpret_cast<uint4*>(attn_smem + (size_t)kAttnWarps * kAttnStages * kAttnStageBytes + (size_t)G * kHeadDim * 4);   // the new key, the new value
    if (holds && warp == 0) {
        float f[8];
        if (lane < 16) {
            rope8(qkv_row + (size_t)(nq + kvh) * kHeadDim, tab, l16, 1.0f, f);
        } else {
            const float* src = qkv_row + (size_t)(nq + nkv + kvh) * kHeadDim + 8 * l16;
            const float4 a = *reinterpret_cast<const float4*>(src), b = *reinterpret_cast<const float4*>(src + 4);
            f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
        }
        const uint4 v = pack_bf16x8(f);
        *reinterpret_cast<uint4*>((lane < 16 ? kb : vb) + (size_t)p * kHeadDim + 8 * l16) = v;
        fresh[lane] = v;
    }
    // the group's queries, rotated and scaled to log2 units by 1 / sqrt(128) * log2(e)
    float* qs = reinterpret_cast<float*>(attn_smem + (size_t)kAttnWarps * kAttnStages * kAttnStageBytes);
#pragma unroll
    for (int j = 0; j < QPT; ++j) {
        const int i = tid + 32 * kAttnWarps * j, g = i >> 6, d = i & 63;
        if (g < G) {
            constexpr float kScale = 0.08838834764831845f * 1.4426950408889634f;
            qs[g * kHeadDim + d] = (q_lo[j] * q_cs[j].x - q_hi[j] * q_cs[j].y) * kScale;
            qs[g * kHeadDim + 64 + d] = (q_hi[j] * q_cs[j].x + q_lo[j] * q_cs[j].y) * kScale;
        }
    }
    __syncthreads();
    // this lane's rows q and q + 8 of the A operands hold terms of head `h`
    const int h = G > 4 ? q : (q & 3);
    const bool live = h < G;
    auto rows_of = [&](const uint32_t (&t)[3], int set, uint32_t& lo, uint32_t& hi) {   // A registers of rows q and q + 8
        if (G > 4) {
            lo = set ? t[2] : t[0];
            hi = set ? 0u : t[1];
        } else {
            lo = q < 4 ? t[0] : t[1];
            hi = q < 4 ? t[2] : 0u;
        }
    };
    uint32_t qa[SETS][8][4];
#pragma unroll
    for (int kk = 0; kk < 8; ++kk)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const float2 v = live ? *reinterpret_cast<const float2*>(qs + h * kHeadDim + 16 * kk + 8 * half + 2 * c) : make_float2(0.f, 0.f);
            uint32_t t[3];
            split3(v.x, v.y, t);
#pragma unroll
            for (int st = 0; st < SETS; ++st) rows_of(t, st, qa[st][kk][2 * half], qa[st][kk][2 * half + 1]);
        }
    float acc[16][4];   // O: rows q, q + 8 x dimensions 8j + 2c, + 1
#pragma unroll
    for (int j = 0; j < 16; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    float m = -INFINITY, l = 0.f;   // of head h; l over this lane's tokens
    const int kt = (lane >> 4) * 8 + (lane & 7), kc = (lane >> 3) & 1;   // row and piece this lane addresses for K, for V
    const int vt = ((lane >> 3) & 1) * 8 + (lane & 7), vc = lane >> 4;
    int stage = 0, req_stage = kAttnStages - 1;
    for (int base = t0; base < t1; base += 16 * kAttnWarps) {
        request(base + (kAttnStages - 1) * 16 * kAttnWarps, req_stage);   // the stage read in the previous iteration
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kAttnStages - 1) : "memory");
        __syncwarp();
        const int tw = base + 16 * warp;
        if (tw < t1) {
            const uint32_t ks = ring + (uint32_t)(stage * kAttnStageBytes), vs = ks + 4096u;
            if (holds && p < tw + 16) {   // (and p >= tw: the new position is the slice's last) the new key and value in their place
                const uint4 v = fresh[lane];
                const uint32_t r = (uint32_t)(p - tw), at = (lane < 16 ? ks : vs) + r * 256u + (uint32_t)((l16 ^ (int)(r & 7u)) << 4);
                asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(at), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
                __syncwarp();
            }
            float sc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};   // tokens 0-7, 8-15
#pragma unroll
            for (int kk = 0; kk < 8; ++kk) {
                uint32_t kf[4];
                ldsm_x4(ks + (uint32_t)(kt * 256 + (((2 * kk + kc) ^ (kt & 7)) << 4)), kf);
#pragma unroll
                for (int st = 0; st < SETS; ++st) {
                    mma_bf16(sc[0], qa[st][kk], kf[0], kf[1]);
                    mma_bf16(sc[1], qa[st][kk], kf[2], kf[3]);
                }
            }
            float sv[4];   // scores of head h for tokens 2c, 2c + 1, 2c + 8, 2c + 9: the terms' rows added up
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float v = sc[i >> 1][i & 1] + sc[i >> 1][(i & 1) + 2];
                if (G <= 4) v += __shfl_xor_sync(0xffffffffu, v, 16);
                sv[i] = tw + 8 * (i >> 1) + 2 * c + (i & 1) < t1 ? v : -INFINITY;
            }
            float mn = fmaxf(m, fmaxf(fmaxf(sv[0], sv[1]), fmaxf(sv[2], sv[3])));
            mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 1));
            mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 2));
            if (__any_sync(0xffffffffu, mn > m)) {
                const float corr = ex2(m - mn);
                l *= corr;
#pragma unroll
                for (int j = 0; j < 16; ++j) { acc[j][0] *= corr; acc[j][1] *= corr; acc[j][2] *= corr; acc[j][3] *= corr; }
                m = mn;
            }
            float pr[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) { pr[i] = ex2(sv[i] - m); l += pr[i]; }
            uint32_t pa[SETS][4];
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                uint32_t t[3];
                split3(pr[2 * half], pr[2 * half + 1], t);
#pragma unroll
                for (int st = 0; st < SETS; ++st) rows_of(t, st, pa[st][2 * half], pa[st][2 * half + 1]);
            }
#pragma unroll
            for (int jj = 0; jj < 8; ++jj) {
                uint32_t vf[4];
                ldsm_x4_trans(vs + (uint32_t)(vt * 256 + (((2 * jj + vc) ^ (vt & 7)) << 4)), vf);
#pragma unroll
                for (int st = 0; st < SETS; ++st) {
                    mma_bf16(acc[2 * jj], pa[st], vf[0], vf[1]);
                    mma_bf16(acc[2 * jj + 1], pa[st], vf[2], vf[3]);
                }
            }
        }
        __syncwarp();   // every lane has read the stage before it is refilled
        if (++stage == kAttnStages) stage = 0;
        if (++req_stage == kAttnStages) req_stage = 0;
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();   // the rings are done with: their memory now holds the warps' results
    float(*sm_acc)[G][kHeadDim] = reinterpret_cast<float(*)[G][kHeadDim]>(attn_smem);                                // [warps][G][128]
    float(*sm_m)[G] = reinterpret_cast<float(*)[G]>(attn_smem + (size_t)kAttnWarps * G * kHeadDim * 4);              // [warps][G]
    float(*sm_l)[G] = reinterpret_cast<float(*)[G]>(attn_smem + (size_t)kAttnWarps * G * (kHeadDim + 1) * 4);        // [warps][G]
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    const bool owner = q < G && (G > 4 || q < 4);
    if (owner && c == 0) { sm_m[warp][h] = m; sm_l[warp][h] = l; }
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        float x = acc[j][0] + acc[j][2], y = acc[j][1] + acc[j][3];   // the terms' rows
        if (G <= 4) {
            x += __shfl_xor_sync(0xffffffffu, x, 16);
            y += __shfl_xor_sync(0xffffffffu, y, 16);
        }
        if (owner) *reinterpret_cast<float2*>(&sm_acc[warp][h][8 * j + 2 * c]) = make_float2(x, y);
    }
    __syncthreads();
    for (int idx = tid; idx < G * kHeadDim; idx += 32 * kAttnWarps) {
        const int g = idx / kHeadDim, d = idx % kHeadDim;
        float mm = -INFINITY;
#pragma unroll
        for (int w = 0; w < kAttnWarps; ++w) mm = fmaxf(mm, sm_m[w][g]);
        float ll = 0.f, aa = 0.f;
#pragma unroll
        for (int w = 0; w < kAttnWarps; ++w) {
            const float cw = sm_m[w][g] == -INFINITY ? 0.f : ex2(sm_m[w][g] - mm);
            ll += sm_l[w][g] * cw;
            aa += sm_acc[w][g][d] * cw;
        }
        float* dst = part + (((size_t)row * nq + kvh * G + g) * nsplit + split) * kPartStride;
        dst[d] = aa;
        if (d == 0) { dst[kHeadDim] = mm; dst[kHeadDim + 1] = ll; }
    }
    // the last CTA of this (row, kv head) merges the splits: a warp per head, a lane per four dimensions
    __shared__ unsigned s_prev;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_prev = atomicAdd(counters + (size_t)row * nkv + kvh, 1u);
    __syncthreads();
    if (s_prev != (unsigned)(nsplit - 1)) return;
    __threadfence();
    for (int g = threadIdx.x >> 5; g < G; g += 4) {
        const float* src = part + ((size_t)row * nq + kvh * G + g) * nsplit * kPartStride;
        // all loads of up to 32 splits at once, the weights' (nsplit <= 64: two per lane) among them: one trip to L2 each, and
        // a rolled loop's remainder would make one per split
        const bool h0 = lane < nsplit, h1 = lane + 32 < nsplit;
        float4 v[32];
#pragma unroll
        for (int u = 0; u < 32; ++u)
            v[u] = u < nsplit ? __ldcg(reinterpret_cast<const float4*>(src + (size_t)u * kPartStride) + lane) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float2 ml0 = h0 ? __ldcg(reinterpret_cast<const float2*>(src + (size_t)lane * kPartStride + kHeadDim)) : make_float2(-INFINITY, 0.f);
        const float2 ml1 = h1 ? __ldcg(reinterpret_cast<const float2*>(src + (size_t)(lane + 32) * kPartStride + kHeadDim)) : make_float2(-INFINITY, 0.f);
        float mm = fmaxf(ml0.x, ml1.x);
        for (int o = 16; o > 0; o >>= 1) mm = fmaxf(mm, __shfl_xor_sync(0xffffffffu, mm, o));
        const float c0 = ml0.x == -INFINITY ? 0.f : ex2(ml0.x - mm), c1 = ml1.x == -INFINITY ? 0.f : ex2(ml1.x - mm);
        float ll = ml0.y * c0 + ml1.y * c1;
        for (int o = 16; o > 0; o >>= 1) ll += __shfl_xor_sync(0xffffffffu, ll, o);
        float4 aa = make_float4(0.f, 0.f, 0.f, 0.f);
        auto add = [&](float cw) {
#pragma unroll
            for (int u = 0; u < 32; ++u) {
                const float c = __shfl_sync(0xffffffffu, cw, u);
                aa.x += c * v[u].x; aa.y += c * v[u].y; aa.z += c * v[u].z; aa.w += c * v[u].w;
            }
        };
        add(c0);
        if (nsplit > 32) {
#pragma unroll
            for (int u = 0; u < 32; ++u)
                v[u] = u + 32 < nsplit ? __ldcg(reinterpret_cast<const float4*>(src + (size_t)(u + 32) * kPartStride) + lane) : make_float4(0.f, 0.f, 0.f, 0.f);
            add(c1);
        }
        const float inv = 1.0f / ll;
        const __nv_bfloat162 o01 = __floats2bfloat162_rn(aa.x * inv, aa.y * inv), o23 = __floats2bfloat162_rn(aa.z * inv, aa.w * inv);
        *reinterpret_cast<uint2*>(out + ((size_t)row * nq + kvh * G + g) * kHeadDim + 4 * lane) =
            make_uint2(*reinterpret_cast<const uint32_t*>(&o01), *reinterpret_cast<const uint32_t*>(&o23));
    }
    if (threadIdx.x == 0) counters[(size_t)row * nkv + kvh] = 0u;
}

// logits [rows, n] float32 -> (largest value, its index + index_base) per row; ties go to the smaller index.
// Two launches: kArgmaxSlices CTAs per row take the best of a slice each, one warp per row merges them.
constexpr int kArgmaxSlices = 64;
__device__ __forceinline__ void argmax_take(float v, int i, float& bv, int& bi) {
    if (v > bv || (v == bv && i < bi)) { bv = v; bi = i; }
}
__global__ void __launch_bounds__(256) argmax_slices_kernel(const float* __restrict__ logits, int n, float* __restrict__ part_val, int* __restrict__ part_idx) {
    dep_wait();
    __shared__ float sv[8];
    __shared__ int si[8];
    const float* row = logits + (size_t)blockIdx.y * n;
    const int per = (n + kArgmaxSlices - 1) / kArgmaxSlices, i0 = blockIdx.x * per, i1 = min(n, i0 + per);
    float bv = -INFINITY;
    int bi = 0x7FFFFFFF;
#pragma unroll 4
    for (int i = i0 + threadIdx.x; i < i1; i += 256) argmax_take(row[i], i, bv, bi);
    for (int o = 16; o > 0; o >>= 1) argmax_take(__shfl_xor_sync(0xffffffffu, bv, o), __shfl_xor_sync(0xffffffffu, bi, o), bv, bi);
    if ((threadIdx.x & 31) == 0) { sv[threadIdx.x >> 5] = bv; si[threadIdx.x >> 5] = bi; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) argmax_take(sv[w], si[w], bv, bi);
        part_val[blockIdx.y * kArgmaxSlices + blockIdx.x] = bv;
        part_idx[blockIdx.y * kArgmaxSlices + blockIdx.x] = bi;
    }
}
__global__ void __launch_bounds__(32) argmax_merge_kernel(const float* __restrict__ part_val, const int* __restrict__ part_idx, int index_base,
                                                          float* __restrict__ best_val, int* __restrict__ best_idx) {
    dep_wait();
    const int lane = threadIdx.x;
    float bv = -INFINITY;
    int bi = 0x7FFFFFFF;
    for (int j = lane; j < kArgmaxSlices; j += 32) argmax_take(part_val[blockIdx.x * kArgmaxSlices + j], part_idx[blockIdx.x * kArgmaxSlices + j], bv, bi);
    for (int o = 16; o > 0; o >>= 1) argmax_take(__shfl_xor_sync(0xffffffffu, bv, o), __shfl_xor_sync(0xffffffffu, bi, o), bv, bi);
    if (lane == 0) { best_val[blockIdx.x] = bv; best_idx[blockIdx.x] = bi + index_base; }
}

// Vocabulary shards: gathered [world][rows] (value, index as float) -> winning token per row (smaller rank on ties).
__global__ void argmax_pick_kernel(const float* __restrict__ gathered, int world, int rows, int* __restrict__ token) {
    dep_wait();
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= rows) return;
    float bv = -INFINITY;
    int bi = 0;
    for (int w = 0; w < world; ++w) {
        const float v = gathered[((size_t)w * rows + r) * 2], idx = gathered[((size_t)w * rows + r) * 2 + 1];
        if (v > bv) { bv = v; bi = (int)idx; }
    }
    token[r] = bi;
}
// This rank's (value, index) pairs into its slot of a zeroed [world][rows][2] vector (summing the ranks' vectors gathers them).
__global__ void argmax_pack_kernel(const float* __restrict__ val, const int* __restrict__ idx, int rank, int world, int rows, float* __restrict__ out) {
    dep_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= world * rows * 2) return;
    const int w = i / (rows * 2), r = (i / 2) % rows, f = i & 1;
    out[i] = w == rank ? (f ? (float)idx[r] : val[r]) : 0.f;
}

// Embedding rows: h[r, :] = table[ids[r], :] (bf16 table) as float32.
__global__ void embed_rows_kernel(const int* __restrict__ ids, const __nv_bfloat16* __restrict__ table, float* __restrict__ h, int H, int vocab) {
    dep_wait();
    const int r = blockIdx.x;
    const int id = min(max(ids[r], 0), vocab - 1);
    const uint2* src = reinterpret_cast<const uint2*>(table + (size_t)id * H);   // H is a multiple of 8: four bf16 per load
    float4* dst = reinterpret_cast<float4*>(h + (size_t)r * H);
    for (int i = threadIdx.x; i < (H >> 2); i += blockDim.x) {
        const uint2 v = __ldg(src + i);
        dst[i] = make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xFFFF0000u), __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xFFFF0000u));
    }
}

// Seeded synthetic cache contents (a stand-in for the prefill pass): values of unit scale.  Buffer blockIdx.y takes seed +
// blockIdx.y.  One launch for up to 64 buffers: a launch each was 6 us for the 4 us of one sequence's buffer (64 of them 0.47
// ms).  Bound by integer instructions, twelve a value, two in three at half rate.
constexpr int kFillMax = 64;
struct FillArgs {
    uint4* p[kFillMax];
    size_t n8;
    unsigned seed;
};
__global__ void __launch_bounds__(256) fill_cache_kernel(const __grid_constant__ FillArgs a) {   // eight values a thread and turn
    uint4* __restrict__ p = a.p[blockIdx.y];
    const unsigned seed = a.seed + blockIdx.y;
    for (size_t i8 = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i8 < a.n8; i8 += (size_t)gridDim.x * blockDim.x) {
        const size_t i0 = 8 * i8;
        const unsigned first = (unsigned)i0 * 2654435761u, mix = seed ^ (unsigned)(i0 >> 32) * 40503u;
        float f[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            unsigned x = (first + (unsigned)j * 2654435761u) ^ mix;
            x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; x ^= x >> 16;
            // (float)(x & 0xFFFF) - 32768, exactly: the 16 bits under the exponent of 2^23
            f[j] = (__uint_as_float(__byte_perm(x, 0x4B00u, 0x5410)) - 8421376.f) * (1.f / 18918.f);   // uniform, unit variance
        }
        p[i8] = pack_bf16x8(f);
    }
}
__global__ void fill_pos_kernel(int* p, int n, int v) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = v;
}
__global__ void fill_f32_kernel(float* p, size_t n, float v) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) p[i] = v;
}
__global__ void add_one_kernel(int* p, int n) {
    dep_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] += 1;
}

}  // namespace mfqb

using namespace mfqb;

struct DecoderLayer {
    const mfqb_weight *qkv = nullptr, *o = nullptr, *gate_up = nullptr, *down = nullptr;   // borrowed handles
    DevBuf gamma_attn, gamma_ffn;                                                        // [H] float32
    DevBuf kcache, vcache;                                                               // [batch][nkv_local][max_ctx][128] bf16
};

struct mfqb_decoder {
    mfqb_decoder_config cfg{};
    int rank = 0, world = 1, device = 0;
    mfqb_comm* comm = nullptr;       // borrowed; null when world == 1
    int nq = 0, nkv = 0, f = 0, vshard = 0, vbase = 0, sms = 0, attn_per_sm = 4;
    // Single-row steps could run the residual add + RMSNorm inside the q|k|v, gate|up and lm_head products
    // (mfqb_mul_mat_rmsnorm).  Measured on the 8B-shaped model it loses: every CTA of those products repeats the
    // normalisation of the row (2.29 against 2.14 ms per step), so the two-kernel form stays the default.
    bool fused_norm = false;
    std::vector<DecoderLayer> layers;
    const mfqb_weight* lm_head = nullptr;
    const void* embedding = nullptr;   // bf16 [vocab, H] on the device, borrowed
    DevBuf gamma_final;
    // workspaces
    DevBuf h, h2, xn, qkv, attn, attn_count, inv_freq, rope_table, proj, proj_sum, act, logits, part, best_val, best_idx, part_val, part_idx, gathered, gathered_sum, pos;
};

// Context splits of the decode attention.  A CTA costs about as much as 96 tokens of its scan before and after it (queries,
// first copies, merge); the split count with the shortest schedule, in tokens of the longest sequence of CTAs on a slot.
static int attn_splits(const mfqb_decoder* d, int rows, int ctx_bound) {
    const long long slots = (long long)d->attn_per_sm * d->sms, groups = (long long)d->nkv * rows;
    int best = 1;
    long long best_cost = -1;
    for (int n = 1; n <= kMaxSplits; ++n) {
        const long long waves = (groups * n + slots - 1) / slots, cost = waves * ((ctx_bound + n - 1) / n + 96);
        if (best_cost < 0 || cost < best_cost) { best = n; best_cost = cost; }
    }
    return best;
}

// The step's rotation table (cos, sin per sequence and pair), before the first block that uses it.
static void launch_rope_table(mfqb_decoder* d, int rows, cudaStream_t s) {
    launch_dep(rope_table_kernel, dim3(rows), dim3(64), s, static_cast<const int*>(d->pos.p), static_cast<const float*>(d->inv_freq.p),
               static_cast<float2*>(d->rope_table.p));
}

static void check_weight_shape(const mfqb_weight* w, int64_t n, int64_t k, const char* what) {
    mfqb_weight_info info;
    if (mfqb_weight_info_get(w, &info) != MFQB_OK) fail(MFQB_ERR_ARG, "%s: bad weight handle", what);
    if (info.n != n || info.k != k) fail(MFQB_ERR_ARG, "%s must be [%lld, %lld], got [%lld, %lld]", what, (long long)n, (long long)k, (long long)info.n, (long long)info.k);
}

static void launch_fill_f32(void* p, size_t n, float v, cudaStream_t s) {
    fill_f32_kernel<<<(unsigned)std::min<size_t>((n + 255) / 256, 1024), 256, 0, s>>>(static_cast<float*>(p), n, v);
}

// sum over ranks of a float32 vector (in place semantics: out may equal in is not allowed by the collective, hence two buffers)
static const float* rank_sum(mfqb_decoder* d, const float* in, float* out, size_t n, cudaStream_t s) {
    if (d->world == 1) return in;
    const int rc = mfqb_allreduce_f32(d->comm, in, out, n, s);
    if (rc != MFQB_OK) throw Error(rc, mfqb_last_error());
    return out;
}

// Batched steps: residual add, RMSNorm and product with the normalised row going straight into the batched kernel's activation
// layout.  False when this weight or batch has neither of the two kernels: the caller normalises, then multiplies.
static bool norm_mul_mat(mfqb_decoder* d, const mfqb_weight* w, const float* delta, const void* gamma, int rows, void* y, int y_dtype, bool glu, cudaStream_t s) {
    if (rows < 5) return false;
    reserve_fewer_rows(w, rows, glu, s);
    const TileNorm norm{static_cast<float*>(d->h.p), delta, static_cast<const float*>(gamma), d->cfg.rms_eps};
    return launch_rows_product(weight_device_layout(w), nullptr, rows, y, y_dtype, d->device, s, glu, &norm) ||
           launch_tile_product(weight_device_layout(w), nullptr, rows, y, y_dtype, d->device, s, glu, &norm);
}

static void mul_mat(const mfqb_weight* w, const void* x, int m, void* y, cudaStream_t s) {
    const int rc = mfqb_mul_mat(w, x, m, y, MFQB_F32, s);
    if (rc != MFQB_OK) throw Error(rc, mfqb_last_error());
}

// One transformer block on the residual stream d->h for `rows` sequences; `delta` is the previous
// block's (already rank-summed) FFN output still to be added, and on return `*delta_out` is this
// block's: the add is fused into the next RMSNorm.
static const float* layer_forward(mfqb_decoder* d, int li, int rows, const float* delta, cudaStream_t s) {
    DecoderLayer& L = d->layers[li];
    const int H = d->cfg.hidden;
    const int G = d->cfg.n_q_heads / d->cfg.n_kv_heads;
    // One row: the residual add and the normalisation run inside the products that consume them (h + delta goes to
    // h2, h2 + attention output back to h).  Batches: a normalisation kernel, then the batched product.
    bool fused = rows == 1 && d->fused_norm;
    if (fused) {
        const int rc = mfqb_mul_mat_rmsnorm(L.qkv, static_cast<const float*>(d->h.p), delta, static_cast<const float*>(L.gamma_attn.p), d->cfg.rms_eps,
                                            static_cast<float*>(d->h2.p), d->qkv.p, MFQB_F32, 0, s);
        if (rc == MFQB_ERR_UNSUPPORTED) d->fused_norm = fused = false;   // weights this form does not take: the two-kernel form from here on
        else if (rc != MFQB_OK) throw Error(rc, mfqb_last_error());
    }
    if (!fused && !norm_mul_mat(d, L.qkv, delta, L.gamma_attn.p, rows, d->qkv.p, MFQB_F32, false, s)) {
        launch_dep(add_rmsnorm_kernel, dim3(rows), dim3(1024), s, static_cast<float*>(d->h.p), delta, static_cast<const float*>(L.gamma_attn.p),
                   static_cast<__nv_bfloat16*>(d->xn.p), H, d->cfg.rms_eps);
        mul_mat(L.qkv, d->xn.p, rows, d->qkv.p, s);
    }
    const int nsplit = attn_splits(d, rows, d->cfg.max_ctx);
    const dim3 agrid(nsplit, d->nkv, rows);
    auto attn = [&](auto kernel) {
        launch_dep_smem(kernel, agrid, dim3(32 * kAttnWarps), attn_smem_bytes(G), s, static_cast<const float*>(d->qkv.p), static_cast<__nv_bfloat16*>(L.kcache.p),
                   static_cast<__nv_bfloat16*>(L.vcache.p), static_cast<const int*>(d->pos.p), static_cast<float*>(d->part.p),
                   static_cast<unsigned*>(d->attn_count.p), static_cast<__nv_bfloat16*>(d->attn.p), d->nq, d->nkv, d->cfg.max_ctx, nsplit,
                   static_cast<const float2*>(d->rope_table.p));
    };
    switch (G) {
        case 1: attn(attn_decode_kernel<1>); break;
        case 2: attn(attn_decode_kernel<2>); break;
        case 4: attn(attn_decode_kernel<4>); break;
        case 8: attn(attn_decode_kernel<8>); break;
        default: fail(MFQB_ERR_UNSUPPORTED, "query heads per KV head must be 1, 2, 4 or 8, got %d", G);
    }
    // output projection: row-parallel under tensor parallelism
    const float* o_out;
    if (d->world > 1 && rows == 1) {
        const int rc = mfqb_mul_mat_allreduce(L.o, d->attn.p, 1, d->comm, d->proj_sum.p, MFQB_F32, s);
        if (rc != MFQB_OK) throw Error(rc, mfqb_last_error());
        o_out = static_cast<const float*>(d->proj_sum.p);
    } else {
        mul_mat(L.o, d->attn.p, rows, d->proj.p, s);
        o_out = rank_sum(d, static_cast<const float*>(d->proj.p), static_cast<float*>(d->proj_sum.p), (size_t)rows * H, s);
    }
    // gate|up with the activation in the epilogue: the fused weight alternates 16-row blocks of gate and up rows
    if (fused) {
        const int rc = mfqb_mul_mat_rmsnorm(L.gate_up, static_cast<const float*>(d->h2.p), o_out, static_cast<const float*>(L.gamma_ffn.p), d->cfg.rms_eps,
                                            static_cast<float*>(d->h.p), d->act.p, MFQB_BF16, 1, s);
        if (rc != MFQB_OK) throw Error(rc, mfqb_last_error());
    } else if (!norm_mul_mat(d, L.gate_up, o_out, L.gamma_ffn.p, rows, d->act.p, MFQB_BF16, true, s)) {
        launch_dep(add_rmsnorm_kernel, dim3(rows), dim3(1024), s, static_cast<float*>(d->h.p), o_out, static_cast<const float*>(L.gamma_ffn.p),
                   static_cast<__nv_bfloat16*>(d->xn.p), H, d->cfg.rms_eps);
        const int rc = mfqb_mul_mat_glu(L.gate_up, d->xn.p, rows, d->act.p, MFQB_BF16, s);
        if (rc != MFQB_OK) throw Error(rc, mfqb_last_error());
    }
    if (d->world > 1 && rows == 1) {
        const int rc = mfqb_mul_mat_allreduce(L.down, d->act.p, 1, d->comm, d->proj_sum.p, MFQB_F32, s);
        if (rc != MFQB_OK) throw Error(rc, mfqb_last_error());
        return static_cast<const float*>(d->proj_sum.p);
    }
    mul_mat(L.down, d->act.p, rows, d->proj.p, s);
    return rank_sum(d, static_cast<const float*>(d->proj.p), static_cast<float*>(d->proj_sum.p), (size_t)rows * H, s);
}

extern "C" {
#pragma GCC visibility push(default)

int mfqb_decoder_create(const mfqb_decoder_config* cfg, int rank, int world, mfqb_comm* comm, int device, mfqb_decoder** out) {
    return guarded([&] {
        if (!cfg || !out) fail(MFQB_ERR_ARG, "mfqb_decoder_create: null argument");
        if (world < 1 || rank < 0 || rank >= world) fail(MFQB_ERR_ARG, "mfqb_decoder_create: rank %d / world %d", rank, world);
        if (world > 1 && !comm) fail(MFQB_ERR_ARG, "mfqb_decoder_create: tensor parallelism needs a communicator");
        if (cfg->head_dim != kHeadDim) fail(MFQB_ERR_UNSUPPORTED, "head_dim must be %d", kHeadDim);
        if (cfg->n_q_heads % cfg->n_kv_heads || cfg->n_kv_heads % world || cfg->ffn % world || cfg->layers < 1 || cfg->max_batch < 1 ||
            cfg->hidden != cfg->n_q_heads * kHeadDim || cfg->hidden % 8 || (cfg->ffn / world) % 16)
            fail(MFQB_ERR_ARG, "mfqb_decoder_create: head counts, FFN width and hidden size must divide over %d ranks (hidden = heads x 128)", world);
        auto d = std::make_unique<mfqb_decoder>();
        d->cfg = *cfg;
        d->rank = rank;
        d->world = world;
        d->comm = world > 1 ? comm : nullptr;
        d->device = device;
        d->sms = device_sm_count(device);
        d->nq = cfg->n_q_heads / world;
        d->nkv = cfg->n_kv_heads / world;
        d->f = cfg->ffn / world;
        // vocabulary rows in shards of whole 16-row blocks
        const int per = ((cfg->vocab + world - 1) / world + 15) / 16 * 16;
        d->vbase = std::min(cfg->vocab, rank * per);
        d->vshard = std::max(0, std::min(cfg->vocab, d->vbase + per) - d->vbase);
        DeviceGuard guard(device);
        const size_t B = cfg->max_batch, H = cfg->hidden;
        d->layers.resize(cfg->layers);
        for (auto& L : d->layers) {
            L.gamma_attn.alloc(H * 4);
            L.gamma_ffn.alloc(H * 4);
            launch_fill_f32(L.gamma_attn.p, H, 1.f, nullptr);
            launch_fill_f32(L.gamma_ffn.p, H, 1.f, nullptr);
            const size_t cache = B * d->nkv * cfg->max_ctx * kHeadDim * 2;
            L.kcache.alloc(cache);
            L.vcache.alloc(cache);
        }
        d->gamma_final.alloc(H * 4);
        launch_fill_f32(d->gamma_final.p, H, 1.f, nullptr);
        d->h.alloc(B * H * 4);
        d->h2.alloc(B * H * 4);
        d->xn.alloc(B * H * 2);
        d->qkv.alloc(B * (d->nq + 2 * d->nkv) * kHeadDim * 4);
        {   // rotary frequencies theta^(-2i/128), i = 0..63
            float freq[kHeadDim / 2];
            for (int i = 0; i < kHeadDim / 2; ++i) freq[i] = (float)std::pow((double)cfg->rope_theta, -2.0 * i / kHeadDim);
            d->inv_freq.alloc(sizeof(freq));
            MFQB_CUDA(cudaMemcpy(d->inv_freq.p, freq, sizeof(freq), cudaMemcpyHostToDevice));
        }
        {   // resident CTAs per SM of the attention kernel this model uses
            int per_sm = 0;
            cudaError_t e = cudaErrorInvalidValue;
            switch (cfg->n_q_heads / cfg->n_kv_heads) {
                case 1:
                    MFQB_CUDA(cudaFuncSetAttribute(attn_decode_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)attn_smem_bytes(1)));
                    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, attn_decode_kernel<1>, 32 * kAttnWarps, attn_smem_bytes(1));
                    break;
                case 2:
                    MFQB_CUDA(cudaFuncSetAttribute(attn_decode_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)attn_smem_bytes(2)));
                    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, attn_decode_kernel<2>, 32 * kAttnWarps, attn_smem_bytes(2));
                    break;
                case 4:
                    MFQB_CUDA(cudaFuncSetAttribute(attn_decode_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)attn_smem_bytes(4)));
                    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, attn_decode_kernel<4>, 32 * kAttnWarps, attn_smem_bytes(4));
                    break;
                case 8:
                    MFQB_CUDA(cudaFuncSetAttribute(attn_decode_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)attn_smem_bytes(8)));
                    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, attn_decode_kernel<8>, 32 * kAttnWarps, attn_smem_bytes(8));
                    break;
                default: fail(MFQB_ERR_UNSUPPORTED, "query heads per KV head must be 1, 2, 4 or 8, got %d", cfg->n_q_heads / cfg->n_kv_heads);
            }
            MFQB_CUDA(e);
            d->attn_per_sm = std::max(1, per_sm);
        }
        d->attn_count.alloc(B * d->nkv * 4);
        MFQB_CUDA(cudaMemset(d->attn_count.p, 0, B * d->nkv * 4));
        d->attn.alloc(B * d->nq * kHeadDim * 2);
        d->proj.alloc(B * H * 4);
        d->proj_sum.alloc(B * H * 4);
        d->act.alloc(B * d->f * 2);
        d->logits.alloc(B * std::max(d->vshard, 1) * 4);
        d->part.alloc(B * d->nq * kMaxSplits * kPartStride * 4);
        d->rope_table.alloc(B * 64 * sizeof(float2));
        d->best_val.alloc(B * 4);
        d->part_val.alloc(B * kArgmaxSlices * 4);
        d->part_idx.alloc(B * kArgmaxSlices * 4);
        d->best_idx.alloc(B * 4);
        d->gathered.alloc((size_t)world * B * 2 * 4);
        d->gathered_sum.alloc((size_t)world * B * 2 * 4);
        d->pos.alloc(B * 4);
        MFQB_CUDA(cudaMemset(d->pos.p, 0, B * 4));
        MFQB_CUDA(cudaDeviceSynchronize());
        *out = d.release();
    });
}

int mfqb_decoder_set_layer(mfqb_decoder* d, int layer, const mfqb_weight* qkv, const mfqb_weight* o, const mfqb_weight* gate_up,
                           const mfqb_weight* down) {
    return guarded([&] {
        if (!d || !qkv || !o || !gate_up || !down || layer < 0 || layer >= d->cfg.layers) fail(MFQB_ERR_ARG, "mfqb_decoder_set_layer: bad argument");
        const int64_t H = d->cfg.hidden;
        check_weight_shape(qkv, (int64_t)(d->nq + 2 * d->nkv) * kHeadDim, H, "qkv (query | key | value rows of this rank)");
        check_weight_shape(o, H, (int64_t)d->nq * kHeadDim, "o_proj (input slice of this rank)");
        check_weight_shape(gate_up, 2 * (int64_t)d->f, H, "gate_up (gate rows, then up rows of this rank)");
        check_weight_shape(down, H, d->f, "down_proj (input slice of this rank)");
        DecoderLayer& L = d->layers[layer];
        L.qkv = qkv;
        L.o = o;
        L.gate_up = gate_up;
        L.down = down;
    });
}

int mfqb_decoder_set_head(mfqb_decoder* d, const mfqb_weight* lm_head, const void* embedding_bf16) {
    return guarded([&] {
        if (!d || !lm_head || !embedding_bf16) fail(MFQB_ERR_ARG, "mfqb_decoder_set_head: null argument");
        check_weight_shape(lm_head, d->vshard, d->cfg.hidden, "lm_head (vocabulary rows of this rank)");
        d->lm_head = lm_head;
        d->embedding = embedding_bf16;
    });
}

int mfqb_decoder_vocab_shard(const mfqb_decoder* d, int* begin, int* rows) {
    return guarded([&] {
        if (!d || !begin || !rows) fail(MFQB_ERR_ARG, "mfqb_decoder_vocab_shard: null argument");
        *begin = d->vbase;
        *rows = d->vshard;
    });
}

int mfqb_decoder_fill_cache(mfqb_decoder* d, int ctx_len, unsigned seed, mfqb_stream_t stream) {
    return guarded([&] {
        if (!d || ctx_len < 0 || ctx_len >= d->cfg.max_ctx) fail(MFQB_ERR_ARG, "mfqb_decoder_fill_cache: context length must be in [0, max_ctx)");
        DeviceGuard guard(d->device);
        FillArgs a{};
        a.n8 = d->layers[0].kcache.bytes / 16;   // rows are 128 values; all caches are of one size
        const unsigned grid = (unsigned)std::min<size_t>((a.n8 + 255) / 256, 8 * (size_t)d->sms);
        for (size_t done = 0; done < 2 * d->layers.size(); done += kFillMax) {
            const int count = (int)std::min<size_t>(kFillMax, 2 * d->layers.size() - done);
            for (int i = 0; i < count; ++i) {
                const DecoderLayer& L = d->layers[(done + i) / 2];
                a.p[i] = static_cast<uint4*>((done + i) % 2 ? L.vcache.p : L.kcache.p);
            }
            a.seed = seed + (unsigned)done;
            fill_cache_kernel<<<dim3(grid, (unsigned)count), 256, 0, stream>>>(a);
        }
        fill_pos_kernel<<<(d->cfg.max_batch + 127) / 128, 128, 0, stream>>>(static_cast<int*>(d->pos.p), d->cfg.max_batch, ctx_len);
        MFQB_CUDA(cudaGetLastError());
    });
}

int mfqb_decoder_step(mfqb_decoder* d, const int32_t* ids_in, int batch, int32_t* ids_out, mfqb_stream_t stream) {
    return guarded([&] {
        if (!d || !ids_in || !ids_out) fail(MFQB_ERR_ARG, "mfqb_decoder_step: null argument");
        if (batch < 1 || batch > d->cfg.max_batch) fail(MFQB_ERR_ARG, "mfqb_decoder_step: batch %d outside [1, %d]", batch, d->cfg.max_batch);
        if (!d->lm_head || !d->embedding) fail(MFQB_ERR_ARG, "mfqb_decoder_step: head weights are not set");
        for (const auto& L : d->layers)
            if (!L.qkv) fail(MFQB_ERR_ARG, "mfqb_decoder_step: a layer has no weights");
        DeviceGuard guard(d->device);
        cudaStream_t s = stream;
        const int H = d->cfg.hidden;
        launch_dep(embed_rows_kernel, dim3(batch), dim3(1024), s, static_cast<const int*>(ids_in), static_cast<const __nv_bfloat16*>(d->embedding),
                   static_cast<float*>(d->h.p), H, d->cfg.vocab);
        launch_rope_table(d, batch, s);
        const float* delta = nullptr;
        for (int li = 0; li < d->cfg.layers; ++li) delta = layer_forward(d, li, batch, delta, s);
        bool fused_head = batch == 1 && d->fused_norm;
        if (fused_head) {
            const int rc = mfqb_mul_mat_rmsnorm(d->lm_head, static_cast<const float*>(d->h.p), delta, static_cast<const float*>(d->gamma_final.p),
                                                d->cfg.rms_eps, nullptr, d->logits.p, MFQB_F32, 0, s);
            if (rc == MFQB_ERR_UNSUPPORTED) fused_head = false;
            else if (rc != MFQB_OK) throw Error(rc, mfqb_last_error());
        }
        if (!fused_head && !norm_mul_mat(d, d->lm_head, delta, d->gamma_final.p, batch, d->logits.p, MFQB_F32, false, s)) {
            launch_dep(add_rmsnorm_kernel, dim3(batch), dim3(1024), s, static_cast<float*>(d->h.p), delta, static_cast<const float*>(d->gamma_final.p),
                       static_cast<__nv_bfloat16*>(d->xn.p), H, d->cfg.rms_eps);
            mul_mat(d->lm_head, d->xn.p, batch, d->logits.p, s);
        }
        launch_dep(argmax_slices_kernel, dim3(kArgmaxSlices, batch), dim3(256), s, static_cast<const float*>(d->logits.p), d->vshard,
                   static_cast<float*>(d->part_val.p), static_cast<int*>(d->part_idx.p));
        launch_dep(argmax_merge_kernel, dim3(batch), dim3(32), s, static_cast<const float*>(d->part_val.p), static_cast<const int*>(d->part_idx.p),
                   d->vbase, static_cast<float*>(d->best_val.p), static_cast<int*>(d->best_idx.p));
        if (d->world == 1) {
            MFQB_CUDA(cudaMemcpyAsync(ids_out, d->best_idx.p, (size_t)batch * 4, cudaMemcpyDeviceToDevice, s));
        } else {
            const int n = d->world * batch * 2;
            launch_dep(argmax_pack_kernel, dim3((n + 255) / 256), dim3(256), s, static_cast<const float*>(d->best_val.p),
                       static_cast<const int*>(d->best_idx.p), d->rank, d->world, batch, static_cast<float*>(d->gathered.p));
            const float* g = rank_sum(d, static_cast<const float*>(d->gathered.p), static_cast<float*>(d->gathered_sum.p), (size_t)n, s);
            launch_dep(argmax_pick_kernel, dim3((batch + 127) / 128), dim3(128), s, g, d->world, batch, static_cast<int*>(ids_out));
        }
        launch_dep(add_one_kernel, dim3((batch + 127) / 128), dim3(128), s, static_cast<int*>(d->pos.p), batch);
    });
}

// One block only, for parity checks: h_in [rows, H] float32 -> h_out = the residual stream after
// block `layer` (attention and FFN added), computed at the cache positions currently set.
int mfqb_decoder_layer(mfqb_decoder* d, int layer, const float* h_in, int rows, float* h_out, mfqb_stream_t stream) {
    return guarded([&] {
        if (!d || !h_in || !h_out || layer < 0 || layer >= d->cfg.layers || rows < 1 || rows > d->cfg.max_batch)
            fail(MFQB_ERR_ARG, "mfqb_decoder_layer: bad argument");
        DeviceGuard guard(d->device);
        const size_t bytes = (size_t)rows * d->cfg.hidden * 4;
        MFQB_CUDA(cudaMemcpyAsync(d->h.p, h_in, bytes, cudaMemcpyDeviceToDevice, stream));
        launch_rope_table(d, rows, stream);
        const float* delta = layer_forward(d, layer, rows, nullptr, stream);
        // fold the FFN output in with a norm whose bf16 output is discarded
        launch_dep(add_rmsnorm_kernel, dim3(rows), dim3(1024), stream, static_cast<float*>(d->h.p), delta, static_cast<const float*>(d->gamma_final.p),
                   static_cast<__nv_bfloat16*>(d->xn.p), d->cfg.hidden, d->cfg.rms_eps);
        MFQB_CUDA(cudaMemcpyAsync(h_out, d->h.p, bytes, cudaMemcpyDeviceToDevice, stream));
    });
}

// Copies the logits of the last step, this rank's vocabulary rows: out [rows, shard rows] float32.
int mfqb_decoder_read_logits(const mfqb_decoder* d, int rows, float* out, mfqb_stream_t stream) {
    return guarded([&] {
        if (!d || !out || rows < 1 || rows > d->cfg.max_batch) fail(MFQB_ERR_ARG, "mfqb_decoder_read_logits: bad argument");
        DeviceGuard guard(d->device);
        MFQB_CUDA(cudaMemcpyAsync(out, d->logits.p, (size_t)rows * d->vshard * 4, cudaMemcpyDeviceToDevice, stream));
    });
}

// Reads back one layer's cache rows [nkv_local][ctx][128] of sequence `row` (bf16), for parity checks.
int mfqb_decoder_read_cache(const mfqb_decoder* d, int layer, int row, int which, int ctx, void* out_bf16, mfqb_stream_t stream) {
    return guarded([&] {
        if (!d || !out_bf16 || layer < 0 || layer >= d->cfg.layers || row < 0 || row >= d->cfg.max_batch || ctx < 0 || ctx > d->cfg.max_ctx)
            fail(MFQB_ERR_ARG, "mfqb_decoder_read_cache: bad argument");
        DeviceGuard guard(d->device);
        const DecoderLayer& L = d->layers[layer];
        const char* base = static_cast<const char*>(which ? L.vcache.p : L.kcache.p);
        for (int hh = 0; hh < d->nkv; ++hh)
            MFQB_CUDA(cudaMemcpyAsync(static_cast<char*>(out_bf16) + (size_t)hh * ctx * kHeadDim * 2,
                                      base + (((size_t)row * d->nkv + hh) * d->cfg.max_ctx) * kHeadDim * 2, (size_t)ctx * kHeadDim * 2,
                                      cudaMemcpyDeviceToDevice, stream));
    });
}

int mfqb_decoder_free(mfqb_decoder* d) {
    return guarded([&] {
        if (!d) return;
        DeviceGuard guard(d->device);
        delete d;
    });
}

#pragma GCC visibility pop
}  // extern "C"
