// Byte-lane NINT: decoder kernel and the launch planning of the GEMV kernels.
#include <algorithm>
#include <mutex>
#include <type_traits>

#include "common.h"
#include "cuda_util.h"
#include "nint_gemv_bl_launch.cuh"

namespace mfqb {

// ---- reference decoder on the GPU -----------------------------------------------------------
// One thread per (row, group, quad of four slots): reads its codes and the two scale bytes
// through the same accessors as the GEMV and writes w = fl(fl(d*q) - m), d = fl(ns*ss),
// m = fl(nm*sm): three separately rounded float32 operations, as the reference decoder does
// (mfq/quantize/nint_quant.py:896-908).
template <int BITS>
__global__ void nint_bl_dequant_kernel(const NintDevB w, void* out, int out_dtype) {
    using BU = ByteUnit<BITS>;
    const int quads = 2 * w.t8;
    const size_t total = (size_t)w.n * w.ng * quads;
    for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (size_t)gridDim.x * blockDim.x) {
        const int j = (int)(idx % quads);
        const size_t rg = idx / quads;
        const int grp = (int)(rg % w.ng), row = (int)(rg / w.ng);
        if (4 * j >= w.gs) continue;
        const int rb = row >> 4, q = row & 7, hi = (row >> 3) & 1, ch = grp / kChunkGroupsB, g = grp % kChunkGroupsB;
        const int f = g >> 2, o = g & 3;
        const int lane = 4 * q + 2 * (o & 1) + (j & 1);
        const int reg = (f * w.t8 + (j >> 1)) * 4 + 2 * (o >> 1) + hi;
        const uint32_t* rec = w.items + ((size_t)rb * w.nchunks + ch) * w.rec_words;
        uint32_t uw[BU::U];
#pragma unroll
        for (int u = 0; u < BU::U; ++u) uw[u] = rec[((reg / BU::NP) * BU::U + u) * 32 + lane];
        const uint32_t codes = BU::at(uw, reg % BU::NP);
        const int slane = 4 * q + (g >> 1), sbyte = 8 * (2 * hi + (g & 1));
        const float ss = (float)((rec[w.wc * 32 + slane] >> sbyte) & 0xFF), sm = (float)((rec[(w.wc + 1) * 32 + slane] >> sbyte) & 0xFF);
        const uint32_t an = w.anchors[row];
        const float2 nsm = __half22float2(*reinterpret_cast<const __half2*>(&an));
        const float d = __fmul_rn(nsm.x, ss), m = __fmul_rn(nsm.y, sm);
        const int k0 = grp * w.gs + 4 * j;
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = __fsub_rn(__fmul_rn(d, (float)((codes >> (8 * e)) & 0xFF)), m);
        const int live = min(4, min(w.gs - 4 * j, w.k - k0));
        if (live > 0) store_quad(out, out_dtype, (size_t)row * w.k + k0, v, live);
    }
}

void launch_nint_bl_dequant(const NintDevB& w, void* out, int out_dtype, cudaStream_t s) {
    const size_t total = (size_t)w.n * w.ng * 2 * w.t8;
    const int block = 256;
    const int grid = (int)std::min<size_t>((total + block - 1) / block, 148 * 32);
    switch (w.bits) {
        case 2: nint_bl_dequant_kernel<2><<<grid, block, 0, s>>>(w, out, out_dtype); break;
        case 3: nint_bl_dequant_kernel<3><<<grid, block, 0, s>>>(w, out, out_dtype); break;
        case 4: nint_bl_dequant_kernel<4><<<grid, block, 0, s>>>(w, out, out_dtype); break;
        case 5: nint_bl_dequant_kernel<5><<<grid, block, 0, s>>>(w, out, out_dtype); break;
        case 6: nint_bl_dequant_kernel<6><<<grid, block, 0, s>>>(w, out, out_dtype); break;
        case 8: nint_bl_dequant_kernel<8><<<grid, block, 0, s>>>(w, out, out_dtype); break;
        default: fail(MFQB_ERR_UNSUPPORTED, "NINT%d has no kernel", w.bits);
    }
    MFQB_CUDA(cudaGetLastError());
}

bool nint_bl_supported(int bits, int gs) {
    const int t8 = (gs + 7) / 8;
    return gs >= 8 && gs <= 64 && nint_bl_in_catalog(bits, t8);
}

// ---- GEMV launch planning ---------------------------------------------------------------------
cudaError_t launch_gemv_bl_nvq(const GemvArgsB& a, const GemvPlanB& p, cudaStream_t stream);

static void dispatch(const GemvArgsB& a, const GemvPlanB& p, cudaStream_t s, const char* what) {
    cudaError_t e;
    switch (a.w.bits) {
        case 0: e = launch_gemv_bl_nvq(a, p, s); break;   // lattice records
        case 2: e = launch_gemv_bl_bits<2>(a, p, s); break;
        case 3: e = launch_gemv_bl_bits<3>(a, p, s); break;
        case 4: e = launch_gemv_bl_bits<4>(a, p, s); break;
        case 5: e = launch_gemv_bl_bits<5>(a, p, s); break;
        case 6: e = launch_gemv_bl_bits<6>(a, p, s); break;
        case 8: e = launch_gemv_bl_bits<8>(a, p, s); break;
        default: fail(MFQB_ERR_UNSUPPORTED, "NINT%d has no kernel", a.w.bits);
    }
    if (e != cudaSuccess)
        fail(MFQB_ERR_CUDA, "%s%d gs=%d %s launch: %s", a.w.bits ? "NINT" : "NVQ index bits ", a.w.bits ? a.w.bits : a.w.index_bits, a.w.gs, what,
             cudaGetErrorString(e));
}

constexpr size_t kGemvSmemLimit = 200 * 1024;

// Shared-memory tables of the record's codec (lattice records: signed table + state scales).
static size_t codec_ctx_bytes(const NintDevB& w) { return w.table ? (size_t)w.table_words * 4 + 64 : 0; }
// CTAs of `smem` bytes each that fit an SM, at most `cap`.
static int ctas_per_sm(size_t smem, int cap) { return std::max(1, std::min(cap, (int)((220 * 1024) / (smem + 1024)))); }

// Per-warp copies of the partial sums while they stay small; shared copy with atomics beyond.
static bool gemv1_private_sums(int rb_per_cta) { return rb_per_cta <= 8; }
static size_t gemv1_smem(const NintDevB& w, int rb_per_cta, int warps) {
    const int copies = gemv1_private_sums(rb_per_cta) ? warps : 1;
    return codec_ctx_bytes(w) + (size_t)(copies + 1) * rb_per_cta * 16 * 4 + (size_t)warps * gemv1_bl_stages(w.rec_words) * w.rec_words * 4;
}
// Warps per CTA of the single-row kernel: each warp owns whole chunks of K, so 8 to 12 warps are
// chosen to make the largest number of chunks per warp as small as possible (wide records and the
// larger lattice codebooks stay at 8: their kernels are built for 256 threads).
static int gemv1_warps(const NintDevB& w) {
    if ((w.table && w.index_bits != 8) || w.wc > 24) return 8;
    int best = 8;
    for (int n = 9; n <= 12; ++n)
        if ((w.nchunks + n - 1) / n < (w.nchunks + best - 1) / best) best = n;
    return best;
}
static size_t gemvn_smem(const NintDevB& w, int rb_per_cta, int passes) {
    const int mb = 2 * passes;
    return codec_ctx_bytes(w) + (size_t)(mb + 1) * rb_per_cta * 16 * 4 + (size_t)8 * 2 * mb * gemvn_bl_row_bytes(w.t8) +
           (size_t)8 * gemvn_bl_stages(w.rec_words, passes) * w.rec_words * 4;
}

// Bytes of the quantised planes of `rows` activation rows for this weight.
size_t nint_bl_planes_bytes(const NintDevB& w, int rows) {
    return (size_t)rows * w.nchunks * kChunkGroupsB * (gemv1_bl_qstride(w.t8) + 1) * 8;
}

// Quantises x [rows, k] (bf16, or float32 when x_f32) into `planes` (nint_bl_planes_bytes): xq for all rows, then gtab.
void launch_x_planes(const NintDevB& w, const void* x, int rows, void* planes, const uint2** xq_g, const float2** gtab_g, cudaStream_t s,
                     bool x_f32) {
    const int ngp = w.nchunks * kChunkGroupsB, qs = gemv1_bl_qstride(w.t8);
    uint2* xq = static_cast<uint2*>(planes);
    float2* gtab = reinterpret_cast<float2*>(xq + (size_t)rows * ngp * qs);
    *xq_g = xq;
    *gtab_g = gtab;
    // 64 groups per CTA: one pass of its 256 threads (four threads per group)
    const dim3 grid((unsigned)((ngp + 63) / 64), (unsigned)rows);
    auto go = [&](auto t8) {
        constexpr int T = decltype(t8)::value;
        if (x_f32) x_planes_kernel<T, float><<<grid, 256, 0, s>>>(static_cast<const float*>(x), w.k, w.gs, ngp, 64, xq, gtab);
        else x_planes_kernel<T, __nv_bfloat16><<<grid, 256, 0, s>>>(static_cast<const __nv_bfloat16*>(x), w.k, w.gs, ngp, 64, xq, gtab);
    };
    switch (w.t8) {
        case 2: go(std::integral_constant<int, 2>{}); break;
        case 3: go(std::integral_constant<int, 3>{}); break;
        case 4: go(std::integral_constant<int, 4>{}); break;
        case 5: go(std::integral_constant<int, 5>{}); break;
        case 6: go(std::integral_constant<int, 6>{}); break;
        case 8: go(std::integral_constant<int, 8>{}); break;
        default: fail(MFQB_ERR_UNSUPPORTED, "group size %d has no kernel", w.gs);
    }
    MFQB_CUDA(cudaGetLastError());
}

// Library scratch for the planes of a plain batched product (per device, grow-only).
static GrowOnlyScratch g_planes;
static void* planes_scratch(int device, size_t bytes, cudaStream_t s) { return g_planes.get(device, bytes, s, "mfqb_mul_mat (quantised activation planes)"); }
// Room for the batches that the tile kernel leaves to the integer one (up to four rows).
void reserve_planes(const NintDevB& w, int device, cudaStream_t s) { g_planes.reserve(device, nint_bl_planes_bytes(w, 4), s, "mfqb_mul_mat (quantised activation planes)"); }

static int passes_for(int m) { return m <= 2 ? 1 : (m <= 4 ? 2 : 4); }

// Largest number of two-row passes (4, 2 or 1) whose plane buffers and record rings fit one CTA.
int nint_bl_max_passes(const NintDevB& w) {
    for (int p = 4; p > 1; p /= 2)
        if (gemvn_smem(w, 2, p) <= kGemvSmemLimit) return p;
    return 1;
}

// y[m, n] = x[m, k] * W^T for m <= 8 (the caller loops larger batches).  swiglu (m = 1 only): x is the
// float32 gate|up row [2k] and the product is taken with up * silu(gate).  glu (m = 1 only): the weight's
// 16-row blocks alternate gate and up rows and y [n / 2] receives up * silu(gate).
void launch_bl_gemv(const NintDevB& w, const void* x, int m, void* y, int y_dtype, int ldy, int device, cudaStream_t s, bool swiglu, bool glu) {
    GemvArgsB a{};
    a.w = w;
    a.x = static_cast<const __nv_bfloat16*>(x);
    a.y = y;
    a.m = m;
    a.ldy = ldy;
    a.y_dtype = y_dtype;
    GemvPlanB p;
    const int sms = device_sm_count(device);
    if (m == 1) {
        // three CTAs per SM, all resident at once; row-blocks are split evenly inside the kernel
        const int warps = gemv1_warps(w);
        p.threads = warps * 32;
        p.grid = std::min(w.nrb, ctas_per_sm(gemv1_smem(w, 1, warps), warps > 8 ? 2 : 3) * sms);
        a.rb_per_cta = (w.nrb + p.grid - 1) / p.grid;
        if (glu) {   // (gate, up) pairs of row-blocks stay together
            if ((w.nrb & 1) || (w.n & 31)) fail(MFQB_ERR_ARG, "gated product: the weight needs whole (gate, up) pairs of 16-row blocks, n = %d", w.n);
            p.grid = std::min(w.nrb / 2, p.grid);
            a.rb_per_cta = 2 * ((w.nrb / 2 + p.grid - 1) / p.grid);
            a.glu = 1;
        }
        a.private_sums = gemv1_private_sums(a.rb_per_cta);
        p.smem = gemv1_smem(w, a.rb_per_cta, warps);
        if (swiglu) {
            p.passes = -2;
            a.x_mode = 2;
        }
    } else {
        if (swiglu || glu) fail(MFQB_ERR_ARG, "the fused activation belongs to the single-row kernel");
        const int max_rows = 2 * nint_bl_max_passes(w);
        if (m > max_rows) {   // wide records: the batch goes through in several launches
            const size_t ysz = y_dtype == MFQB_F32 ? 4 : 2;
            for (int m0 = 0; m0 < m; m0 += max_rows)
                launch_bl_gemv(w, static_cast<const char*>(x) + (size_t)m0 * w.k * 2, std::min(max_rows, m - m0),
                               static_cast<char*>(y) + (size_t)m0 * ldy * ysz, y_dtype, ldy, device, s, false, false);
            return;
        }
        launch_x_planes(w, x, m, planes_scratch(device, nint_bl_planes_bytes(w, m), s), &a.xq_g, &a.gtab_g, s, false);
        p.passes = passes_for(m);
        // at least two row-blocks per CTA where the matrix allows: a chunk's planes then serve several items
        const int cap = ctas_per_sm(gemvn_smem(w, 2, p.passes), p.passes == 4 ? 2 : 3) * sms;
        p.grid = std::max(1, std::min(w.nrb >= 2 * sms ? w.nrb / 2 : w.nrb, cap));
        a.rb_per_cta = (w.nrb + p.grid - 1) / p.grid;
        p.smem = gemvn_smem(w, a.rb_per_cta, p.passes);
        if (p.smem > kGemvSmemLimit) fail(MFQB_ERR_UNSUPPORTED, "batched product: %d row-blocks per CTA do not fit shared memory", a.rb_per_cta);
    }
    dispatch(a, p, s, "GEMV");
}

// Single-row product on the residual row with the add + RMSNorm fused in (GemvArgsB::norm_*): y = W . norm(h + delta),
// or the gated form of it (glu).  The normalised row lives in shared memory behind the rings.
void launch_bl_gemv_norm(const NintDevB& w, const float* h, const float* delta, const float* gamma, float eps, float* h_out, void* y, int y_dtype,
                         bool glu, int device, cudaStream_t s) {
    if (w.k % 4) fail(MFQB_ERR_ARG, "fused normalisation needs a row length that is a multiple of 4, got %d", w.k);
    GemvArgsB a{};
    a.w = w;
    a.x = reinterpret_cast<const __nv_bfloat16*>(h);
    a.y = y;
    a.m = 1;
    a.ldy = w.n;
    a.y_dtype = y_dtype;
    a.x_mode = 3;
    a.norm_delta = delta;
    a.norm_gamma = gamma;
    a.norm_eps = eps;
    a.norm_h_out = h_out;
    GemvPlanB p;
    const int warps = gemv1_warps(w), sms = device_sm_count(device);
    const size_t row_bytes = (size_t)w.k * 4;
    p.threads = warps * 32;
    p.passes = -4;
    p.grid = std::min(w.nrb, ctas_per_sm(gemv1_smem(w, 1, warps) + row_bytes, warps > 8 ? 2 : 3) * sms);
    a.rb_per_cta = (w.nrb + p.grid - 1) / p.grid;
    if (glu) {   // (gate, up) pairs of row-blocks stay together
        if ((w.nrb & 1) || (w.n & 31)) fail(MFQB_ERR_ARG, "gated product: the weight needs whole (gate, up) pairs of 16-row blocks, n = %d", w.n);
        p.grid = std::min(w.nrb / 2, p.grid);
        a.rb_per_cta = 2 * ((w.nrb / 2 + p.grid - 1) / p.grid);
        a.glu = 1;
    }
    a.private_sums = gemv1_private_sums(a.rb_per_cta);
    p.smem = gemv1_smem(w, a.rb_per_cta, warps) + row_bytes;
    if (p.smem > kGemvSmemLimit) fail(MFQB_ERR_UNSUPPORTED, "fused normalisation: a row of %d columns does not fit shared memory beside the rings", w.k);
    dispatch(a, p, s, "GEMV with fused RMSNorm");
}

// Streamed single-row product (nint_gemvs.cuh).  `fix` is the weight's own scratch for row-blocks
// that straddle CTAs: [sms][16] (value, flag) pairs, all zero between calls.  Returns false when the
// activation planes of this row length and a useful ring do not fit one CTA; the caller then
// takes the ring kernel.
static cudaError_t dispatch_gemvs(const GemvSArgs& a, const GemvSPlan& p, cudaStream_t s) {
    switch (a.w.bits) {
        case 2: return launch_gemvs_bits<2>(a, p, s);
        case 3: return launch_gemvs_bits<3>(a, p, s);
        case 4: return launch_gemvs_bits<4>(a, p, s);
        case 5: return launch_gemvs_bits<5>(a, p, s);
        case 6: return launch_gemvs_bits<6>(a, p, s);
        case 8: return launch_gemvs_bits<8>(a, p, s);
        default: return cudaErrorInvalidValue;
    }
}

#ifdef MFQB_GEMVS_TRACE
static unsigned long long* g_gemvs_trace = nullptr;
extern "C" __attribute__((visibility("default"))) void mfqb_debug_set_gemvs_trace(void* p) { g_gemvs_trace = static_cast<unsigned long long*>(p); }
#endif

size_t gemvs_fix_bytes(int device) { return (size_t)device_sm_count(device) * 16 * sizeof(uint2); }

bool launch_bl_gemvs(const NintDevB& w, const void* x, int x_dtype, void* y, int y_dtype, int device, void* fix, int* error, cudaStream_t s) {
    if (w.table || !fix || x_dtype != MFQB_BF16) return false;   // lattice records stay on the ring kernel
    const int sms = device_sm_count(device);
    const long long total = (long long)w.nrb * w.nchunks;
    if (total < 1 || total * (sms + 1) >= (1ll << 31)) return false;
    const int grid = (int)std::min<long long>(sms, total);
    const size_t recb = (size_t)w.rec_words * 4;
    const int ngp = w.nchunks * kChunkGroupsB;
    const size_t planes = (size_t)ngp * 16 + 288 + (size_t)ngp * gemvs_group_bytes(w.t8) + 128;   // group table, maxima, sums | zeros | planes
    const long long n_b = (total + grid - 1) / grid;
    GemvSArgs a{};
    GemvSPlan p;
    bool found = false;
    // two CTAs (this product's and the next one's) share an SM when a CTA stays below half of it
    // Most warps first (they hide the latency of the arithmetic and share the staging work), as long as
    // every warp keeps two records in flight.  A CTA below half an SM lets the next product's CTA
    // move in early; records too wide for eight such warps take the whole SM instead.
    struct Try { size_t budget; int warps; };
    for (const Try t : {Try{110 * 1024, 16}, Try{110 * 1024, 12}, Try{110 * 1024, 8}, Try{200 * 1024, 8}, Try{110 * 1024, 4}, Try{200 * 1024, 4}}) {
        const int warps = t.warps;
        if (warps * 32 > gemvs_max_threads(w.wc)) continue;
        const long long n_w = (n_b + warps - 1) / warps;
        const int maxseg = (int)((n_w - 1) / w.nchunks) + 2;
        const int maxrb = (int)(n_b / w.nchunks) + 2;
        const size_t fixed = planes + (size_t)warps * maxseg * 64 + (size_t)(maxrb + 3) / 4 * 16 + 16;
        if (fixed >= t.budget) continue;
        int stages = (int)std::min<size_t>(8, (t.budget - fixed) / (warps * (recb + 8)));
        stages = (int)std::min<long long>(stages, std::max<long long>(n_w, 1));
        const int need = (int)std::min<long long>(2, std::max<long long>(n_w, 1));
        if (stages < need) continue;
        p.grid = grid;
        p.threads = warps * 32;
        p.smem = fixed + (size_t)warps * stages * (recb + 8);
        a.stages = stages;
        a.maxseg = maxseg;
        a.maxrb = maxrb;
        found = true;
        break;
    }
    if (!found) return false;
    a.w = w;
    a.x = x;
    a.x_dtype = x_dtype;
    a.y = y;
    a.y_dtype = y_dtype;
    a.fix_slots = static_cast<uint2*>(fix);
    a.error = error;
#ifdef MFQB_GEMVS_TRACE
    a.trace = g_gemvs_trace;
#endif
    const cudaError_t e = dispatch_gemvs(a, p, s);
    if (e != cudaSuccess) fail(MFQB_ERR_CUDA, "NINT%d gs=%d streamed GEMV launch (%d x %d threads, %zu bytes): %s", w.bits, w.gs, p.grid, p.threads, p.smem,
                               cudaGetErrorString(e));
    return true;
}

// Several weights of one shape class applied to the same activation row in one launch (q|k|v, gate|up:
// the reference's NintLinearGroup, cpp_runtime/mfq_decode.cpp:8618-8743): grid = (CTAs per weight, weights).
void launch_bl_gemv_multi(const NintDevB* ws, void* const* ys, int count, const void* x, int y_dtype, int device, cudaStream_t s) {
    if (count < 1 || count > kGemvMultiMax) fail(MFQB_ERR_ARG, "a multi-weight launch takes 1 to %d weights, got %d", kGemvMultiMax, count);
    GemvArgsB a{};
    a.w = ws[0];
    a.x = static_cast<const __nv_bfloat16*>(x);
    a.m = 1;
    a.y_dtype = y_dtype;
    GemvMultiTable table{};
    int max_nrb = 0;
    for (int i = 0; i < count; ++i) {
        const NintDevB& w = ws[i];
        if (w.table || w.bits != ws[0].bits || w.gs != ws[0].gs || w.k != ws[0].k || w.rec_words != ws[0].rec_words)
            fail(MFQB_ERR_ARG, "the weights of a multi-weight launch must share family, code width, group size and k");
        table.e[i] = GemvMultiEntry{w.items, w.anchors, ys[i], w.n, w.nrb};
        max_nrb = std::max(max_nrb, w.nrb);
    }
    a.ldy = 0;
    GemvPlanB p;
    const int warps = gemv1_warps(ws[0]), sms = device_sm_count(device);
    p.threads = warps * 32;
    p.passes = -1;
    p.multi = &table;
    // all CTAs resident at once: the SMs' slots shared out over the weights
    const int per_weight = std::max(1, ctas_per_sm(gemv1_smem(ws[0], 1, warps), warps > 8 ? 2 : 3) * sms / count);
    a.rb_per_cta = (max_nrb + std::min(max_nrb, per_weight) - 1) / std::min(max_nrb, per_weight);
    p.grid = (max_nrb + a.rb_per_cta - 1) / a.rb_per_cta;   // no more CTAs than that many row-blocks each need: an even split
    p.grid_y = count;
    a.private_sums = gemv1_private_sums(a.rb_per_cta);
    p.smem = gemv1_smem(ws[0], a.rb_per_cta, warps);
    if (p.smem > kGemvSmemLimit) fail(MFQB_ERR_UNSUPPORTED, "multi-weight launch: %d row-blocks per CTA do not fit shared memory", a.rb_per_cta);
    dispatch(a, p, s, "multi-weight GEMV");
}

// Single-row product whose epilogue reduces over ranks (row-parallel shards): see PeerReduce.
void launch_bl_gemv_reduce(const NintDevB& w, const void* x, void* y, int y_dtype, int device, const PeerReduce& pr, cudaStream_t s) {
    GemvArgsB a{};
    a.w = w;
    a.x = static_cast<const __nv_bfloat16*>(x);
    a.y = y;
    a.m = 1;
    a.ldy = w.n;
    a.y_dtype = y_dtype;
    a.reduce = pr;
    GemvPlanB p;
    const int warps = gemv1_warps(w), sms = device_sm_count(device);
    p.threads = warps * 32;
    // Every CTA waits for its peers inside the kernel, so the whole grid must be resident at once: the
    // grid is sized from the occupancy the runtime reports for this kernel, block size and shared memory
    // (which itself grows with the row-blocks per CTA, hence the second look).
    p.grid = std::min(w.nrb, ctas_per_sm(gemv1_smem(w, 1, warps), warps > 8 ? 2 : 3) * sms);
    for (int round = 0; round < 3; ++round) {
        a.rb_per_cta = (w.nrb + p.grid - 1) / p.grid;
        a.private_sums = gemv1_private_sums(a.rb_per_cta);
        p.smem = gemv1_smem(w, a.rb_per_cta, warps);
        if (p.smem > kGemvSmemLimit) fail(MFQB_ERR_UNSUPPORTED, "weight of %d rows is too tall for one resident grid", w.n);
        int per_sm = 0;
        GemvPlanB query = p;
        query.occupancy_out = &per_sm;
        dispatch(a, query, s, "row-parallel GEMV (occupancy)");
        if (per_sm < 1) fail(MFQB_ERR_UNSUPPORTED, "row-parallel GEMV: a CTA of %d threads and %zu bytes does not fit an SM", p.threads, p.smem);
        if (p.grid <= per_sm * sms) break;
        if (round == 2) fail(MFQB_ERR_UNSUPPORTED, "row-parallel GEMV: no grid of this weight's %d row-blocks is resident at once", w.nrb);
        p.grid = per_sm * sms;
    }
    dispatch(a, p, s, "row-parallel GEMV");
}

// Routed single-row launch over (splits, pairs) CTAs for one cohort; see GemvArgsB.
void launch_nint_bl_gemv_routed(GemvArgsB a, int pairs, int device, cudaStream_t s) {
    const NintDevB& w = a.w;
    a.m = 1;
    GemvPlanB p;
    const int want = (3 * device_sm_count(device) + pairs - 1) / std::max(pairs, 1);
    const int splits = std::max(1, std::min(a.rb_per_expert, want));
    a.rb_per_cta = (a.rb_per_expert + splits - 1) / splits;
    a.private_sums = gemv1_private_sums(a.rb_per_cta);
    p.smem = gemv1_smem(w, a.rb_per_cta, 8);
    p.grid = splits;
    p.grid_y = pairs;
    p.passes = -3;
    dispatch(a, p, s, "routed GEMV");
}

// Batched kernel over route-plan tiles (up to tile_m = 2, 4 or 8 pairs of one expert each) for one cohort.
void launch_nint_bl_gemv_tiles(GemvArgsB a, int tile_m, int max_tiles, int device, cudaStream_t s) {
    const NintDevB& w = a.w;
    a.m = tile_m;
    GemvPlanB p;
    p.passes = tile_m / 2;
    // max_tiles is an upper bound and a launch covers one cohort only, so most of its tiles return at
    // once: split an expert's rows finely (about eight row-blocks per CTA) to keep the SMs busy
    const int want = (2 * device_sm_count(device) + max_tiles - 1) / std::max(max_tiles, 1);
    const int splits = std::max(1, std::min(a.rb_per_expert, std::max(a.rb_per_expert / 8, want)));
    a.rb_per_cta = (a.rb_per_expert + splits - 1) / splits;
    p.smem = gemvn_smem(w, a.rb_per_cta, p.passes);
    p.grid = splits;
    p.grid_y = max_tiles;
    dispatch(a, p, s, "routed tile GEMV");
}

}  // namespace mfqb
