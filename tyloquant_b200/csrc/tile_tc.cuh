// Batched products of packed weights on tcgen05 tensor cores, weights decoded straight into tensor memory.
//
//   y[token, n] = sum_k x[token, k] * W[n, k]
//
// A CTA works on tiles of 128 weight rows x N tokens (N <= 256), one chunk (8 groups) of K at a time, and every warp has one
// role for the whole kernel:
//   * record loader: bulk copies of the chunk's eight packed records (one per 16-row block) into a ring in shared memory; the
//     weights are constants, so it starts before the kernel waits for its predecessor in the stream;
//   * activation loader: bulk copies of 64-column slabs of the scaled f16 activations, which x_tiles_kernel has already
//     written in the order, padding and 128-byte swizzle the tensor core reads (no tensor map);
//   * 16 decoders: warp (row-block, half of the chunk) turns codes into f16 pairs in registers -- in byte-lane fragment order
//     these ARE rows q, q + 8 of a 16 x 16 A operand -- and stores them with tcgen05.st into the A ring in tensor memory.
//     The A operand never touches shared memory, whose bandwidth the B operand needs (8 KB in and 8 KB out per 128 cycles
//     for N = 256);
//   * mma issuer: one thread, tcgen05.mma with A from tensor memory, B from shared memory, D in tensor memory;
//   * 4 epilogue warps: tcgen05.ld, scaling by row and token factors, stores.
//
// Arithmetic.  A row of W is factored as F * (a ss (q - mid) + (mid a ss - b sm)) with a = ns / F, b = nm / F (tile_row_const):
// F is applied to the finished sums in float32, and since a is a power of two the step a ss is exact in f16.  The offset is
// formed with two fused multiply-adds (b as high and low f16 part), so a weight is rounded twice in f16, about 2.4e-4 relative
// L2 on the product.  Group sizes that are no multiple of eight have integer kernels (4e-6) as their other path, so their
// weights are fed as two f16 terms that carry 22 bits.  Lattice weights are integers ss * code <= 225,
// exact in f16; the scales of a joint-codebook record are f16 numbers, and where some product with a code has more than 11
// bits the weight is fed as two f16 terms whose sum is exact.  Activations: one power-of-two scale per token
// (largest magnitude next to 2^15), exact for bf16 values within 2^-28 of the row's largest.
//
// Work split.  Plain products: the (tile, chunk) units are cut into equal contiguous ranges, one per CTA, or every tile into
// as many parts.  The CTAs that share a tile leave their parts in L2, and the last one to arrive adds them up in the order of
// K, so a product has the same bits in every call (no CTA ever waits for another; float32 reductions into one copy, whose order
// is that of arrival, took 84.1 us for four products of 16 rows, NINT6 4096 x 14336, this 84.4; 77 rows, three parts of 80
// columns, NINT5 5000 x 2888: 70.6 and 76.0).  Expert products (route plan): item = (row
// tile, token tile of one expert), strided over the CTAs.
//
// Every mbarrier wait is bounded: on expiry the CTA raises the device's status word, waits (bounded) for its own copies and
// leaves through the common exit, which frees the tensor memory.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "common.h"
#include "lane_unit.h"
#include "nint_blayout.h"
#include "tc05.cuh"
#include "tile_tc.h"

namespace mfqb {

constexpr int kTileRows = 128, kTileDecoders = 16, kTileEpilogue = 4;
constexpr int kTileWarpMma = kTileDecoders + kTileEpilogue, kTileWarpRec = kTileWarpMma + 1, kTileWarpX = kTileWarpMma + 2;
constexpr int kTileThreads = (kTileDecoders + kTileEpilogue + 3) * 32;
constexpr size_t kTileDynSmem = 212 * 1024;   // beside 14 KB of barriers and tables
constexpr int kTileGroup = 12;   // parts of a shared tile that are added at once; more go in two steps
constexpr int kTileMaxPools = 16, kTileRecStages = 8, kTileXStages = 8, kTileAStages = 8, kTileSegs = 4;

struct TileArgs {
    NintDevB pools[kTileMaxPools];   // the weight (entry 0), or the cohorts of an expert record
    // lattice records: f16 state scales normalised by a power of two, and its inverse
    uint16_t lut16[16];
    float lut_undo;                  // (1 for scalar records)
    const unsigned char* x;          // activation tiles (x_tiles_kernel)
    size_t x_row_bytes;              // bytes of one row in the tiles' buffer (2 x the padded K, the largest among the cohorts)
    int x_rows;                      // most rows of a tile; a tile of c rows is stored with (c + 7) / 8 * 8 rows per 64-column slab
    const float* x_down;             // inverse scale per token, or per position of the route plan
    void* y;
    int y_dtype, ldy;
    int glu;                         // plain product: rows come in 16-row blocks, gate and up in turn; y gets up * silu(gate) (the launch picks the kernel)
    int m, ntok;                     // plain product: tokens, token tiles
    int units, split;                // plain product: (tile, chunk) units; CTAs per tile, or 0: equal ranges of units
    float* partial;                  // [2 grid][N][128] float32 parts of tiles that several CTAs share, see tile_part
    unsigned* counters;              // arrivals at a group of parts [grid], by the group's first CTA, and of groups at a tile [grid], by the tile's; zero from x_tiles_kernel
    int sum_bytes;                   // shared memory that the addition of parts may use
    // expert product over a route plan with tiles of x_rows pairs; tile_bounds == nullptr: plain product
    const int *expert_bounds, *tile_bounds, *pair_order, *expert_pool, *expert_local;
    int n_experts, rb_per_expert, rows_per_expert, only_pool /* -1: every cohort */, scatter /* rows go to pair_order[p], else to p */;
    // shared- and tensor-memory plan
    int n_mma;                       // N of the instruction
    int rec_stages, rec_stage_bytes, x_stages, x_stage_bytes, x_whole /* 0: an activation stage is one 64-column slab; 1: the slabs of a step */, step /* chunks per step */, a_stages, a_cols, d_bufs, d_cols;
    int* error;
};

static_assert(sizeof(TileArgs) <= 4096, "kernel parameters");

// One stretch of work: chunks [ch0, ch1) of a tile.
struct TileSeg {
    int pool, rb0, nrb, row0, row_limit, ch0, ch1, nchunks;
    int tok0, ncols;
    size_t x_off;
    int parts, slot0, last;   // CTAs that share the tile, the first of them; whether it is this CTA's last stretch
};

// First unit of CTA b of a plain product.  split = 0: equal ranges; else `split` CTAs share every tile and none has a part of
// two (see launch_tile_product).
__device__ __forceinline__ int tile_unit_begin(const TileArgs& a, int b) {
    if (a.split == 0) return (int)((long long)b * a.units / gridDim.x);
    const int tile = b / a.split, part = b - tile * a.split, nch = a.pools[0].nchunks;
    return tile * nch + part * nch / a.split;
}
// The CTAs that share a tile: the first one, and how many.
__device__ __forceinline__ void tile_sharers(const TileArgs& a, int tile, int& slot0, int& parts) {
    if (a.split) {
        slot0 = tile * a.split;
        parts = a.split;
        return;
    }
    const int nch = a.pools[0].nchunks, grid = gridDim.x;
    auto owner = [&](int u) { return (int)((((long long)u + 1) * grid - 1) / a.units); };
    slot0 = owner(tile * nch);
    parts = owner((tile + 1) * nch - 1) - slot0 + 1;
}

// Part p of a shared tile: a CTA has at most the end of one tile (or a middle part) and the beginning (part 0) of another.
__device__ __forceinline__ float* tile_part(const TileArgs& a, int slot0, int p) {
    return a.partial + (size_t)(2 * (slot0 + p) + (p == 0)) * a.n_mma * kTileRows;
}

// First row of an expert's tile in the tiles' buffer: every tile starts on a multiple of eight rows, and experts do not overlap.
__host__ __device__ __forceinline__ int tile_x_row(int expert_begin, int expert, int row_in_expert) { return (expert_begin + 7) / 8 * 8 + 8 * expert + row_in_expert; }

// Next stretch of this CTA; `cursor` starts at the CTA's first unit (plain) or item (experts).
__device__ __forceinline__ bool tile_next(const TileArgs& a, int& cursor, TileSeg& s) {
    if (a.tile_bounds == nullptr) {
        const int end = tile_unit_begin(a, blockIdx.x + 1);
        if (cursor >= end) return false;
        const NintDevB& w = a.pools[0];
        const int tile = cursor / w.nchunks, rt = tile / a.ntok, tt = tile - rt * a.ntok;
        s.pool = 0;
        s.ch0 = cursor - tile * w.nchunks;
        s.ch1 = min(w.nchunks, s.ch0 + end - cursor);
        s.nchunks = w.nchunks;
        s.rb0 = rt * 8;
        s.nrb = min(8, w.nrb - s.rb0);
        s.row0 = rt * kTileRows;
        s.row_limit = w.n;
        s.tok0 = tt * a.x_rows;
        s.ncols = min(a.x_rows, a.m - s.tok0);
        s.x_off = (size_t)s.tok0 * a.x_row_bytes;
        tile_sharers(a, tile, s.slot0, s.parts);
        cursor += s.ch1 - s.ch0;
        s.last = cursor >= end;
        return true;
    }
    const int row_tiles = (a.rows_per_expert + kTileRows - 1) / kTileRows, items = a.tile_bounds[a.n_experts] * row_tiles;
    for (; cursor < items; cursor += gridDim.x) {
        const int t = cursor / row_tiles, rt = cursor - t * row_tiles;
        int lo = 0, hi = a.n_experts - 1;   // expert e with tile_bounds[e] <= t < tile_bounds[e + 1]
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (a.tile_bounds[mid] <= t) lo = mid;
            else hi = mid - 1;
        }
        const int pool = a.expert_pool[lo];
        if (pool < 0 || (a.only_pool >= 0 && pool != a.only_pool)) continue;
        s.pool = a.only_pool >= 0 ? 0 : pool;
        s.nchunks = a.pools[s.pool].nchunks;
        s.ch0 = 0;
        s.ch1 = s.nchunks;
        s.rb0 = a.expert_local[lo] * a.rb_per_expert + rt * 8;
        s.nrb = min(8, a.rb_per_expert - rt * 8);
        s.row0 = rt * kTileRows;
        s.row_limit = a.rows_per_expert;
        s.tok0 = a.expert_bounds[lo] + (t - a.tile_bounds[lo]) * a.x_rows;
        s.ncols = min(a.x_rows, a.expert_bounds[lo + 1] - s.tok0);
        s.x_off = (size_t)tile_x_row(a.expert_bounds[lo], lo, (t - a.tile_bounds[lo]) * a.x_rows) * a.x_row_bytes;
        s.slot0 = s.last = 0;
        s.parts = 1;
        cursor += gridDim.x;
        return true;
    }
    return false;
}
__device__ __forceinline__ int tile_first(const TileArgs& a) { return a.tile_bounds == nullptr ? tile_unit_begin(a, blockIdx.x) : (int)blockIdx.x; }

__device__ __forceinline__ __half2 h2_bits(uint32_t v) { return *reinterpret_cast<const __half2*>(&v); }
__device__ __forceinline__ uint32_t bits_h2(__half2 v) { return *reinterpret_cast<const uint32_t*>(&v); }

// ---- codecs: decode one warp's half of a chunk record into the A ring ---------------------------------------------------
// Row(consts, lane): what depends on the row-block only, from the 16 rows' constants.  half<F>(rec, lane, row, ctx, taddr): family F of the record at `rec`
// (shared memory) to the 16 tensor-memory lanes at taddr, columns 16 t + 8 h + {0..7} for octet t and group pair h.
// The two values of a column are slots i, i + 2 of a quad (the bytes a 16-bit lane mask picks), columns c / 4 + c slots 0, 2 /
// 1, 3 of quad c: x_tiles_kernel writes the activations in this order.
// TERMS 2: two terms whose sum carries some 22 bits, by error-free sums and products.
template <int BITS, int T_, int TERMS_ = 1>
struct TileNint {
    static constexpr int T = T_, TERMS = TERMS_;
    using BU = ByteUnit<BITS>;
    static constexpr int WC = BU::words_for(8 * T);
    static constexpr int MID = 1 << (BITS - 1);
    // Bit position inside a byte at which register a (= r % 4) is read: where the packing leaves it, so that it is not shifted.
    __host__ __device__ static constexpr int pos(int a) { return BITS == 2 ? 2 * a : ((BITS == 3 || BITS == 4) ? BITS * (a & 1) : 0); }
    __host__ __device__ static size_t ctx_bytes(const NintDevB&) { return 0; }
    __device__ static void ctx_init(unsigned char*, const TileArgs&, int, int) {}

    struct Row {
        __half2 step[2];      // a * scale * 2^-pos for rows q, q + 8, per group pair h
        __half2 mid;          // a * scale * mid
        __half2 nb_hi, nb_lo; // -b * scale, high and low part
        __device__ __forceinline__ Row(const NintDevB&, const uint4* consts, int lane) {
            const uint4 c0 = consts[lane >> 2], c1 = consts[8 + (lane >> 2)];
            const __half2 a2 = h2_bits(__byte_perm(c0.x, c1.x, 0x5410));
#pragma unroll
            for (int h = 0; h < 2; ++h) step[h] = __hmul2(a2, __floats2half2_rn(1.f / (float)(1 << pos(2 * h)), 1.f / (float)(1 << pos(2 * h + 1))));
            mid = __hmul2(a2, __float2half2_rn((float)MID));
            nb_hi = h2_bits(__byte_perm(c0.x, c1.x, 0x7632));
            nb_lo = h2_bits(__byte_perm(c0.y, c1.y, 0x5410));
        }
    };
    // register r as two f16 pairs 1024 + q 2^pos: bytes 0, 2 and bytes 1, 3
    template <int R>
    __device__ static __forceinline__ void pairs(const uint32_t* rec, int lane, __half2& even, __half2& odd) {
        constexpr int P = pos(R % 4), TT = R % BU::NP, UNIT = R / BU::NP;
        constexpr uint32_t M = ((1u << BITS) - 1u) << P, MASK = M | (M << 16);
        uint32_t v;
        if constexpr (TT < BU::U * BU::F) {   // a whole field of one word, at its place
            static_assert((TT % BU::F) * BITS == P, "field position");
            v = rec[(UNIT * BU::U + TT / BU::F) * 32 + lane];
        } else {
            uint32_t u[BU::U];
#pragma unroll
            for (int i = 0; i < BU::U; ++i) u[i] = rec[(UNIT * BU::U + i) * 32 + lane];
            v = BU::at(u, TT) << P;
        }
        even = h2_bits((v & MASK) | 0x64006400u);
        odd = h2_bits(((v >> 8) & MASK) | 0x64006400u);
    }
    template <int R>
    __device__ static __forceinline__ void weights(const uint32_t* rec, int lane, __half2 d, __half2 n, uint32_t& lo, uint32_t& hi) {
        __half2 even, odd;
        pairs<R>(rec, lane, even, odd);
        const __half2 bias = __float2half2_rn(1024.f + (float)(MID << pos(R % 4)));
        lo = bits_h2(__hfma2(__hsub2(even, bias), d, n));
        hi = bits_h2(__hfma2(__hsub2(odd, bias), d, n));
    }
    // q d + n + nl in two terms: p + pe = q d and s + se = p + n exactly.
    __device__ static __forceinline__ void terms(__half2 q, __half2 d, __half2 n, __half2 nl, uint32_t& first, uint32_t& second) {
        const __half2 p = __hmul2_rn(q, d), pe = __hfma2(q, d, __hneg2(p));
        const __half2 s = __hadd2_rn(p, n), b = __hsub2_rn(s, p), se = __hadd2_rn(__hsub2_rn(p, __hsub2_rn(s, b)), __hsub2_rn(n, b));
        first = bits_h2(s);
        second = bits_h2(__hadd2_rn(__hadd2_rn(se, pe), nl));
    }
    template <int R>
    __device__ static __forceinline__ void weights2(const uint32_t* rec, int lane, __half2 d, __half2 n, __half2 nl, uint32_t& lo, uint32_t& hi, uint32_t& lo2, uint32_t& hi2) {
        __half2 even, odd;
        pairs<R>(rec, lane, even, odd);
        const __half2 bias = __float2half2_rn(1024.f + (float)(MID << pos(R % 4)));
        terms(__hsub2(even, bias), d, n, nl, lo, lo2);
        terms(__hsub2(odd, bias), d, n, nl, hi, hi2);
    }
    template <int F, int TI>
    __device__ static __forceinline__ void octets(const uint32_t* rec, int lane, const __half2 (&d)[4], const __half2 (&n)[4], const __half2 (&nl)[4], uint32_t taddr) {
        if constexpr (TI < T && TERMS == 2) {
            constexpr int R = (F * T + TI) * 4;
            uint32_t r[8], e[8];
            weights2<R>(rec, lane, d[0], n[0], nl[0], r[0], r[2], e[0], e[2]);
            weights2<R + 1>(rec, lane, d[1], n[1], nl[1], r[1], r[3], e[1], e[3]);
            weights2<R + 2>(rec, lane, d[2], n[2], nl[2], r[4], r[6], e[4], e[6]);
            weights2<R + 3>(rec, lane, d[3], n[3], nl[3], r[5], r[7], e[5], e[7]);
            tmem_st_16x128b_x4(taddr + 16 * TI, r);
            tmem_st_16x128b_x4(taddr + 16 * T + 16 * TI, e);
            octets<F, TI + 1>(rec, lane, d, n, nl, taddr);
        } else if constexpr (TI < T) {
            constexpr int R = (F * T + TI) * 4;
            uint32_t r[8];
            weights<R>(rec, lane, d[0], n[0], r[0], r[2]);
            weights<R + 1>(rec, lane, d[1], n[1], r[1], r[3]);
            weights<R + 2>(rec, lane, d[2], n[2], r[4], r[6]);
            weights<R + 3>(rec, lane, d[3], n[3], r[5], r[7]);
            tmem_st_16x128b_x4(taddr + 16 * TI, r);
            octets<F, TI + 1>(rec, lane, d, n, nl, taddr);
        }
    }
    // Both halves of a chunk run the same code where the second one's registers start on a word.
    static constexpr bool SPLIT = (4 * T) % BU::NP == 0;
    static constexpr int FW = SPLIT ? 4 * T / BU::NP * BU::U : 0;
    template <int F>
    __device__ static __forceinline__ void half(const uint32_t* rec, int lane, int f, const Row& row, const unsigned char*, uint32_t taddr) {
        const uint32_t sel = (lane & 2) ? 0x4341u : 0x4240u;   // this lane's group of a pair: bytes (row q, row q + 8)
        const __half2 k1024 = __float2half2_rn(1024.f);
        __half2 d[4], n[4], nl[4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t* sc = rec + WC * 32 + (lane & ~3) + 2 * f + h;
            const __half2 ss = __hsub2(h2_bits(__byte_perm(sc[0], 0x64646464u, sel)), k1024);
            const __half2 sm = __hsub2(h2_bits(__byte_perm(sc[32], 0x64646464u, sel)), k1024);
            const __half2 d2 = __hmul2(ss, row.step[h]);
            __half2 n2, l2;
            if constexpr (TERMS == 2) {   // m + (v + ve) in two terms, m and v + ve exact
                const __half2 m = __hmul2_rn(ss, row.mid), v = __hmul2_rn(sm, row.nb_hi), ve = __hfma2(sm, row.nb_hi, __hneg2(v));
                n2 = __hadd2_rn(m, v);
                const __half2 b = __hsub2_rn(n2, m), ne = __hadd2_rn(__hsub2_rn(m, __hsub2_rn(n2, b)), __hsub2_rn(v, b));
                l2 = __hfma2(sm, row.nb_lo, __hadd2_rn(ne, ve));
            } else {
                n2 = l2 = __hfma2(sm, row.nb_lo, __hfma2(sm, row.nb_hi, __hmul2(ss, row.mid)));
            }
            nl[2 * h] = __low2half2(l2);
            nl[2 * h + 1] = __high2half2(l2);
            d[2 * h] = __low2half2(d2);
            d[2 * h + 1] = __high2half2(d2);
            n[2 * h] = __low2half2(n2);
            n[2 * h + 1] = __high2half2(n2);
        }
        octets<F, 0>(rec + (SPLIT ? f * FW * 32 : 0), lane, d, n, nl, taddr);
    }
};

// ---- the kernel ----------------------------------------------------------------------------------------------------------
struct TileShared {
    __align__(8) uint64_t rec_full[kTileRecStages], rec_empty[kTileRecStages], x_full[kTileXStages], x_empty[kTileXStages];
    uint64_t a_full[kTileAStages], a_empty[kTileAStages], d_full[2], d_empty[2], drain;
    uint32_t tmem;
    int failed;
    unsigned last;
    uint64_t sum_full[2];
    // Groups of parts that this CTA was the last to arrive at, and adds up at its end: [0] with its last stretch, [1] with an
    // earlier one (parts == 0: none).
    TileSeg fin[2];
    int fin_col;   // column table of fin[0]; its row factors are in row_factor
    __align__(16) float row_factor[kTileRows];
    __align__(16) uint4 rowc[kTileSegs][kTileRows];   // the stretches' row constants
    uint64_t seg_full[kTileSegs], seg_empty[kTileSegs];
    TileSeg seg[kTileSegs];                            // stretches in order, from the record loader; parts == 0: no more
    __align__(16) int2 col[2][256];   // the epilogue's tile (two in turn): factor (float bits) and output row of every column
};

struct TileRing {
    int stage = 0;
    uint32_t phase = 0;
    __device__ __forceinline__ void step(int n) {
        if (++stage == n) { stage = 0; phase ^= 1u; }
    }
};
template <int N, int I = 0, class Fn>
__device__ __forceinline__ void tile_static_for(Fn&& f) {
    if constexpr (I < N) {
        f(std::integral_constant<int, I>{});
        tile_static_for<N, I + 1>(f);
    }
}
__device__ __forceinline__ bool tile_wait(uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity)); }

// Both barriers with one round trip where both phases are already complete.
__device__ __forceinline__ bool tile_wait2(uint64_t* bar0, uint32_t parity0, uint64_t* bar1, uint32_t parity1) {
    const bool r0 = mbar_test(bar0, parity0), r1 = mbar_test(bar1, parity1);
    if (__all_sync(0xffffffffu, r0 && r1)) return true;
    return tile_wait(bar0, parity0) && tile_wait(bar1, parity1);
}

// Global stores that the compiler does not order against shared-memory loads: with plain stores every look-up of a column's
// table entry waited for the store before it, 70 cycles a column.
__device__ __forceinline__ void st_global(float* p, float v) { asm volatile("st.global.f32 [%0], %1;" ::"l"(p), "f"(v)); }
__device__ __forceinline__ void st_global(__nv_bfloat16* p, __nv_bfloat16 v) { asm volatile("st.global.b16 [%0], %1;" ::"l"(p), "h"(__bfloat16_as_ushort(v))); }

__device__ __forceinline__ float tile_gated(float gate, float up) { return up * gate / (1.0f + expf(-gate)); }

// True for the four epilogue warps when it is true for all of them: they leave together, none waits at a barrier for one that gave up.
__device__ __forceinline__ bool tile_epilogue_all(bool ok) {
    uint32_t all;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbarrier.cta.red.and.pred p, 1, 128, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(all) : "r"((uint32_t)ok) : "memory");
    return all != 0u;
}

// Adding up parts p0, p0 + step, ... of a shared tile, in this order (up to 128 KB each in L2, stored column by column): a block
// of columns at a time comes into the rings' memory with bulk copies, two blocks in flight, then a warp takes a column, four
// rows a lane.  (The four epilogue warps alone, sixteen loads in flight each, took 40,000 cycles for one part of N = 256.)
struct TileSum {
    int slot0, p0, step, count, ncols, cols, blocks;
    __device__ __forceinline__ TileSum(const TileArgs& a, const TileSeg& t, int p0_, int step_, int count_) : slot0(t.slot0), p0(p0_), step(step_), count(count_), ncols(t.ncols) {
        cols = max(1, min(ncols, a.sum_bytes / (2 * count * kTileRows * 4)));
        blocks = (ncols + cols - 1) / cols;
    }
    __device__ __forceinline__ void request(const TileArgs& a, TileShared& sh, float* stage, int b) const {   // one thread
        const int c0 = b * cols;
        const uint32_t bytes = (uint32_t)min(cols, ncols - c0) * kTileRows * 4u;
        asm volatile("fence.proxy.async;" ::: "memory");
        mbar_arrive_expect_tx(&sh.sum_full[b & 1], bytes * (uint32_t)count);
        for (int q = 0; q < count; ++q)
            bulk_load(stage + (size_t)((b & 1) * count + q) * cols * kTileRows, tile_part(a, slot0, p0 + q * step) + (size_t)c0 * kTileRows, bytes, &sh.sum_full[b & 1]);
    }
    __device__ __forceinline__ void request_first(const TileArgs& a, TileShared& sh, float* stage) const {   // the stage is free
        request(a, sh, stage, 0);
        if (blocks > 1) request(a, sh, stage, 1);
    }
    // The whole CTA; the first blocks are requested.  phase: bit b, parity of the next wait on sum_full[b].
    template <class Put>
    __device__ __forceinline__ bool run(const TileArgs& a, TileShared& sh, float* stage, uint32_t& phase, Put&& put) const {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        bool ok = true;
        for (int b = 0; b < blocks && ok; ++b) {
            ok = tile_wait(&sh.sum_full[b & 1], (phase >> (b & 1)) & 1u);
            phase ^= 1u << (b & 1);
            const float* src = stage + (size_t)(b & 1) * count * cols * kTileRows + 4 * lane;
            const int c0 = b * cols, n = min(cols, ncols - c0);
            if (ok)
                for (int c = warp; c < n; c += kTileThreads / 32) {
                    float4 v = *reinterpret_cast<const float4*>(src + c * kTileRows);
                    for (int q = 1; q < count; ++q) {
                        const float4 x = *reinterpret_cast<const float4*>(src + (q * cols + c) * kTileRows);
                        v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
                    }
                    put(c0 + c, v);
                }
            ok = __syncthreads_and(ok);
            if (ok && threadIdx.x == 0 && b + 2 < blocks) request(a, sh, stage, b + 2);
        }
        return ok;
    }
};

// First part of the group that this CTA's part belongs to, and how many the group has.
__device__ __forceinline__ int2 tile_group(const TileSeg& t) {
    const int p0 = ((int)blockIdx.x - t.slot0) / kTileGroup * kTileGroup;
    return make_int2(p0, min(kTileGroup, t.parts - p0));
}
// Adds up a group of parts that this CTA was the last to arrive at, and where that is the last of the tile's groups, writes the
// tile.  The whole CTA; sh.row_factor and `down` (x: the token's factor) are filled, the sum's first blocks requested.
template <bool GLU>
__device__ __forceinline__ bool tile_finish(const TileArgs& a, TileShared& sh, const TileSeg& t, const int2* down_of, float* stage, uint32_t& phase) {
    const int tid = threadIdx.x, lane = tid & 31, groups = (t.parts + kTileGroup - 1) / kTileGroup;
    const int2 g = tile_group(t);
    TileSum sum(a, t, g.x, 1, g.y);
    bool ok = true;
    if (groups > 1) {
        float* group_sum = tile_part(a, t.slot0, g.x) + 4 * lane;
        ok = sum.run(a, sh, stage, phase, [&](int c, const float4& v) { __stcg(reinterpret_cast<float4*>(group_sum + (size_t)c * kTileRows), v); });
        __threadfence();
        __syncthreads();
        sum = TileSum(a, t, 0, kTileGroup, groups);
        if (ok && tid == 0) {
            unsigned* counter = a.counters + gridDim.x + t.slot0;
            sh.last = atomicAdd(counter, 1u);
            if (sh.last == (unsigned)(groups - 1)) {
                __threadfence();
                sum.request_first(a, sh, stage);
            }
        }
        __syncthreads();
        if (ok && sh.last != (unsigned)(groups - 1)) return true;
    }
    int row = t.row0 + 4 * lane, n = min(4, t.row_limit - row);
    if constexpr (GLU) {   // gate rows are lanes 0-3 of every eight, their up rows lanes 4-7
        if (lane & 4) n = 0;
        row = (row >> 5) * 16 + (row & 15);
    }
    const float4 f = *reinterpret_cast<const float4*>(sh.row_factor + 4 * lane);
    const bool vec = n == 4 && (a.ldy & 3) == 0 && (reinterpret_cast<uintptr_t>(a.y) & 15) == 0;
    ok = ok && sum.run(a, sh, stage, phase, [&](int c, const float4& v) {
        const float down = __int_as_float(down_of[c].x);
        float o[4] = {v.x * (f.x * down), v.y * (f.y * down), v.z * (f.z * down), v.w * (f.w * down)};
        if constexpr (GLU) {
#pragma unroll
            for (int i = 0; i < 4; ++i) o[i] = tile_gated(o[i], __shfl_xor_sync(0xffffffffu, o[i], 4));
        }
        const size_t at = (size_t)(t.tok0 + c) * a.ldy + row;   // (a plain product: its output rows are the tokens)
        if (a.y_dtype == 0 /* MFQB_F32 */) {
            float* y = reinterpret_cast<float*>(a.y) + at;
            if (vec) *reinterpret_cast<float4*>(y) = make_float4(o[0], o[1], o[2], o[3]);
            else
                for (int i = 0; i < n; ++i) y[i] = o[i];
        } else {
            __nv_bfloat16* y = reinterpret_cast<__nv_bfloat16*>(a.y) + at;
            if (vec) {
                const __nv_bfloat162 b0 = __floats2bfloat162_rn(o[0], o[1]), b1 = __floats2bfloat162_rn(o[2], o[3]);
                *reinterpret_cast<uint2*>(y) = make_uint2(*reinterpret_cast<const uint32_t*>(&b0), *reinterpret_cast<const uint32_t*>(&b1));
            } else {
                for (int i = 0; i < n; ++i) y[i] = __float2bfloat16_rn(o[i]);
            }
        }
    });
    return ok;
}

// The decoder warps' share of one stretch.
template <class C, int F>
__device__ __forceinline__ bool tile_decode(const TileArgs& a, TileShared& sh, const TileSeg& s, unsigned char* rec_ring, const unsigned char* ctx, TileRing& rr,
                                            TileRing& ar, int rbl, int f, int lane, uint32_t taddr, const uint4* consts, uint64_t* seg_done, int& runway) {
    const NintDevB& w = a.pools[s.pool];
    const bool mine = rbl < s.nrb;   // a tile at the end of the matrix has fewer row-blocks: their rows of D are never read
    const typename C::Row row(w, consts + (mine ? rbl : 0) * 16, lane);
    __syncwarp();
    if (lane == 0) mbar_arrive(seg_done);
    for (int ch = s.ch0; ch < s.ch1; ch += a.step) {
        if (runway == 0) asm volatile("griddepcontrol.wait;" ::: "memory");   // from here on the A ring empties only once the activations are there
        --runway;
        if (!tile_wait2(&sh.rec_full[rr.stage], rr.phase, &sh.a_empty[ar.stage], ar.phase ^ 1u)) return false;
        if (mine) {
            tc_fence_after_sync();
            const uint32_t* rec = reinterpret_cast<const uint32_t*>(rec_ring + (size_t)rr.stage * a.rec_stage_bytes) + rbl * a.step * w.rec_words;
            const uint32_t at = taddr + ar.stage * a.a_cols;
            C::template half<F>(rec, lane, f, row, ctx, at);
            if (a.step > 1 && ch + 1 < s.ch1) C::template half<F>(rec + w.rec_words, lane, f, row, ctx, at + 16 * C::T * C::TERMS);
            __syncwarp();
        }
        if (lane == 0) mbar_arrive(&sh.rec_empty[rr.stage]);
        if (mine) {
            tmem_wait_st();
            tc_fence_before_sync();
            __syncwarp();
        }
        if (lane == 0) mbar_arrive(&sh.a_full[ar.stage]);
        rr.step(a.rec_stages);
        ar.step(a.a_stages);   // the other half's stage, then this half's next one
        ar.step(a.a_stages);
    }
    return true;
}

// The issuer's share of one chunk of T octets: 4T slabs of 16 columns of K, 2T per decoder half.  An elected lane issues runs of
// instructions between the waits; the runs are unrolled and their operands made warp-uniform with a shuffle, so that descriptors
// stay in uniform registers (an issue inside a rolled loop, operands in lane registers, took 200 cycles, more than its 128
// tensor cycles for N = 256).  tile_issue: activation stages of 64 columns.  tile_issue_step: small N, an activation stage holds
// the n <= 2 chunks of a step and each half is one run; with a wait costing 200 cycles, what counts there is their number.
// XTERMS 2: activations in two terms; the product of two second terms is left out (2^-22).
template <int TERMS, int XTERMS>
__device__ __forceinline__ void tile_mma(uint32_t td, uint32_t at, uint32_t second_at, uint64_t bdesc, uint32_t second_b, uint32_t idesc, bool acc) {
    tc_mma_f16_ts(td, at, bdesc, idesc, acc);
    if constexpr (TERMS == 2) tc_mma_f16_ts(td, at + second_at, bdesc, idesc, true);
    if constexpr (XTERMS == 2) tc_mma_f16_ts(td, at, bdesc + (uint64_t)(second_b >> 4), idesc, true);
}

template <int TERMS, int XTERMS, int T>
__device__ __forceinline__ bool tile_issue_step(const TileArgs& a, TileShared& sh, TileRing& ar, TileRing& xr, unsigned char* x_ring, uint32_t x_pitch, uint32_t tmem_a,
                                                uint32_t td, uint32_t idesc, bool acc, int n) {
    if (!tile_wait(&sh.x_full[xr.stage], xr.phase)) return false;
    const uint32_t xb = __shfl_sync(0xffffffffu, smem_u32(x_ring) + (uint32_t)(xr.stage * a.x_stage_bytes), 0);
#pragma unroll
    for (int f = 0; f < 2; ++f) {
        if (!tile_wait(&sh.a_full[ar.stage], ar.phase)) return false;
        tc_fence_after_sync();
        const uint32_t at = __shfl_sync(0xffffffffu, tmem_a + (uint32_t)(ar.stage * a.a_cols), 0);
        if (elect_one()) {
#pragma unroll
            for (int g = 0; g < 2; ++g)
                if (g < n) {
#pragma unroll
                    for (int i = 0; i < 2 * T; ++i) {
                        const int sl = (g * 2 + f) * 2 * T + i;
                        const uint64_t bdesc = smem_desc_sw128(xb + (uint32_t)((sl >> 2) * XTERMS) * x_pitch) + (uint64_t)(2 * (sl & 3));
                        tile_mma<TERMS, XTERMS>(td, at + (uint32_t)(16 * T * g * TERMS + 8 * i), 16u * T, bdesc, x_pitch, idesc, sl > 0 || acc);
                    }
                }
            if (f == 1) tc_commit(&sh.x_empty[xr.stage]);
            tc_commit(&sh.a_empty[ar.stage]);
        }
        __syncwarp();
        ar.step(a.a_stages);
    }
    xr.step(a.x_stages);
    return true;
}

template <int TERMS, int XTERMS, int T>
__device__ __forceinline__ bool tile_issue(const TileArgs& a, TileShared& sh, TileRing& ar, TileRing& xr, unsigned char* x_ring, uint32_t x_pitch, uint32_t tmem_a, uint32_t td, uint32_t idesc,
                                           bool acc) {
    auto run = [&](auto first_c, auto len_c, bool x_done) {   // slabs [first, first + len) of the chunk, all in half first / 2T
        constexpr int FIRST = decltype(first_c)::value, LEN = decltype(len_c)::value, H0 = FIRST % (2 * T);
        const uint32_t at = __shfl_sync(0xffffffffu, tmem_a + (uint32_t)(ar.stage * a.a_cols), 0);
        const uint64_t bdesc = smem_desc_sw128(__shfl_sync(0xffffffffu, smem_u32(x_ring) + (uint32_t)(xr.stage * a.x_stage_bytes), 0));
        if (elect_one()) {
#pragma unroll
            for (int i = 0; i < LEN; ++i) {
                const int sl = FIRST + i;
                tile_mma<TERMS, XTERMS>(td, at + (uint32_t)(8 * (H0 + i)), 16u * T, bdesc + (uint64_t)(2 * (sl & 3)), x_pitch, idesc, sl > 0 || acc);
            }
            if (x_done) tc_commit(&sh.x_empty[xr.stage]);
            if (H0 + LEN == 2 * T) tc_commit(&sh.a_empty[ar.stage]);
        }
        __syncwarp();
        if (x_done) xr.step(a.x_stages);
        if (H0 + LEN == 2 * T) ar.step(a.a_stages);
    };
    auto wait_a = [&]() {
        const bool ok = tile_wait(&sh.a_full[ar.stage], ar.phase);
        tc_fence_after_sync();
        return ok;
    };
    auto wait_x = [&]() { return tile_wait(&sh.x_full[xr.stage], xr.phase); };
    using std::integral_constant;
    constexpr int ODD = T & 1;   // an odd number of octets: the middle 64-column slab belongs to both halves
    bool ok = wait_a();
    auto atoms = [&](auto first_c, auto count_c) {
        constexpr int A0 = decltype(first_c)::value, N = decltype(count_c)::value;
        tile_static_for<N>([&](auto i_c) {
            if (ok && (ok = wait_x())) run(integral_constant<int, 4 * A0 + 4 * decltype(i_c)::value>{}, integral_constant<int, 4>{}, true);
        });
    };
    atoms(integral_constant<int, 0>{}, integral_constant<int, T / 2>{});
    if constexpr (ODD) {
        if (ok && (ok = wait_x())) run(integral_constant<int, 2 * T - 2>{}, integral_constant<int, 2>{}, false);
        if (ok && (ok = wait_a())) run(integral_constant<int, 2 * T>{}, integral_constant<int, 2>{}, true);
    } else {
        ok = ok && wait_a();
    }
    // remaining whole slabs of the second half
    tile_static_for<T / 2>([&](auto i_c) {
        if (ok && (ok = wait_x())) run(integral_constant<int, 4 * (T / 2 + ODD) + 4 * decltype(i_c)::value>{}, integral_constant<int, 4>{}, true);
    });
    return ok;
}

// Sets::dispatch(w, f) calls f(Codec{}) for the codec of a cohort; Sets::ctx describes the codec context (lattice tables);
// Sets::XTERMS: f16 terms per activation (2: a 64-column slab of second terms follows every slab of first terms).
// GLU: the gated epilogue (TileArgs::glu).  1024 in the launch bound holds the kernel to 64 registers, which leaves room on the
// SM for the CTAs of the kernel before it.
template <class Sets, bool GLU>
__global__ void __launch_bounds__(1024, 1) tile_tc_kernel(const __grid_constant__ TileArgs a) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ TileShared sh;
    unsigned char* x_ring = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const uint32_t x_stage_bytes = (uint32_t)a.x_stage_bytes;
    unsigned char* rec_ring = x_ring + (size_t)a.x_stages * x_stage_bytes;
    unsigned char* ctx = rec_ring + (size_t)a.rec_stages * a.rec_stage_bytes;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    if (tid == 0) {
        for (int i = 0; i < kTileRecStages; ++i) { mbar_init(&sh.rec_full[i], 1); mbar_init(&sh.rec_empty[i], kTileDecoders); }
        for (int i = 0; i < kTileXStages; ++i) { mbar_init(&sh.x_full[i], 1); mbar_init(&sh.x_empty[i], 1); }
        for (int i = 0; i < kTileAStages; ++i) { mbar_init(&sh.a_full[i], kTileDecoders / 2); mbar_init(&sh.a_empty[i], 1); }
        for (int i = 0; i < kTileSegs; ++i) { mbar_init(&sh.seg_full[i], 1); mbar_init(&sh.seg_empty[i], kTileDecoders + kTileEpilogue + 2); }
        for (int i = 0; i < 2; ++i) { mbar_init(&sh.d_full[i], 1); mbar_init(&sh.d_empty[i], kTileEpilogue); }
        mbar_init(&sh.drain, 1);
        for (int i = 0; i < 2; ++i) mbar_init(&sh.sum_full[i], 1);
        sh.fin[0].parts = sh.fin[1].parts = 0;
        sh.failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kTileWarpMma) tmem_alloc(&sh.tmem, 512u);
    Sets::ctx_init(ctx, a, tid, kTileThreads);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t tmem_d = sh.tmem, tmem_a = tmem_d + (uint32_t)(a.d_bufs * a.d_cols);

    // Weights are constants: the record loader of a plain product fills its ring and the decoders theirs before the previous
    // kernel has finished (each waits for it before it could block on what depends on it); all else waits here.
    if (warp >= kTileDecoders && (warp != kTileWarpRec || a.tile_bounds != nullptr)) asm volatile("griddepcontrol.wait;" ::: "memory");

    TileSeg s;
    TileRing sr;
    // The next stretch; false at the end or after a failure (ok).
    auto next = [&](bool& ok) {
        ok = tile_wait(&sh.seg_full[sr.stage], sr.phase);
        if (!ok) return false;
        s = sh.seg[sr.stage];
        return s.parts != 0;
    };
    auto seg_done = [&]() {
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh.seg_empty[sr.stage]);
        sr.step(kTileSegs);
    };
    if (warp < kTileDecoders) {
        // -------- decoders: row-block 2 (warp & 3) + ((warp >> 2) & 1) of the tile, half (warp >> 3) of the chunk --------
        const int rbl = 2 * (warp & 3) + ((warp >> 2) & 1), f = warp >> 3;
        const uint32_t taddr = tmem_a + ((uint32_t)(rbl * 16) << 16);
        TileRing rr, ar;
        if (f) ar.step(a.a_stages);
        bool ok = true;
        int runway = (a.a_stages - f + 1) / 2;   // this half's stages of the ring
        while (ok && next(ok)) {
            const uint4* consts = sh.rowc[sr.stage];
            uint64_t* done = &sh.seg_empty[sr.stage];
            Sets::dispatch(a.pools[s.pool], [&](auto codec) {
                using C = decltype(codec);
                if (C::SPLIT || !f) ok = tile_decode<C, 0>(a, sh, s, rec_ring, ctx, rr, ar, rbl, f, lane, taddr, consts, done, runway);
                else ok = tile_decode<C, 1>(a, sh, s, rec_ring, ctx, rr, ar, rbl, f, lane, taddr, consts, done, runway);
            });
            sr.step(kTileSegs);
        }
        if (!ok) sh.failed = 1;
    } else if (warp < kTileWarpMma) {
        // -------- epilogue: lane = row of the warp's quarter of the tile --------
        const int quarter = warp & 3, row_l = quarter * 32 + lane;
        TileRing dr;
        bool ok = true;
        for (int buf = 0; ok && next(ok); buf ^= 1) {
            const int row = s.row0 + row_l;
            const bool row_ok = row < s.row_limit;
            const float undo = row_ok ? __uint_as_float(sh.rowc[sr.stage][row_l].z) * a.lut_undo : 0.f;
            seg_done();
            for (int i = tid - kTileDecoders * 32; i < s.ncols; i += kTileEpilogue * 32)
                sh.col[buf][i] = make_int2(__float_as_int(__ldcg(a.x_down + s.tok0 + i)), a.scatter ? __ldcg(a.pair_order + s.tok0 + i) : s.tok0 + i);
            ok = tile_epilogue_all(tile_wait(&sh.d_full[dr.stage], dr.phase));
            if (!ok) break;
            tc_fence_after_sync();
            const uint32_t td = tmem_d + (uint32_t)(dr.stage * a.d_cols) + ((uint32_t)(quarter * 32) << 16);
            // finished sums of columns cb .. cb + 7, this lane's row
            auto put8 = [&](int cb, const float (&v)[8]) {
                if constexpr (!GLU && Sets::ONE) {   // (the all-cohort expert kernel has few columns per tile: the second form cost it 5 %)
                    // Whole eights of neighbouring tokens: a running pointer.  One warp per scheduler writes while nothing else can
                    // use the only accumulator of N > 128, so its instructions count: with a 64-bit product and a check for
                    // every element, 2010 tokens through NINT4 8412 x 1112 took 82 us instead of 69.
                    if (!a.scatter && s.ncols - cb >= 8) {
                        if (!row_ok) return;
                        float f[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) f[i] = v[i] * (undo * __int_as_float(sh.col[buf][cb + i].x));
                        const size_t at = (size_t)(s.tok0 + cb) * a.ldy + row;
                        if (a.y_dtype == 0 /* MFQB_F32 */) {
                            float* y = reinterpret_cast<float*>(a.y) + at;
#pragma unroll
                            for (int i = 0; i < 8; ++i, y += a.ldy) st_global(y, f[i]);
                        } else {
                            __nv_bfloat16* y = reinterpret_cast<__nv_bfloat16*>(a.y) + at;
#pragma unroll
                            for (int i = 0; i < 8; ++i, y += a.ldy) st_global(y, __float2bfloat16_rn(f[i]));
                        }
                        return;
                    }
                }
                int2 col[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) col[i] = sh.col[buf][cb + i];
                int n = row_ok ? s.ncols - cb : 0;
                if constexpr (GLU) {   // gate rows are lanes 0-15 of the warp, their up rows lanes 16-31
                    if (lane >= 16) n = 0;
                    const int half = (row >> 5) * 16 + (row & 15);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float f = v[i] * (undo * __int_as_float(col[i].x)), up = __shfl_xor_sync(0xffffffffu, f, 16), o = tile_gated(f, up);
                        if (i < n) {
                            if (a.y_dtype == 0 /* MFQB_F32 */) st_global(reinterpret_cast<float*>(a.y) + (size_t)col[i].y * a.ldy + half, o);
                            else st_global(reinterpret_cast<__nv_bfloat16*>(a.y) + (size_t)col[i].y * a.ldy + half, __float2bfloat16_rn(o));
                        }
                    }
                    return;
                }
                if (a.y_dtype == 0 /* MFQB_F32 */) {
                    float* y = reinterpret_cast<float*>(a.y) + row;
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        if (i < n) st_global(y + (size_t)col[i].y * a.ldy, v[i] * (undo * __int_as_float(col[i].x)));
                } else {
                    __nv_bfloat16* y = reinterpret_cast<__nv_bfloat16*>(a.y) + row;
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        if (i < n) st_global(y + (size_t)col[i].y * a.ldy, __float2bfloat16_rn(v[i] * (undo * __int_as_float(col[i].x))));
                }
            };
            if (!Sets::ONE || s.parts == 1) {   // (the all-cohort expert kernel shares no tiles)
                for (int cb = 0; cb < s.ncols; cb += 16) {
                    uint32_t r[16];
                    tmem_ld16(td + (uint32_t)cb, r);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        float v[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[8 * h + i]);
                        put8(cb + 8 * h, v);
                    }
                }
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.d_empty[dr.stage]);
            } else if constexpr (Sets::ONE) {
                // this CTA's part of a tile that others share
                float* mine = tile_part(a, s.slot0, (int)blockIdx.x - s.slot0) + row_l;
                for (int cb = 0; cb < s.ncols; cb += 16) {
                    uint32_t r[16];
                    tmem_ld16(td + (uint32_t)cb, r);
#pragma unroll
                    for (int i = 0; i < 16; ++i) st_global(mine + (size_t)(cb + i) * kTileRows, __uint_as_float(r[i]));
                }
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.d_empty[dr.stage]);
                if (s.last) sh.row_factor[row_l] = undo;
                const int2 g = tile_group(s);
                const TileSum sum(a, s, g.x, 1, g.y);
                __threadfence();
                asm volatile("bar.sync 1, 128;" ::: "memory");
                if (warp == kTileDecoders && lane == 0) {
                    unsigned* counter = a.counters + s.slot0 + g.x;
                    if (atomicAdd(counter, 1u) == (unsigned)(g.y - 1)) {   // nearly always with the last stretch: part 0 of a tile is one
                        __threadfence();
                        if (s.last) sum.request_first(a, sh, reinterpret_cast<float*>(x_ring));   // nothing uses the rings' memory any more
                        sh.fin[s.last ? 0 : 1] = s;
                        sh.fin_col = buf;
                    }
                }
            }
            dr.step(a.d_bufs);
        }
        if (!ok) sh.failed = 1;
    } else if (warp == kTileWarpMma) {
        // -------- mma issuer: the warp stays together, an elected lane issues --------
        const uint32_t idesc = instr_desc_f16(kTileRows, a.n_mma);
        TileRing ar, xr, dr;
        bool ok = true;
        while (ok && next(ok)) {
            seg_done();
            const int t8 = a.pools[s.pool].t8;
            if (!tile_wait(&sh.d_empty[dr.stage], dr.phase ^ 1u)) { ok = false; break; }
            tc_fence_after_sync();
            // Everything that the products' operands are made of is made warp-uniform here, and the loop over chunks runs inside the
            // choice of T: beside busy decoders an instruction of this warp takes some ten clocks (NINT4 in groups of 32
            // 14336 x 4096, 512 rows: 68.3 us, 64.2 with this form; NINT6 28672 x 4096, 64 rows: 41.6, 38.8).
            const int n = __shfl_sync(0xffffffffu, s.ch1 - s.ch0, 0);
            const uint32_t td = __shfl_sync(0xffffffffu, tmem_d + (uint32_t)(dr.stage * a.d_cols), 0), ta = __shfl_sync(0xffffffffu, tmem_a, 0);
            const uint32_t x_pitch = __shfl_sync(0xffffffffu, (uint32_t)((s.ncols + 7) & ~7) * 128u, 0);
            auto issue = [&](auto t_c) {
                constexpr int T = decltype(t_c)::value;
                if (a.x_whole)
                    for (int c = 0; c < n && ok; c += a.step) ok = tile_issue_step<Sets::TERMS, Sets::XTERMS, T>(a, sh, ar, xr, x_ring, x_pitch, ta, td, idesc, c > 0, min(a.step, n - c));
                else
                    for (int c = 0; c < n && ok; ++c) ok = tile_issue<Sets::TERMS, Sets::XTERMS, T>(a, sh, ar, xr, x_ring, x_pitch, ta, td, idesc, c > 0);
            };
            switch (t8) {
                case 2: issue(std::integral_constant<int, 2>{}); break;
                case 3: issue(std::integral_constant<int, 3>{}); break;
                case 4: issue(std::integral_constant<int, 4>{}); break;
                case 5: issue(std::integral_constant<int, 5>{}); break;
                case 6: issue(std::integral_constant<int, 6>{}); break;
                default: issue(std::integral_constant<int, 8>{}); break;
            }
            if (ok && elect_one()) tc_commit(&sh.d_full[dr.stage]);
            __syncwarp();
            dr.step(a.d_bufs);
        }
        if (!ok) {
            sh.failed = 1;
            if (elect_one()) tc_commit(&sh.drain);   // what was issued still reads the rings and the tensor memory
            tile_wait(&sh.drain, 0);
        }
    } else if (warp == kTileWarpRec) {
        // -------- record loader: also finds the stretches and hands them to the other warps with their row constants --------
        TileRing rr;
        bool ok = true, more = true;
        int issued = 0, cursor = tile_first(a);
        while (ok && more) {
            more = tile_next(a, cursor, s);
            if (!tile_wait(&sh.seg_empty[sr.stage], sr.phase ^ 1u)) { ok = false; break; }
            const NintDevB& w = a.pools[more ? s.pool : 0];
            if (elect_one()) {
                if (!more) s.parts = 0;
                sh.seg[sr.stage] = s;
                const uint32_t bytes = more ? (uint32_t)s.nrb * 16u * 16u : 0u;
                mbar_arrive_expect_tx(&sh.seg_full[sr.stage], bytes);
                if (more) bulk_load(sh.rowc[sr.stage], w.rowc + (size_t)s.rb0 * 16, bytes, &sh.seg_full[sr.stage]);
            }
            __syncwarp();
            sr.step(kTileSegs);
            if (!more) break;
            const uint32_t pitch = (uint32_t)(a.step * w.rec_words) * 4u;
            const size_t rb_words = (size_t)w.nchunks * w.rec_words;
            const uint32_t* src = w.items + (size_t)s.rb0 * rb_words + (size_t)s.ch0 * w.rec_words;
            for (int ch = s.ch0; ch < s.ch1; ch += a.step, src += (size_t)a.step * w.rec_words) {
                const uint32_t bytes = (uint32_t)(min(a.step, s.ch1 - ch) * w.rec_words) * 4u;   // a row-block's records of a step are neighbours
                if (issued == a.rec_stages) asm volatile("griddepcontrol.wait;" ::: "memory");
                if (!tile_wait(&sh.rec_empty[rr.stage], rr.phase ^ 1u)) { ok = false; break; }
                if (elect_one()) {
                    mbar_arrive_expect_tx(&sh.rec_full[rr.stage], bytes * (uint32_t)s.nrb);
                    unsigned char* dst = rec_ring + (size_t)rr.stage * a.rec_stage_bytes;
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        if (i < s.nrb) bulk_load(dst + i * pitch, src + (size_t)i * rb_words, bytes, &sh.rec_full[rr.stage]);
                }
                __syncwarp();
                rr.step(a.rec_stages);
                ++issued;
            }
        }
        if (!ok) {
            sh.failed = 1;
            if (issued > 0) tile_wait(&sh.seg_full[(sr.stage + kTileSegs - 1) % kTileSegs], sr.phase ^ (sr.stage == 0 ? 1u : 0u));
            for (int i = 0; i < min(issued, a.rec_stages); ++i) tile_wait(&sh.rec_full[(rr.stage + a.rec_stages - 1 - i) % a.rec_stages], rr.phase ^ (i >= rr.stage ? 1u : 0u));
        }
    } else {
        // -------- activation loader --------
        TileRing xr;
        bool ok = true;
        int issued = 0;
        while (ok && next(ok)) {
            seg_done();
            const int t8 = a.pools[s.pool].t8, atoms = a.x_whole ? a.step * t8 : 1;
            const uint32_t pitch = (uint32_t)((s.ncols + 7) & ~7) * 128u * (uint32_t)Sets::XTERMS;
            const unsigned char* src = a.x + s.x_off + (size_t)s.ch0 * t8 * pitch;
            for (int at = s.ch0 * t8; at < s.ch1 * t8; at += atoms, src += (size_t)atoms * pitch) {
                const uint32_t bytes = pitch * (uint32_t)min(atoms, s.ch1 * t8 - at);
                if (!tile_wait(&sh.x_empty[xr.stage], xr.phase ^ 1u)) { ok = false; break; }
                if (elect_one()) {
                    mbar_arrive_expect_tx(&sh.x_full[xr.stage], bytes);
                    bulk_load(x_ring + (size_t)xr.stage * x_stage_bytes, src, bytes, &sh.x_full[xr.stage]);
                }
                __syncwarp();
                xr.step(a.x_stages);
                ++issued;
            }
        }
        if (!ok) {
            sh.failed = 1;
            for (int i = 0; i < min(issued, a.x_stages); ++i) tile_wait(&sh.x_full[(xr.stage + a.x_stages - 1 - i) % a.x_stages], xr.phase ^ (i >= xr.stage ? 1u : 0u));
        }
    }
    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    if (warp == kTileWarpMma) {
        tc_fence_after_sync();
        tmem_free(tmem_d, 512u);
        if (lane == 0 && sh.failed) atomicExch(a.error, MFQB_ERR_TIMEOUT);
    }
    if constexpr (Sets::ONE) {
        if (!sh.failed && (sh.fin[0].parts | sh.fin[1].parts)) {
            float* stage = reinterpret_cast<float*>(x_ring);
            bool ok = true;
            uint32_t phase = 0u;
            if (sh.fin[0].parts) ok = tile_finish<GLU>(a, sh, sh.fin[0], sh.col[sh.fin_col], stage, phase);
            if (ok && sh.fin[1].parts) {   // its tables have made room for later stretches'
                const TileSeg& t = sh.fin[1];
                __syncthreads();
                for (int r = tid; r < kTileRows; r += kTileThreads)
                    sh.row_factor[r] = t.row0 + r < t.row_limit ? __uint_as_float(__ldg(&a.pools[0].rowc[(size_t)t.rb0 * 16 + r]).z) * a.lut_undo : 0.f;
                for (int c = tid; c < t.ncols; c += kTileThreads) sh.col[0][c].x = __float_as_int(__ldcg(a.x_down + t.tok0 + c));
                if (tid == 0) TileSum(a, t, tile_group(t).x, 1, tile_group(t).y).request_first(a, sh, stage);
                __syncthreads();
                ok = tile_finish<GLU>(a, sh, t, sh.col[0], stage, phase);
            }
            if (!ok && tid == 0) atomicExch(a.error, MFQB_ERR_TIMEOUT);
        }
    }
}

}  // namespace mfqb
