// Products of a packed weight with a few activation rows (at most 16) on mma.sync, weights decoded in registers.
//
//   y[token, n] = sum_k x[token, k] * W[n, k]
//
// For a handful of tokens the tensor-memory tile kernel (tile_tc.cuh) spends its time on its pipeline: its roles pass every chunk
// on through barriers whose round trips take 100 to 300 clocks each, and a tile of 128 rows is shared by several CTAs that add
// their sums up through L2.  Here a warp does everything for a 16-row record by itself: it loads the record's words into
// registers one record ahead (asked into L2 four ahead: NINT6 28672 x 4096, 8 rows 26.6 us; not at all 28.9, eight 28.9), turns
// them into A operands -- in byte-lane fragment order two registers ARE rows q, q + 8 of a 16 x 16 operand -- and multiplies on
// mma.m16n8k16.  There is no barrier between the first and the last record of a CTA.
//   * rows_x_kernel writes the activations once as B operands (f16, group sums beside them); a CTA brings its slice of K into
//     shared memory with bulk copies.
//   * A CTA has a slice of K (mostly all of it) and some row-blocks; their records are one list that its 20 warps share out
//     evenly, in the order of K, so a row-block's partial sums are few and added in a fixed order: a product has the same bits in
//     every call.  20 warps of 96 registers leave room for a CTA of rows_x_kernel, which is there when the predecessor ends.
//
// Arithmetic.  An integer below 2048 in the low bits of a half IS the f16 number n 2^-24, so a masked field needs no conversion:
// one multiplication (centred widths: one fused multiply-add) gives (q - mid) ss 2^-20, exact below 2^11: widths 2 to 5 with the
// usual sub-scales are exact throughout (1e-6 on the product, float32 sums), six are rounded once (1.3e-4; the tile
// kernel's two roundings 2.4e-4).  What the offsets add, -nm sm X_g and for centred widths ns mid ss X_g with the group sums
// X_g of the activations in two f16 terms, is one more k-step whose A operand are the record's scale bytes as they lie.
//
// Measured (us, 16 / 8 rows; in brackets the tile kernel): NINT4 4096 x 4096 9.2 / 7.7 (13.1 / 12.8), 6144 x 4096 10.6 / 9.0
// (14.4), 28672 x 4096 25.2 / 21.0 (28.3), NINT6 28672 x 4096 31.7 / 26.6 (32.1), 4096 x 14336 19.6 / 16.9 (20.7), NINT3 14336 x
// 4096 16.0 / 13.9 (20.1), NINT5 in groups of 28 5000 x 2888 10.2 / 9.1 (17.0), 28672 x 4096 33 / 28 (72), NVQ3 17408 x 5120 8
// rows 21.0 (23.6), 5120 x 5120 12.1 (20.1); 3 rows (in brackets the integer kernel): NINT4 6144 x 4096 8.9 (16.4), NINT3 14336 x
// 4096 13.8 (21.9).  Bound by the latency of the chain inside a warp (scales, codes, products, sums): some 390 instructions a
// record (16 rows x 192 columns x 16 tokens) at 2.2 of 4 a clock from 20 warps, no pipe above 40 %, memory at 35 %.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "common.h"
#include "lane_unit.h"
#include "nint_blayout.h"
#include "rows_mma.h"
#include "tc05.cuh"
#include "tile_tc.h"

namespace mfqb {

constexpr int kRowsWarps = 20, kRowsThreads = 32 * kRowsWarps;
constexpr int kRowsSlot = 20;      // floats of a token's 16 rows in a slot: 20 keeps a fragment's stores off each other's banks
constexpr int kRowsChunks = 64;    // most chunks of a slice
constexpr int kRowsPass = 24;      // most row-blocks that a CTA adds up at a time
constexpr int kRowsSlices = 8;     // most slices of K
constexpr int kRowsAhead = 4;      // records of a warp that are asked into L2 ahead of the one in registers

struct RowsArgs {
    NintDevB w;
    uint16_t lut16[16];        // lattice: f16 state scales, normalised by a power of two
    float undo;                // its inverse, and that of the weights' common factor
    const unsigned char* x;    // activation fragments, see rows_x_kernel
    void* y;
    int m, ldy, y_dtype, glu;
    int tiles, slices;         // CTA = (row-block tile, slice of K)
    int pass_rb;               // row-blocks a CTA adds up at a time
    int x_bytes;               // shared memory of the activations
    float* parts;              // slices > 1: [grid][pass row-blocks][m][16]
    unsigned* counters;        // slices > 1: arrivals per tile, cleared by rows_x_kernel
    int* error;
};

// What rows_x_kernel writes and where: per chunk the slabs of token fragments, then a float factor per token.
struct RowsXArgs {
    const __nv_bfloat16* x;
    int m, k, gs, nt, nchunks;
    float factor;              // of the group sums
    unsigned char* out;
    unsigned* counters;
    int n_counters;
};
// Factor of the group sums: what the widths from five bits on, centred, multiply by ss, else only what keeps them f16 numbers.
constexpr __host__ __device__ float rows_x_factor(int bits) { return bits >= 5 ? (float)(1 << (bits - 1)) / 1048576.f : 1.f / 4096.f; }
constexpr __host__ __device__ int rows_chunk_bytes(int t8, int nt) { return (4 * t8 + 1) * 256 * nt + 32 * nt; }

__device__ __forceinline__ __half2 rows_h2(uint32_t v) { return *reinterpret_cast<const __half2*>(&v); }
__device__ __forceinline__ uint32_t rows_u32(__half2 v) { return *reinterpret_cast<const uint32_t*>(&v); }
__device__ __forceinline__ uint32_t rows_ldg(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.global.nc.L1::no_allocate.b32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint4 rows_ldg4(const uint32_t* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void rows_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// the first product of a sum
__device__ __forceinline__ void rows_mma0(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
template <int N, int I = 0, class Fn>
__device__ __forceinline__ void rows_static_for(Fn&& f) {
    if constexpr (I < N) {
        f(std::integral_constant<int, I>{});
        rows_static_for<N, I + 1>(f);
    }
}

// Scalar codes.  An integer n < 2048 in the low bits of a half IS the f16 number n 2^-24, so a masked field needs no conversion:
// field q at bit pos is q 2^(pos - 24), times d = ss 2^(4 - pos) gives q ss 2^-20 with one rounding (none below 2^11).  Widths
// from five bits on are centred, (q - mid) ss 2^-20, by the addend of the same instruction; mid ss X_g comes back through one
// more k-step (S1).
template <int BITS, int T_>
struct RowsNint {
    static constexpr int T = T_, MID = BITS >= 5 ? 1 << (BITS - 1) : 0;
    static constexpr bool S1 = BITS >= 5, S2 = true, TABLE = false;
    using BU = ByteUnit<BITS>;
    static constexpr int WC = BU::words_for(8 * T), SW = 2;
    // Wide records come into registers by halves (the second half's registers start on a word): a lane's words of a whole record
    // beside the sums of two activation tiles spilled (16 rows 28672 x 4096, NINT6-32 34.3 us, by halves 29.6; NINT6-48 48.6 and 38.6).
    static constexpr bool HALVES = WC >= 24 && (4 * T) % BU::NP == 0;
    static constexpr int CW = HALVES ? WC / 2 : WC, REGS = HALVES ? 4 * T : 8 * T;   // words in registers, registers decoded from them
    // last register that reads word w: a unit's words are all read by its last register where fields are rebuilt from left-over bits
    static constexpr int last_reg(int w) {
        const int unit = w / BU::U, tt = BU::EXTRA ? BU::NP - 1 : BU::F * (w % BU::U + 1) - 1, r = unit * BU::NP + tt;
        return r < REGS ? r : REGS - 1;
    }
    __host__ __device__ static constexpr int pos(int a) { return BITS == 2 ? 2 * a : ((BITS == 3 || BITS == 4) ? BITS * (a & 1) : 0); }
    static constexpr float X_FACTOR = rows_x_factor(BITS);
    static constexpr float OUT_MIN = 16777216.f / X_FACTOR;

    struct Scales {
        uint4 quad;          // word 0 of the lanes of this quad
        uint32_t own, min;   // word 0, word 1 of this lane
        __device__ __forceinline__ void load_late(const uint32_t* rec, int lane) {
            min = rows_ldg(rec + (WC + 1) * 32 + lane);
            if constexpr (S1) own = rows_ldg(rec + WC * 32 + lane);
        }
    };
    struct Half {
        __half2 d[4], n[4];
    };
    template <int F>
    __device__ static __forceinline__ void half(const Scales& sc, int lane, const unsigned char*, Half& o) {
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const int h = a >> 1;
            const uint32_t word = F == 0 ? (h ? sc.quad.y : sc.quad.x) : (h ? sc.quad.w : sc.quad.z);
            // bytes: (row q, even group), (q, odd), (q + 8, even), (q + 8, odd); this lane's group is the odd one for c >= 2
            const uint32_t sel = (a & 1) ? ((lane & 2) ? 0x4343u : 0x4242u) : ((lane & 2) ? 0x4141u : 0x4040u);
            const __half2 s1024 = rows_h2(__byte_perm(word, 0x64646464u, sel));
            const float k = (float)(1 << 4) / (float)(1 << pos(a));
            o.d[a] = __hfma2(s1024, __float2half2_rn(k), __float2half2_rn(-1024.f * k));
            if constexpr (MID != 0) o.n[a] = __hmul2(o.d[a], __float2half2_rn(-(float)MID / 16777216.f * (float)(1 << pos(a))));
        }
    }
    template <int R>
    __device__ static __forceinline__ void weights(const uint32_t (&code)[CW], const Half& s, uint32_t, const unsigned char*, uint32_t& even, uint32_t& odd, uint32_t) {
        constexpr int P = pos(R % 4), TT = R % REGS % BU::NP, UNIT = R % REGS / BU::NP, A = R & 3;
        constexpr uint32_t M = ((1u << BITS) - 1u) << P, MASK = M | (M << 16);
        uint32_t v;
        if constexpr (TT < BU::U * BU::F) {
            static_assert((TT % BU::F) * BITS == P, "field position");
            v = code[UNIT * BU::U + TT / BU::F];
        } else {
            uint32_t u[BU::U];
#pragma unroll
            for (int i = 0; i < BU::U; ++i) u[i] = code[UNIT * BU::U + i];
            v = BU::at(u, TT) << P;
        }
        const __half2 e = rows_h2(v & MASK), o = rows_h2((v >> 8) & MASK);
        if constexpr (MID != 0) {
            even = rows_u32(__hfma2(e, s.d[A], s.n[A]));
            odd = rows_u32(__hfma2(o, s.d[A], s.n[A]));
        } else {
            even = rows_u32(__hmul2(e, s.d[A]));
            odd = rows_u32(__hmul2(o, s.d[A]));
        }
    }
    __device__ static void ctx_init(unsigned char*, const RowsArgs&, int) {}
};


// Lattice vectors: a field is a look-up in the signed table (shared memory, codes biased by 128).  Plain records: (code + 128)
// 2^-24 times 16 ss less 128 of it, integers below 2048, exact.  Joint-codebook records: code times the state's f16 scale, for
// records whose products are f16 numbers (tile_terms 1).
template <int IB, bool JSC>
struct RowsNvq {
    static constexpr int T = 3, FB = IB + 4, WC = (24 * FB + 31) / 32, SW = 1, CW = WC;
    static constexpr bool HALVES = false;
    static constexpr int last_reg(int w) { return (32 * w + 31) / FB < 23 ? (32 * w + 31) / FB : 23; }
    static constexpr bool S1 = false, S2 = false, TABLE = true;
    static constexpr float OUT_MIN = 0.f;
    static constexpr uint32_t OFFMASK = ((1u << FB) - 1u) << 2;   // a field as a byte offset into the table
    __device__ static void ctx_init(unsigned char* ctx, const RowsArgs& a, int tid) {
        const uint4* src = reinterpret_cast<const uint4*>(a.w.table);
        for (int i = tid; i < a.w.table_words / 4; i += kRowsThreads) {
            uint4 v = __ldg(src + i);
            v.x ^= 0x80808080u; v.y ^= 0x80808080u; v.z ^= 0x80808080u; v.w ^= 0x80808080u;
            reinterpret_cast<uint4*>(ctx + 64)[i] = v;
        }
        if (tid < 16) reinterpret_cast<uint16_t*>(ctx)[tid] = a.lut16[tid];
    }
    struct Scales {
        uint4 quad;
        uint32_t own, min;
        __device__ __forceinline__ void load_late(const uint32_t* rec, int lane) {
            if constexpr (JSC) own = rows_ldg(rec + WC * 32 + lane);
        }
    };
    struct Half {
        __half2 d[4], n[4];
    };
    template <int F>
    __device__ static __forceinline__ void half(const Scales& sc, int lane, const unsigned char* ctx, Half& o) {
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const int h = a >> 1;
            const uint32_t word = F == 0 ? (h ? sc.quad.y : sc.quad.x) : (h ? sc.quad.w : sc.quad.z);
            const uint32_t st = (word >> (8 * ((lane >> 1) & 1) + 16 * (a & 1))) & 15u;
            if constexpr (JSC) {
                o.d[a] = __half2half2(__ushort_as_half(reinterpret_cast<const uint16_t*>(ctx)[st]));
            } else {
                o.d[a] = __hfma2(rows_h2(st * 0x10001u | 0x64006400u), __float2half2_rn(16.f), __float2half2_rn(-16384.f));
                o.n[a] = __hmul2(o.d[a], __float2half2_rn(-128.f / 16777216.f));
            }
        }
    }
    template <int R>
    __device__ static __forceinline__ void weights(const uint32_t (&code)[CW], const Half& s, uint32_t own, const unsigned char* ctx, uint32_t& even, uint32_t& odd, uint32_t bank_bytes) {
        constexpr int POS = R * FB, WI = POS >> 5, SH = POS & 31, A = R & 3;
        uint32_t off;
        if constexpr (SH + FB <= 32) off = (SH >= 2 ? code[WI] >> (SH >= 2 ? SH - 2 : 0) : code[WI] << (SH < 2 ? 2 - SH : 0)) & OFFMASK;
        else off = __funnelshift_r(code[WI], code[WI + 1], SH - 2) & OFFMASK;   // a field that straddles two words starts above bit 2
        if constexpr (JSC) {
            constexpr int I = (R / 12) * 4 + (R & 3);   // the (row, group) pair of this register: its bank travels in the lane's own scale word
            off += ((own >> (8 * (I >> 1) + 4 + 2 * (I & 1))) & 3u) * bank_bytes;
        }
        const uint32_t v = *reinterpret_cast<const uint32_t*>(ctx + 64 + off);
        if constexpr (!JSC) {
            even = rows_u32(__hfma2(rows_h2(v & 0x00FF00FFu), s.d[A], s.n[A]));
            odd = rows_u32(__hfma2(rows_h2((v >> 8) & 0x00FF00FFu), s.d[A], s.n[A]));
        } else {
            const __half2 k1152 = __float2half2_rn(1152.f);
            even = rows_u32(__hmul2(__hsub2(rows_h2((v & 0x00FF00FFu) | 0x64006400u), k1152), s.d[A]));
            odd = rows_u32(__hmul2(__hsub2(rows_h2(((v >> 8) & 0x00FF00FFu) | 0x64006400u), k1152), s.d[A]));
        }
    }
};

// (2^e, 2^-e) with 2^e * max in [2^14, 2^15); (1, 1) for a zero or subnormal maximum.  A chunk with an infinity or NaN is scaled by
// NaN: every product with it is one, so all outputs of the token are (an infinity left as it is gives infinities: lattice records
// have no products with the sums, which would make NaN of it).
__device__ __forceinline__ float2 rows_x_scale(uint32_t absmax_bits) {
    int eb = (int)(absmax_bits >> 23);
    if (eb == 0) return make_float2(1.f, 1.f);
    if (eb == 255) return make_float2(__uint_as_float(0x7FC00000u), 1.f);
    eb = max(eb, 15);
    return make_float2(__uint_as_float((uint32_t)(268 - eb) << 23), __uint_as_float((uint32_t)(eb - 14) << 23));
}

// T octets of one group's columns as bf16 pairs, from slot s0 on (PART), zero past the group size and past the row.
template <int T>
struct RowsGroup {
    uint32_t v[4 * T];
    // form 2: 16-byte pieces, 1: 8-byte pieces, 0: single values (a row in shared memory is padded with zeros to whole pieces)
    template <bool SHARED, bool PART>
    __device__ __forceinline__ void load(const __nv_bfloat16* row, int k, int gs, int g, int form, bool live, int s0 = 0) {
        const int k0 = g * gs + s0;
        gs -= s0;
        if (form == 2) {
#pragma unroll
            for (int t = 0; t < T; ++t) {
                uint4 r = make_uint4(0u, 0u, 0u, 0u);
                if (live && (!PART || 8 * t < gs) && k0 + 8 * t < k) r = SHARED ? *reinterpret_cast<const uint4*>(row + k0 + 8 * t) : __ldcg(reinterpret_cast<const uint4*>(row + k0 + 8 * t));
                v[4 * t] = r.x; v[4 * t + 1] = r.y; v[4 * t + 2] = r.z; v[4 * t + 3] = r.w;
            }
        } else if (form == 1) {
#pragma unroll
            for (int t = 0; t < 2 * T; ++t) {
                uint2 r = make_uint2(0u, 0u);
                if (live && 4 * t < gs && k0 + 4 * t < k) r = SHARED ? *reinterpret_cast<const uint2*>(row + k0 + 4 * t) : __ldcg(reinterpret_cast<const uint2*>(row + k0 + 4 * t));
                v[2 * t] = r.x; v[2 * t + 1] = r.y;
            }
        } else {
#pragma unroll
            for (int i = 0; i < 4 * T; ++i) {
                const unsigned short* at = reinterpret_cast<const unsigned short*>(row) + k0 + 2 * i;
                uint32_t lo = 0u, hi = 0u;
                if (live && 2 * i < gs && k0 + 2 * i < k) lo = SHARED ? *at : __ldcg(at);
                if (live && 2 * i + 1 < gs && k0 + 2 * i + 1 < k) hi = SHARED ? at[1] : __ldcg(at + 1);
                v[i] = lo | hi << 16;
            }
        }
    }
    __device__ __forceinline__ uint32_t absmax(uint32_t m) const {   // bf16 magnitudes order like their bits
#pragma unroll
        for (int i = 0; i < 4 * T; ++i) m = max(m, max(v[i] & 0x7FFF0000u, (v[i] << 16) & 0x7FFF0000u));
        return m;
    }
};

// One group of a token's activations as B operands, by eight neighbouring lanes for the eight groups of a chunk (PARTS 2: sixteen,
// each with half of a group's octets): values scaled by a power of two per token and chunk (largest magnitude next to 2^15; exact
// for bf16 values within 2^-28 of it), the group's sum as two f16 terms, the factor's inverse. Slab 2 (f T + t) + h of a chunk
// holds octet t of groups 4 f + 2 h and the next: lane 4 q + c (token q of a tile of eight) reads quad c & 1 of group c >> 1,
// slots 0, 2 and 1, 3 in its two registers -- the order in which the decoders' byte pairs come.  Lanes are XORed with 4 h + f,
// which spreads a token's groups over the banks.
template <int T, int PARTS>
__device__ __forceinline__ void rows_x_group(const RowsGroup<(T + PARTS - 1) / PARTS>& v, unsigned char* chunk, int t, int g, int part, int nt, float factor, bool live) {
    constexpr int TP = (T + PARTS - 1) / PARTS;
    uint32_t mx = v.absmax(0u);
    for (int o = 1; o < 8 * PARTS; o <<= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (PARTS == 1 && !live) return;
    const float2 sc = rows_x_scale(mx);
    const int q = t & 7, j = t >> 3, b = g & 1, h = (g >> 1) & 1, f = g >> 2, slab = 256 * nt;
    auto at = [&](int s, int unit) { return chunk + (size_t)s * slab + (nt == 1 ? unit * 8 : unit * 16 + j * 8); };   // this token's eight bytes of a lane
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < TP; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const uint32_t u0 = v.v[4 * i + 2 * e], u1 = v.v[4 * i + 2 * e + 1];
            const float x0 = __uint_as_float(u0 << 16) * sc.x, x1 = __uint_as_float(u0 & 0xFFFF0000u) * sc.x;
            const float x2 = __uint_as_float(u1 << 16) * sc.x, x3 = __uint_as_float(u1 & 0xFFFF0000u) * sc.x;
            sum += (x0 + x1) + (x2 + x3);
            if (PARTS == 1 || (live && (T % PARTS == 0 || part * TP + i < T)))
                *reinterpret_cast<uint2*>(at(2 * (f * T + part * TP + i) + h, (4 * q + 2 * b + e) ^ (4 * h + f))) =
                    make_uint2(rows_u32(__floats2half2_rn(x0, x2)), rows_u32(__floats2half2_rn(x1, x3)));
        }
    if constexpr (PARTS == 2) sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    if (PARTS == 2 && (!live || part != 0)) return;
    sum *= factor;   // k-slots (group) and 8 + (group) of the chunk's last slab
    const __half hi = __float2half_rn(sum), lo = __float2half_rn(sum - __half2float(hi));
    unsigned char* p = at(4 * T, 4 * q + (g >> 1)) + 2 * b;
    *reinterpret_cast<__half*>(p) = hi;
    *reinterpret_cast<__half*>(p + 4) = lo;
    if (g == 0) *reinterpret_cast<float*>(chunk + (size_t)(4 * T + 1) * slab + 4 * t) = sc.y;
}

// At most 128 threads of 32 registers a CTA: it then fits beside the 20 warps of 96 registers of the kernel before it, which leave
// each of the SM's four schedulers 1024, and waits there for its end (with more it is launched after that end: 16 rows through
// NINT4 4096 x 4096 14.7 us instead of 9.2, through NINT4-48 16.2 instead of 9.3).  A CTA per chunk, a thread per (token, group)
// or, for more than four octets, two of them: 1.3 us of a product's chain (a factor per whole row, as the tile kernel has it,
// needs a pass for the maxima before: 2.8).
constexpr int rows_x_parts(int t8) { return t8 <= 4 ? 1 : 2; }
template <int T>
__global__ void __launch_bounds__(128, 16) rows_x_kernel(const __grid_constant__ RowsXArgs a) {
    constexpr int PARTS = rows_x_parts(T), LANES = 8 * PARTS, TP = (T + PARTS - 1) / PARTS;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int t = (int)(blockIdx.y * (128 / LANES) + threadIdx.x / LANES), g = threadIdx.x % LANES / PARTS, part = threadIdx.x % PARTS;
    if (blockIdx.x == 0 && blockIdx.y == 0)
        for (int i = threadIdx.x; i < a.n_counters; i += blockDim.x) a.counters[i] = 0u;
    const bool al16 = (reinterpret_cast<uintptr_t>(a.x) & 15) == 0 && (a.k & 7) == 0 && (a.gs & 7) == 0;
    const bool al8 = (reinterpret_cast<uintptr_t>(a.x) & 7) == 0 && (a.k & 3) == 0 && (a.gs & 3) == 0;
    RowsGroup<TP> v;
    v.template load<false, PARTS == 2>(a.x + (size_t)(t < a.m ? t : 0) * a.k, a.k, a.gs, 8 * (int)blockIdx.x + g, al16 ? 2 : (al8 ? 1 : 0), t < a.m, 8 * TP * part);
    rows_x_group<T, PARTS>(v, a.out + (size_t)blockIdx.x * rows_chunk_bytes(T, a.nt), t, g, part, a.nt, a.factor, t < a.m);
}

// The same behind a residual add and RMSNorm, one CTA per row: the row stays in registers between the sum of squares and the
// scaling, and in shared memory as bf16 after it.
template <int T>
__global__ void __launch_bounds__(1024) rows_norm_kernel(const __grid_constant__ RowsXArgs a, const __grid_constant__ TileNorm nm) {
    constexpr int KEEP = 2;
    extern __shared__ __align__(16) unsigned char rows_norm_row[];
    __shared__ float red[32];
    const int tid = threadIdx.x, nv = a.k >> 2, p = blockIdx.x;
    float4* row = reinterpret_cast<float4*>(nm.h + (size_t)p * a.k);
    const float4* drow = nm.delta ? reinterpret_cast<const float4*>(nm.delta + (size_t)p * a.k) : nullptr;
    const float4* g4 = reinterpret_cast<const float4*>(nm.gamma);
    uint2* xs = reinterpret_cast<uint2*>(rows_norm_row);
    float4 v[KEEP], gm[KEEP];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#pragma unroll
    for (int j = 0; j < KEEP; ++j)   // gamma is a constant of the model: fetched while the predecessor still runs
        if (tid + j * 1024 < nv) gm[j] = __ldg(g4 + tid + j * 1024);
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
    float total = red[tid & 31];
    for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    const float inv = rsqrtf(total / (float)a.k + nm.eps);
    auto put = [&](int i, const float4& t, const float4& gg) {
        const __nv_bfloat162 lo = __floats2bfloat162_rn(t.x * inv * gg.x, t.y * inv * gg.y), hi = __floats2bfloat162_rn(t.z * inv * gg.z, t.w * inv * gg.w);
        xs[i] = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    };
#pragma unroll
    for (int j = 0; j < KEEP; ++j)
        if (tid + j * 1024 < nv) put(tid + j * 1024, v[j], gm[j]);
    for (int i = tid + KEEP * 1024; i < nv; i += 1024) put(i, row[i], __ldg(g4 + i));
    if (tid == 0 && (nv & 1)) xs[nv] = make_uint2(0u, 0u);
    if (p == 0)
        for (int i = tid; i < a.n_counters; i += 1024) a.counters[i] = 0u;
    __syncthreads();
    const __nv_bfloat16* x = reinterpret_cast<const __nv_bfloat16*>(rows_norm_row);
    const int form = (a.gs & 7) == 0 ? 2 : ((a.gs & 3) == 0 ? 1 : 0);
    for (int g0 = 0; g0 < 8 * a.nchunks; g0 += 1024) {   // (whole chunks: the same for all lanes of eight)
        const int g = g0 + tid;
        const bool live = g < 8 * a.nchunks;
        RowsGroup<T> w;
        w.template load<true, false>(x, a.k, a.gs, g, form, live);
        rows_x_group<T, 1>(w, a.out + (size_t)(live ? g >> 3 : 0) * rows_chunk_bytes(T, a.nt), p, g & 7, 0, a.nt, a.factor, live);
    }
}

template <int NT>
struct RowsB {   // a lane's B registers of one slab: eight bytes per token tile
    uint32_t r[NT][2];
    __device__ __forceinline__ void load(const unsigned char* slab, uint32_t off) {
        if constexpr (NT == 1) {
            const uint2 v = *reinterpret_cast<const uint2*>(slab + off);
            r[0][0] = v.x; r[0][1] = v.y;
        } else {
            const uint4 v = *reinterpret_cast<const uint4*>(slab + off);
            r[0][0] = v.x; r[0][1] = v.y; r[1][0] = v.z; r[1][1] = v.w;
        }
    }
};

__device__ __forceinline__ float rows_gated(float gate, float up) { return up * gate / (1.0f + expf(-gate)); }

template <class C, int NT>
__global__ void __launch_bounds__(kRowsThreads, 1) rows_mma_kernel(const __grid_constant__ RowsArgs a) {
    extern __shared__ __align__(128) unsigned char rows_smem[];
    constexpr int T = C::T, SLAB = 256 * NT, CHUNK = rows_chunk_bytes(T, NT), N = 8 * NT;
    unsigned char* xs = rows_smem;
    float* slots = reinterpret_cast<float*>(rows_smem + a.x_bytes);
    unsigned char* ctx = rows_smem + a.x_bytes + (size_t)(a.pass_rb + kRowsWarps) * N * kRowsSlot * 4;
    __shared__ __align__(8) uint64_t x_full[kRowsChunks];
    __shared__ unsigned last;
    __shared__ short from[kRowsPass], to[kRowsPass];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, q = lane >> 2, c = lane & 3;
    const NintDevB& w = a.w;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    const int tile = blockIdx.x / a.slices, slice = blockIdx.x - tile * a.slices;
    const int ch0 = (int)((long long)slice * w.nchunks / a.slices), nch = (int)((long long)(slice + 1) * w.nchunks / a.slices) - ch0;
    const int unit = a.glu ? 2 : 1, units = w.nrb / unit;
    const int rb_begin = (int)((long long)tile * units / a.tiles) * unit, rb_end = (int)((long long)(tile + 1) * units / a.tiles) * unit;
    const size_t rb_words = (size_t)w.nchunks * w.rec_words, jump = rb_words - (size_t)(nch - 1) * w.rec_words;   // from a slice's last record to the next row-block's first
    const uint32_t rec_bytes = (uint32_t)w.rec_words * 4u;

    if (tid < nch) mbar_init(&x_full[tid], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    C::ctx_init(ctx, a, tid);
    bool first = true;
    for (int rb0 = rb_begin; rb0 < rb_end; rb0 += a.pass_rb) {
        const int nrb = min(a.pass_rb, rb_end - rb0), items = nrb * nch;
        const int it0 = warp * items / kRowsWarps, it1 = (warp + 1) * items / kRowsWarps;
        int rb = it0 / nch, ch = it0 - rb * nch;
        const uint32_t* rec = w.items + (size_t)(rb0 + rb) * rb_words + (size_t)(ch0 + ch) * w.rec_words;   // the item's record
        // records on their way into L2
        const uint32_t* pf = rec;
        int pf_ch = ch, pf_left = it1 - it0;
        auto ahead = [&]() {
            if (pf_left > 0) {
                if (lane == 0) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(pf), "r"(rec_bytes) : "memory");
                --pf_left;
                if (++pf_ch == nch) { pf_ch = 0; pf += jump; }
                else pf += w.rec_words;
            }
        };
        for (int i = 0; i < kRowsAhead; ++i) ahead();
        uint32_t code[C::CW];
        typename C::Scales sc;
        if (it0 < it1) {
#pragma unroll
            for (int i = 0; i < C::CW; ++i) code[i] = rows_ldg(rec + i * 32 + lane);
            sc.quad = rows_ldg4(rec + C::WC * 32 + (lane & ~3));
            sc.load_late(rec, lane);
        }
        __syncthreads();   // barriers, tables; the slots of the pass before
        if (first) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            if (tid < nch) {
                mbar_arrive_expect_tx(&x_full[tid], CHUNK);
                bulk_load(xs + (size_t)tid * CHUNK, a.x + (size_t)(ch0 + tid) * CHUNK, CHUNK, &x_full[tid]);
            }
            first = false;
        }
        float acc[NT][4], tot[NT][4], tot2[NT][4];
        auto zero = [&]() {
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int i = 0; i < 4; ++i) tot[j][i] = tot2[j][i] = 0.f;
        };
        zero();
        uint32_t boff[4];   // this lane's place in a slab, by 2 h + f
#pragma unroll
        for (int i = 0; i < 4; ++i) boff[i] = (uint32_t)((lane ^ (4 * (i >> 1) + (i & 1))) * (NT == 1 ? 8 : 16));
        const uint32_t bank_bytes = (uint32_t)w.entries * 64u;
        uint32_t anchor0 = 0u, anchor1 = 0u;
        if (it0 < it1) {
            anchor0 = __ldg(w.anchors + (size_t)(rb0 + rb) * 16 + q);
            anchor1 = __ldg(w.anchors + (size_t)(rb0 + rb) * 16 + q + 8);
        }
#pragma unroll 1
        for (int it = it0; it < it1; ++it) {
            const bool row_end = ch + 1 == nch, more = it + 1 < it1;
            const uint32_t* next = more ? rec + (row_end ? jump : (size_t)w.rec_words) : rec;
            ahead();
            if (it - it0 < nch && !mbar_wait(&x_full[ch], 0u)) atomicExch(a.error, MFQB_ERR_TIMEOUT);
            __syncwarp();
            const unsigned char* xc = xs + (size_t)ch * CHUNK;
            const uint4 next_quad = rows_ldg4(next + C::WC * 32 + (lane & ~3));
            typename C::Half hs;
            rows_static_for<2 * T>([&](auto s_c) {
                constexpr int S = decltype(s_c)::value, F = S / T;
                if constexpr (S % T == 0) C::template half<F>(sc, lane, ctx, hs);
                rows_static_for<2>([&](auto h_c) {
                    constexpr int H = decltype(h_c)::value, R = 4 * S + 2 * H;
                    RowsB<NT> b;
                    b.load(xc + (size_t)(2 * S + H) * SLAB, boff[2 * H + F]);
                    uint32_t a0, a1, a2, a3;
                    C::template weights<R>(code, hs, sc.own, ctx, a0, a2, bank_bytes);
                    C::template weights<R + 1>(code, hs, sc.own, ctx, a1, a3, bank_bytes);
#pragma unroll
                    for (int j = 0; j < NT; ++j) {
                        if constexpr (R == 0) rows_mma0(acc[j], a0, a1, a2, a3, b.r[j][0], b.r[j][1]);
                        else rows_mma(acc[j], a0, a1, a2, a3, b.r[j][0], b.r[j][1]);
                    }
                });
                // words that are used up make room for the next record's, or the second half's
                rows_static_for<C::CW>([&](auto i_c) {
                    constexpr int I = decltype(i_c)::value;
                    if constexpr (C::HALVES && C::last_reg(I) / 4 == S) code[I] = rows_ldg(rec + (C::CW + I) * 32 + lane);
                    else if constexpr (C::last_reg(I) / 4 == (C::HALVES ? S - T : S)) code[I] = rows_ldg(next + I * 32 + lane);
                });
            });
            float s2[NT][4];
            if constexpr (C::S2) {
                RowsB<NT> b;
                b.load(xc + (size_t)(4 * T) * SLAB, (uint32_t)(lane * (NT == 1 ? 8 : 16)));
                const uint32_t m0 = __byte_perm(sc.min, 0u, 0x4140u), m1 = __byte_perm(sc.min, 0u, 0x4342u);
#pragma unroll
                for (int j = 0; j < NT; ++j) rows_mma0(s2[j], m0, m1, m0, m1, b.r[j][0], b.r[j][1]);
                if constexpr (C::S1) {
                    const __half2 k1024 = __float2half2_rn(1024.f);
                    const uint32_t g0 = rows_u32(__hsub2(rows_h2(__byte_perm(sc.own, 0x64646464u, 0x4140u)), k1024));
                    const uint32_t g1 = rows_u32(__hsub2(rows_h2(__byte_perm(sc.own, 0x64646464u, 0x4342u)), k1024));
#pragma unroll
                    for (int j = 0; j < NT; ++j) rows_mma(acc[j], g0, g1, g0, g1, b.r[j][0], b.r[j][1]);
                }
            }
            sc.load_late(next, lane);
            sc.quad = next_quad;
            const float* xscale = reinterpret_cast<const float*>(xc + (size_t)(4 * T + 1) * SLAB);
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                const float2 d = *reinterpret_cast<const float2*>(xscale + 8 * j + 2 * c);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    tot[j][i] += acc[j][i] * ((i & 1) ? d.y : d.x);
                    if constexpr (C::S2) tot2[j][i] += s2[j][i] * ((i & 1) ? d.y : d.x);
                }
            }
            if (row_end || !more) {
                const float ns0 = __half2float(__ushort_as_half((unsigned short)(anchor0 & 0xFFFFu))) * a.undo, ns1 = __half2float(__ushort_as_half((unsigned short)(anchor1 & 0xFFFFu))) * a.undo;
                const float nm0 = __half2float(__ushort_as_half((unsigned short)(anchor0 >> 16))) * C::OUT_MIN, nm1 = __half2float(__ushort_as_half((unsigned short)(anchor1 >> 16))) * C::OUT_MIN;
                float* slot = slots + (size_t)(warp + rb) * N * kRowsSlot;
#pragma unroll
                for (int j = 0; j < NT; ++j)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        float v = tot[j][i] * (i < 2 ? ns0 : ns1);
                        if constexpr (C::S2) v -= tot2[j][i] * (i < 2 ? nm0 : nm1);
                        slot[(8 * j + 2 * c + (i & 1)) * kRowsSlot + q + 8 * (i >> 1)] = v;
                    }
                zero();
                ch = -1;
                ++rb;
                if (more) {
                    anchor0 = __ldg(w.anchors + (size_t)(rb0 + rb) * 16 + q);
                    anchor1 = __ldg(w.anchors + (size_t)(rb0 + rb) * 16 + q + 8);
                }
            }
            ++ch;
            rec = next;
        }
        if (tid < nrb) {   // the warps that had parts of a row-block
            int w0 = 0, w1 = kRowsWarps - 1;
            while ((w0 + 1) * items / kRowsWarps <= tid * nch) ++w0;
            while (w1 * items / kRowsWarps >= (tid + 1) * nch) --w1;
            from[tid] = (short)w0;
            to[tid] = (short)w1;
        }
        __syncthreads();
        // rows of a row-block are added up over these warps, in the order of K
        auto rows_sum = [&](int rb, int tok, int quad) {
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int w1 = from[rb]; w1 <= to[rb]; ++w1) {
                if (w1 * items / kRowsWarps == (w1 + 1) * items / kRowsWarps) continue;   // fewer records than warps
                const float4 u = *reinterpret_cast<const float4*>(slots + ((size_t)(w1 + rb) * N + tok) * kRowsSlot + 4 * quad);
                v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
            }
            return v;
        };
        auto put = [&](int tok, int row, int limit, const float4& v) {
            const float o[4] = {v.x, v.y, v.z, v.w};
            const int live = min(4, limit - row);
            const size_t at = (size_t)tok * a.ldy + row;
            if (a.y_dtype == 0 /* MFQB_F32 */) {
                float* y = static_cast<float*>(a.y) + at;
                if (live == 4 && (reinterpret_cast<uintptr_t>(y) & 15) == 0) *reinterpret_cast<float4*>(y) = v;
                else
                    for (int i = 0; i < live; ++i) y[i] = o[i];
            } else {
                __nv_bfloat16* y = static_cast<__nv_bfloat16*>(a.y) + at;
                if (live == 4 && (reinterpret_cast<uintptr_t>(y) & 7) == 0)
                    *reinterpret_cast<uint2*>(y) = make_uint2((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(o[0])) | (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(o[1])) << 16,
                                                              (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(o[2])) | (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(o[3])) << 16);
                else
                    for (int i = 0; i < live; ++i) y[i] = __float2bfloat16_rn(o[i]);
            }
        };
        // all rows of the pass: get(row-block, token, quad) gives four sums
        auto write = [&](auto&& get) {
            if (a.glu) {
                for (int i = tid; i < (nrb >> 1) * a.m * 4; i += kRowsThreads) {
                    const int quad = i & 3, p = (i >> 2) % (nrb >> 1), tok = (i >> 2) / (nrb >> 1);
                    const float4 g = get(2 * p, tok, quad), u = get(2 * p + 1, tok, quad);
                    put(tok, ((rb0 >> 1) + p) * 16 + 4 * quad, w.n >> 1,
                        make_float4(rows_gated(g.x, u.x), rows_gated(g.y, u.y), rows_gated(g.z, u.z), rows_gated(g.w, u.w)));
                }
            } else {
                for (int i = tid; i < nrb * a.m * 4; i += kRowsThreads) {
                    const int quad = i & 3, rb = (i >> 2) % nrb, tok = (i >> 2) / nrb;
                    put(tok, (rb0 + rb) * 16 + 4 * quad, w.n, get(rb, tok, quad));
                }
            }
        };
        if (a.slices == 1) {
            write(rows_sum);
        } else {   // the last slice of the tile to arrive adds them, in the order of K (slices > 1: one pass)
            const size_t stride = (size_t)a.pass_rb * a.m * 16;
            float* mine = a.parts + (size_t)blockIdx.x * stride;
            for (int i = tid; i < nrb * a.m * 4; i += kRowsThreads) {
                const int quad = i & 3, rb = (i >> 2) % nrb, tok = (i >> 2) / nrb;
                __stcg(reinterpret_cast<float4*>(mine + ((size_t)tok * nrb + rb) * 16 + 4 * quad), rows_sum(rb, tok, quad));
            }
            __threadfence();
            __syncthreads();
            if (tid == 0) last = atomicAdd(a.counters + tile, 1u);
            __syncthreads();
            if (last == (unsigned)(a.slices - 1)) {
                __threadfence();
                const float* all = a.parts + (size_t)tile * a.slices * stride;
                write([&](int rb, int tok, int quad) {
                    float4 u[kRowsSlices], v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int s = 0; s < kRowsSlices; ++s)   // one trip to L2 for all of them
                        u[s] = s < a.slices ? __ldcg(reinterpret_cast<const float4*>(all + (size_t)s * stride + ((size_t)tok * nrb + rb) * 16 + 4 * quad)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int s = 0; s < kRowsSlices; ++s) { v.x += u[s].x; v.y += u[s].y; v.z += u[s].z; v.w += u[s].w; }
                    return v;
                });
            }
        }
    }
}

}  // namespace mfqb
