// Lattice codec of the tensor-memory tile kernel (tile_tc.cuh); record layout: nvq_blayout.h.
#pragma once
#include "tile_tc.cuh"

namespace mfqb {

// Index bits, joint scale/codebook states, f16 terms per weight.  A register is one table look-up: the signed table holds the
// four int8 weights of (bank, index, sign nibble), in shared memory, biased by 128 so that a byte under the exponent 0x64 is 1152 + code.
template <int IB, bool JSC, int TERMS_>
struct TileNvq {
    static constexpr int T = 3, TERMS = TERMS_, FB = IB + 4, WC = (24 * FB + 31) / 32;
    static constexpr uint32_t OFFMASK = ((1u << FB) - 1u) << 2;   // a field as a byte offset into the table
    __host__ __device__ static size_t ctx_bytes(const NintDevB& w) { return (size_t)w.table_words * 4 + 64; }
    __device__ static void ctx_init(unsigned char* ctx, const TileArgs& a, int tid, int nthreads) {
        const NintDevB& w = a.pools[0];
        const uint4* src = reinterpret_cast<const uint4*>(w.table);
        for (int i = tid; i < w.table_words / 4; i += nthreads) {
            uint4 v = __ldg(src + i);
            v.x ^= 0x80808080u; v.y ^= 0x80808080u; v.z ^= 0x80808080u; v.w ^= 0x80808080u;
            reinterpret_cast<uint4*>(ctx)[i] = v;
        }
        if (tid < 16) reinterpret_cast<uint16_t*>(ctx + (size_t)w.table_words * 4)[tid] = a.lut16[tid];
    }
    struct Row {
        uint32_t bank_bytes, lut_off;
        __device__ __forceinline__ Row(const NintDevB& w, const uint4*, int) : bank_bytes((uint32_t)w.entries * 64u), lut_off((uint32_t)w.table_words * 4u) {}
    };
    template <int R>
    __device__ static __forceinline__ uint32_t codes(const uint32_t* rec, int lane, uint32_t own, const Row& row, const unsigned char* ctx) {
        constexpr int POS = R * FB, WI = POS >> 5, SH = POS & 31;
        uint32_t off;
        if constexpr (SH + FB <= 32) {
            const uint32_t v = rec[WI * 32 + lane];
            off = (SH >= 2 ? v >> (SH >= 2 ? SH - 2 : 0) : v << (SH < 2 ? 2 - SH : 0)) & OFFMASK;
        } else {
            off = __funnelshift_r(rec[WI * 32 + lane], rec[(WI + 1) * 32 + lane], SH - 2) & OFFMASK;   // a field that straddles two words starts above bit 2
        }
        if constexpr (JSC) {
            constexpr int I = (R / 12) * 4 + (R & 3);   // the (row, group) pair of this register: its bank travels in the lane's own scale word
            off += ((own >> (8 * (I >> 1) + 4 + 2 * (I & 1))) & 3u) * row.bank_bytes;
        }
        return *reinterpret_cast<const uint32_t*>(ctx + off);
    }
    // codes of one register times the scale d (as f16 terms): first terms in lo / hi, what rounding cut off in lo2 / hi2
    template <int R>
    __device__ static __forceinline__ void weights(const uint32_t* rec, int lane, uint32_t own, const Row& row, const unsigned char* ctx, __half2 d, __half2 bd,
                                                   uint32_t& lo, uint32_t& hi, uint32_t& lo2, uint32_t& hi2) {
        const uint32_t v = codes<R>(rec, lane, own, row, ctx);
        const __half2 even = h2_bits((v & 0x00FF00FFu) | 0x64006400u), odd = h2_bits(((v >> 8) & 0x00FF00FFu) | 0x64006400u);
        if constexpr (!JSC) {   // d <= 15: 1152 d is exact, so is the integer result
            lo = bits_h2(__hfma2(even, d, bd));
            hi = bits_h2(__hfma2(odd, d, bd));
        } else {
            const __half2 k1152 = __float2half2_rn(1152.f), ce = __hsub2(even, k1152), co = __hsub2(odd, k1152);
            const __half2 pe = __hmul2(ce, d), po = __hmul2(co, d);
            lo = bits_h2(pe);
            hi = bits_h2(po);
            if constexpr (TERMS == 2) {
                lo2 = bits_h2(__hfma2(ce, d, __hneg2(pe)));
                hi2 = bits_h2(__hfma2(co, d, __hneg2(po)));
            }
        }
    }
    template <int F, int TI>
    __device__ static __forceinline__ void octets(const uint32_t* rec, int lane, uint32_t own, const Row& row, const unsigned char* ctx, const __half2 (&d)[4],
                                                  const __half2 (&bd)[4], uint32_t taddr) {
        if constexpr (TI < T) {
            constexpr int R = (F * T + TI) * 4;
            uint32_t r[8], e[8];
            weights<R>(rec, lane, own, row, ctx, d[0], bd[0], r[0], r[2], e[0], e[2]);
            weights<R + 1>(rec, lane, own, row, ctx, d[1], bd[1], r[1], r[3], e[1], e[3]);
            weights<R + 2>(rec, lane, own, row, ctx, d[2], bd[2], r[4], r[6], e[4], e[6]);
            weights<R + 3>(rec, lane, own, row, ctx, d[3], bd[3], r[5], r[7], e[5], e[7]);
            tmem_st_16x128b_x4(taddr + 16 * TI, r);
            if constexpr (TERMS == 2) tmem_st_16x128b_x4(taddr + 16 * T + 16 * TI, e);
            octets<F, TI + 1>(rec, lane, own, row, ctx, d, bd, taddr);
        }
    }
    static constexpr bool SPLIT = false;
    template <int F>
    __device__ static __forceinline__ void half(const uint32_t* rec, int lane, int, const Row& row, const unsigned char* ctx, uint32_t taddr) {
        const uint16_t* lut = reinterpret_cast<const uint16_t*>(ctx + row.lut_off);
        const int odd = (lane >> 1) & 1;
        const uint32_t own = rec[WC * 32 + lane];
        __half2 d[4], bd[4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t sw = rec[WC * 32 + (lane & ~3) + 2 * F + h] >> (8 * odd);
#pragma unroll
            for (int hi = 0; hi < 2; ++hi) {
                const uint32_t st = (sw >> (16 * hi)) & 15u;
                d[2 * h + hi] = __half2half2(__ushort_as_half(lut[st]));
                if constexpr (!JSC) bd[2 * h + hi] = __hmul2(d[2 * h + hi], __float2half2_rn(-1152.f));
            }
        }
        octets<F, 0>(rec, lane, own, row, ctx, d, bd, taddr);
    }
};

}  // namespace mfqb
