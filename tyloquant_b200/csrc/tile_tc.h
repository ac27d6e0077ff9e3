// Host interface of the tensor-memory tile kernel (tile_tc.cuh).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>


#include "nint_blayout.h"

namespace mfqb {

// What the activation rows are: bf16, or float32 gate | up products whose SwiGLU activation is formed on the way.
enum TileX { kTileXBf16 = 0, kTileXSwiglu = 1, kTileXShared = 2 /* bf16 in shared memory */ };
// Residual add + RMSNorm on the way to the product: h [m, k] float32 += delta (may be null), x = bf16(h / rms(h) * gamma).
struct TileNorm {
    float* h;
    const float *delta, *gamma;
    float eps;
};

constexpr float kTileWeightScale = 0.25f;   // of the f16 weights: 8-bit codes x 8-bit sub-scales x offset head-room stay below 65504

#if defined(__CUDACC__)
// Constants of a weight row for the tile kernel, 16 bytes: x = f16 a (times kTileWeightScale) | f16 high part of -b << 16,
// y = f16 low part of -b, z = float32 factor of the row's sums.  Scalar rows: F = |ns| 2^j >= |nm| 2^-(bits + 1) with the smallest
// such j >= 0 (a = ns / F is a power of two), F = |nm| 2^-(bits + 1) where ns = 0, b = nm / F, factor F; lattice rows (bits = 0):
// factor = anchor.
__device__ __forceinline__ uint4 tile_row_const(uint32_t anchor, int bits) {
    const float ns = __half2float(__ushort_as_half((unsigned short)(anchor & 0xFFFFu))), nm = __half2float(__ushort_as_half((unsigned short)(anchor >> 16)));
    uint4 c = make_uint4(0u, 0u, __float_as_uint(ns), 0u);
    if (bits) {
        const float least = fabsf(nm) * __uint_as_float((uint32_t)(126 - bits) << 23);
        float f = fabsf(ns);
        if (f == 0.f) f = least > 0.f ? least : 1.f;
        else if (least > f) f = ldexpf(f, ilogbf(least / f) + 1);
        const float nb = -nm / f * kTileWeightScale;
        const __half hi = __float2half_rn(nb);
        c.x = (uint32_t)__half_as_ushort(__float2half_rn(ns / f * kTileWeightScale)) | (uint32_t)__half_as_ushort(hi) << 16;
        c.y = (uint32_t)__half_as_ushort(__float2half_rn(nb - __half2float(hi)));
        c.z = __float_as_uint(f * (1.f / kTileWeightScale));
    }
    return c;
}
#endif

// y [m, n] = x [m, k] W^T for bf16 x, or for the rows that `norm` gives (x unused).  glu: 16-row blocks of W alternate gate and
// up rows and y [m, n / 2] = up * silu(gate).  False when this weight has no tile kernel (its tables do not fit).
bool launch_tile_product(const NintDevB& w, const void* x, int m, void* y, int y_dtype, int device, cudaStream_t s, bool glu = false, const TileNorm* norm = nullptr);

// f16 terms a lattice weight needs: 1 when every scale x code product is an f16 number, else 2; 0 when the state scales lie too far
// apart to be f16 numbers side by side (no tile kernel then).
int lattice_terms(const float* lut, const int8_t* codes, size_t n_codes);

// f16 state scales of a lattice record, normalised so that code x scale stays below 2^15, and what undoes that.
void tile_lattice_scales(const NintDevB& w, uint16_t (&lut16)[16], float& undo);

// A route plan whose tiles hold up to tile_rows pairs, and where each expert lives.
struct TileRoutes {
    const int *expert_bounds, *tile_bounds, *pair_order, *expert_pool, *expert_local;
    int n_experts, pairs, tile_rows;
};
// Routed expert products over the cohorts of a record.  Weights and the float32 activations of a gated FFN go in as `terms` f16
// terms: two where the record's other kernels are the integer ones, whose accuracy they keep (tile_experts_terms).
int tile_experts_terms(const NintDevB* pools, const int* held, int npools, int pairs, int experts);
// Most pairs per tile that fit, 0: no tile kernel for this record; the pairs per tile to take.
int tile_experts_max_rows(const NintDevB* pools, const int* held, int npools, int terms, bool float_x);
int tile_experts_rows(int pairs, int experts, int max_rows);
size_t tile_experts_x_bytes(const NintDevB* pools, const int* held, int npools, int pairs, int experts, int terms, bool float_x);
// Row p of the plan takes x row pair_order[p] / src_div (src_div = 0: row p) and writes y row pair_order[p] (scatter) or p.  xbuf:
// tile_experts_x_bytes of device memory.
void launch_tile_experts_product(const NintDevB* pools, const int* held, int npools, const TileRoutes& r, int terms, const void* x, TileX kind, int src_div, void* xbuf, void* y,
                                 int y_dtype, bool scatter, int rows_per_expert, int rb_per_expert, int device, cudaStream_t s);

}  // namespace mfqb
