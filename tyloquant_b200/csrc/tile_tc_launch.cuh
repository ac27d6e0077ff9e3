// Launch tables of the tensor-memory tile kernel, one translation unit per code width (tile_tc_b*.cu).
#pragma once
#include <cuda_runtime.h>

#include "tile_tc.cuh"

namespace mfqb {

struct TilePlan {
    int grid = 0;
    size_t smem = 0;
};

// A plain product, or one cohort of an expert product: one codec.
template <class C>
struct TileOne {
    static constexpr bool ONE = true;
    static constexpr int TERMS = C::TERMS, XTERMS = 1;
    template <class Fn>
    __device__ static __forceinline__ void dispatch(const NintDevB&, Fn&& f) { f(C{}); }
    __device__ static void ctx_init(unsigned char* ctx, const TileArgs& a, int tid, int nthreads) { C::ctx_init(ctx, a, tid, nthreads); }
};

template <class Sets, bool GLU>
static cudaError_t launch_tile_form(const TileArgs& a, const TilePlan& p, cudaStream_t stream) {
    auto kernel = tile_tc_kernel<Sets, GLU>;
    static bool attr_set[64] = {};   // per kernel and device: the largest dynamic shared memory any plan asks for
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileDynSmem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);   // see whole_carveout
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)p.grid);
    cfg.blockDim = dim3(kTileThreads);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, a);
}

template <class Sets>
static cudaError_t launch_tile(const TileArgs& a, const TilePlan& p, cudaStream_t stream) {
    return a.glu ? launch_tile_form<Sets, true>(a, p, stream) : launch_tile_form<Sets, false>(a, p, stream);
}

template <int BITS>
cudaError_t launch_tile_bits(const TileArgs& a, const TilePlan& p, cudaStream_t stream);
cudaError_t launch_tile_nvq(const TileArgs& a, const TilePlan& p, int terms, cudaStream_t stream);
cudaError_t launch_tile_experts(const TileArgs& a, const TilePlan& p, int terms, int x_terms, cudaStream_t stream);

template <int BITS, int T>
static cudaError_t launch_tile_if_catalog(const TileArgs& a, const TilePlan& p, cudaStream_t stream) {
    if constexpr (nint_bl_in_catalog(BITS, T)) {
        if (a.pools[0].tile_terms != 2) return launch_tile<TileOne<TileNint<BITS, T>>>(a, p, stream);
        if constexpr (T <= 6) return launch_tile<TileOne<TileNint<BITS, T, 2>>>(a, p, stream);   // beyond, two stages of two terms do not fit tensor memory
    }
    return cudaErrorNotSupported;
}
#define MFQB_TILE_INSTANTIATE(BITS)                                                                          \
    template <>                                                                                              \
    cudaError_t launch_tile_bits<BITS>(const TileArgs& a, const TilePlan& p, cudaStream_t stream) {          \
        switch (a.pools[0].t8) {                                                                             \
            case 2: return launch_tile_if_catalog<BITS, 2>(a, p, stream);                                    \
            case 3: return launch_tile_if_catalog<BITS, 3>(a, p, stream);                                    \
            case 4: return launch_tile_if_catalog<BITS, 4>(a, p, stream);                                    \
            case 5: return launch_tile_if_catalog<BITS, 5>(a, p, stream);                                    \
            case 6: return launch_tile_if_catalog<BITS, 6>(a, p, stream);                                    \
            case 8: return launch_tile_if_catalog<BITS, 8>(a, p, stream);                                    \
            default: return cudaErrorNotSupported;                                                           \
        }                                                                                                    \
    }

}  // namespace mfqb
