// Launch tables of the few-rows kernel, one translation unit per code width (rows_mma_b*.cu).
#pragma once
#include "rows_mma.cuh"

namespace mfqb {

constexpr size_t kRowsSmem = 226 * 1024;   // with the static shared memory at most 227 KB

template <class C, int NT>
static cudaError_t launch_rows_form(const RowsArgs& a, size_t smem, cudaStream_t stream) {
    auto kernel = rows_mma_kernel<C, NT>;
    static bool attr_set[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kRowsSmem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(a.tiles * a.slices));
    cfg.blockDim = dim3(kRowsThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, a);
}
template <class C>
static cudaError_t launch_rows(const RowsArgs& a, size_t smem, cudaStream_t stream) {
    return a.m <= 8 ? launch_rows_form<C, 1>(a, smem, stream) : launch_rows_form<C, 2>(a, smem, stream);
}

template <int BITS>
cudaError_t launch_rows_bits(const RowsArgs& a, size_t smem, cudaStream_t stream);
cudaError_t launch_rows_nvq(const RowsArgs& a, size_t smem, cudaStream_t stream);

template <int BITS, int T>
static cudaError_t launch_rows_if_catalog(const RowsArgs& a, size_t smem, cudaStream_t stream) {
    if constexpr (nint_bl_in_catalog(BITS, T)) return launch_rows<RowsNint<BITS, T>>(a, smem, stream);
    return cudaErrorNotSupported;
}
#define MFQB_ROWS_INSTANTIATE(BITS)                                                                \
    template <>                                                                                    \
    cudaError_t launch_rows_bits<BITS>(const RowsArgs& a, size_t smem, cudaStream_t stream) {      \
        switch (a.w.t8) {                                                                          \
            case 2: return launch_rows_if_catalog<BITS, 2>(a, smem, stream);                       \
            case 3: return launch_rows_if_catalog<BITS, 3>(a, smem, stream);                       \
            case 4: return launch_rows_if_catalog<BITS, 4>(a, smem, stream);                       \
            case 5: return launch_rows_if_catalog<BITS, 5>(a, smem, stream);                       \
            case 6: return launch_rows_if_catalog<BITS, 6>(a, smem, stream);                       \
            case 8: return launch_rows_if_catalog<BITS, 8>(a, smem, stream);                       \
            default: return cudaErrorNotSupported;                                                 \
        }                                                                                          \
    }

}  // namespace mfqb
