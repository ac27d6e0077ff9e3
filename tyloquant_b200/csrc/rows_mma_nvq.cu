#include "rows_mma_launch.cuh"

namespace mfqb {
cudaError_t launch_rows_nvq(const RowsArgs& a, size_t smem, cudaStream_t stream) {
    switch (a.w.index_bits * 2 + (a.w.jsc ? 1 : 0)) {
        case 16: return launch_rows<RowsNvq<8, false>>(a, smem, stream);
        case 17: return launch_rows<RowsNvq<8, true>>(a, smem, stream);
        case 19: return launch_rows<RowsNvq<9, true>>(a, smem, stream);
        case 21: return launch_rows<RowsNvq<10, true>>(a, smem, stream);
        default: return cudaErrorNotSupported;
    }
}
}  // namespace mfqb
