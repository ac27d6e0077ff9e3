#include "rows_mma_launch.cuh"

namespace mfqb {
// up to eight rows: from nine on lattice records take the tile kernel
cudaError_t launch_rows_nvq(const RowsArgs& a, size_t smem, cudaStream_t stream) {
    switch (a.w.index_bits * 2 + (a.w.jsc ? 1 : 0)) {
        case 16: return launch_rows_form<RowsNvq<8, false>, 1>(a, smem, stream);
        case 17: return launch_rows_form<RowsNvq<8, true>, 1>(a, smem, stream);
        case 19: return launch_rows_form<RowsNvq<9, true>, 1>(a, smem, stream);
        case 21: return launch_rows_form<RowsNvq<10, true>, 1>(a, smem, stream);
        default: return cudaErrorNotSupported;
    }
}
}  // namespace mfqb
