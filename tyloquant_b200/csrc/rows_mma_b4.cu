#include "rows_mma_launch.cuh"

namespace mfqb {
MFQB_ROWS_INSTANTIATE(4)
}  // namespace mfqb
