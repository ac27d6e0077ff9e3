#include "rows_mma_launch.cuh"

namespace mfqb {
MFQB_ROWS_INSTANTIATE(5)
}  // namespace mfqb
