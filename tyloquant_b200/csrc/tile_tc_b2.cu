// NINT2 instantiations of the tensor-memory tile kernel.
#include "tile_tc_launch.cuh"

namespace mfqb {
MFQB_TILE_INSTANTIATE(2)
}  // namespace mfqb
