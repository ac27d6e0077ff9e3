// Host interface of the few-rows kernel (rows_mma.cuh).
#pragma once
#include <cuda_runtime.h>

#include "nint_blayout.h"
#include "tile_tc.h"

namespace mfqb {

constexpr int kRowsMax = 16;   // most activation rows

// y [m, n] = x [m, k] W^T for bf16 x, or for the rows that `norm` gives (x unused).  glu: 16-row blocks of W alternate gate and
// up rows and y [m, n / 2] = up * silu(gate).  False where other kernels are the better or the more accurate ones.
bool launch_rows_product(const NintDevB& w, const void* x, int m, void* y, int y_dtype, int device, cudaStream_t s, bool glu = false, const TileNorm* norm = nullptr);
// Scratch for any call with this weight, so that smaller batches can be captured after a larger one.
void reserve_rows(const NintDevB& w, int device, cudaStream_t s);

}  // namespace mfqb
