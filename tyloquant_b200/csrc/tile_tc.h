// Host interface of the tensor-memory tile kernel (tile_tc.cuh).
#pragma once
#include <cuda_runtime.h>

#include "nint_blayout.h"

namespace mfqb {

// What the activation rows are: bf16, float32, or float32 gate | up products whose SwiGLU activation is formed on the way.
enum TileX { kTileXBf16 = 0, kTileXF32 = 1, kTileXSwiglu = 2 };

// y [m, n] = x [m, k] W^T for bf16 x.  False when this weight has no tile kernel (its tables do not fit).
bool launch_tile_product(const NintDevB& w, const void* x, int m, void* y, int y_dtype, int device, cudaStream_t s);

// f16 terms a lattice weight needs: 1 when every scale x code product is an f16 number, else 2.
int lattice_terms(const float* lut, const int8_t* codes, size_t n_codes);

}  // namespace mfqb
