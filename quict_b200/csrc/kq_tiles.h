// Dense gates on 5 to 10 qubits as tiled matrix products (kq_tiles.cu).
#pragma once

#include <cstdint>

#include <cuda_runtime.h>

namespace qs {

// bits[t]: vector bit of target t (matrix-index bit k-1-t); cmask / tmask: control
// and target bits; M: the matrix on the device, row-major.
int apply_kq_tiles(int dtype, void* vec, int n, int k, const int32_t* bits, uint64_t cmask, uint64_t tmask,
                   const double2* M, cudaStream_t st);

}  // namespace qs
