// Device helpers shared by the FP64 QR kernels (qr_small.cu, qr_chunk.cu) and the residual (plain.cu).
#pragma once
#include <cstdint>

#include "common.cuh"

namespace rrd {

// Column j of candidate factor values: contiguous columns from a_col, or
// through the column map (shared factor table) when one is given.
__device__ __forceinline__ const double* factor_column(const double* A, int64_t n_pad, int64_t a_col, int j,
                                                       const int32_t* colmap) {
  return A + (colmap ? (int64_t)colmap[a_col + j] : a_col + j) * n_pad;
}

}  // namespace rrd
