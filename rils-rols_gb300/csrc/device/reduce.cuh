// Deterministic block reductions (fixed shuffle tree, then warps in order).
#pragma once
#include <cuda_runtime.h>

namespace rrd {

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = __dadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Sum of `v` over the block; every thread gets the same value.
// `red` is shared scratch of at least blockDim.x / 32 doubles.
__device__ __forceinline__ double block_sum(double v, double* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  double s = 0.0;
  for (int i = 0; i < nw; ++i) s = __dadd_rn(s, red[i]);
  return s;
}

// warp_sum of N values per lane at once (N a power of two): while several
// values are left, lanes exchange half of them and each half-warp goes on with
// the other half, so a stride costs half the additions of the one before
// (8 values: 9 additions, not 40) and every addition is warp_sum's.  Lane l
// returns the total of value index_of(l), the top log2(N) bits of l.
template <int N>
__device__ __forceinline__ double warp_sum_many(double (&v)[N]) {
  const int lane = threadIdx.x & 31;
  int o = 16;
#pragma unroll
  for (int n = N; n > 1; n >>= 1, o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < n / 2; ++i) {
      const double keep = up ? v[i + n / 2] : v[i], send = up ? v[i] : v[i + n / 2];
      v[i] = __dadd_rn(keep, __shfl_xor_sync(0xffffffffu, send, o));
    }
  }
#pragma unroll
  for (; o > 0; o >>= 1) v[0] = __dadd_rn(v[0], __shfl_xor_sync(0xffffffffu, v[0], o));
  return v[0];
}

// Lane fold of cnt <= CG values per thread of a 256-thread block (RR256's
// fold: halving strides inside each 32-lane group, then the eight group
// totals in order from 0) into out[0 .. cnt) (shared).  red: 8 * CG shared
// doubles.  CG a power of two.
template <int CG>
__device__ __forceinline__ void fold_lanes(const double (&v)[CG], int cnt, double* red, double* out) {
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (CG == 1 || cnt == 1) {
    const double s = warp_sum(v[0]);
    if (l == 0) red[w * CG] = s;
  } else {
    double x[CG];
#pragma unroll
    for (int j = 0; j < CG; ++j) x[j] = v[j];
    const double s = warp_sum_many<CG>(x);
    if ((l & (32 / CG - 1)) == 0) red[w * CG + l / (32 / CG)] = s;
  }
  __syncthreads();
  if (threadIdx.x < cnt) {
    double s = 0.0;
    for (int i = 0; i < 8; ++i) s = __dadd_rn(s, red[i * CG + threadIdx.x]);
    out[threadIdx.x] = s;
  }
  __syncthreads();
}

}  // namespace rrd
