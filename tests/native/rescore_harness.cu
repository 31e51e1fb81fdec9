// The lists of launch_rescore_levels (csrc/device/rescore.cu) for host arrays.
#include <cstdint>

#include "../../rils-rols_gb300/csrc/device/rescore.cu"

namespace rrd {
bool launch_ok(const char*) { return cudaGetLastError() == cudaSuccess; }
}  // namespace rrd

extern "C" int rescore_levels(const uint8_t* need, const uint8_t* kind, const int32_t* level_end, int32_t n_levels,
                              int32_t* cols, int32_t* count, int32_t* fac, int32_t* fac_count) {
  const int32_t n = level_end[n_levels - 1];
  uint8_t *d_need = nullptr, *d_kind = nullptr;
  int32_t *d_end = nullptr, *d_out = nullptr;  // cols, count, fac, fac_count
  const size_t words = 2 * (size_t)n + n_levels + 1;
  bool ok = cudaMalloc(&d_need, n) == cudaSuccess && cudaMalloc(&d_kind, n) == cudaSuccess &&
            cudaMalloc(&d_end, 4 * n_levels) == cudaSuccess && cudaMalloc(&d_out, 4 * words) == cudaSuccess &&
            cudaMemset(d_out, 0xff, 4 * words) == cudaSuccess &&
            cudaMemcpy(d_need, need, n, cudaMemcpyHostToDevice) == cudaSuccess &&
            cudaMemcpy(d_kind, kind, n, cudaMemcpyHostToDevice) == cudaSuccess &&
            cudaMemcpy(d_end, level_end, 4 * n_levels, cudaMemcpyHostToDevice) == cudaSuccess &&
            rrd::launch_rescore_levels(d_need, d_kind, d_end, n_levels, d_out, d_out + n, d_out + n + n_levels,
                                       d_out + 2 * n + n_levels, nullptr) &&
            cudaMemcpy(cols, d_out, 4 * n, cudaMemcpyDeviceToHost) == cudaSuccess &&
            cudaMemcpy(count, d_out + n, 4 * n_levels, cudaMemcpyDeviceToHost) == cudaSuccess &&
            cudaMemcpy(fac, d_out + n + n_levels, 4 * n, cudaMemcpyDeviceToHost) == cudaSuccess &&
            cudaMemcpy(fac_count, d_out + 2 * n + n_levels, 4, cudaMemcpyDeviceToHost) == cudaSuccess;
  cudaFree(d_need);
  cudaFree(d_kind);
  cudaFree(d_end);
  cudaFree(d_out);
  return ok ? 0 : 1;
}
