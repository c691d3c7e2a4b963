// One row of a compressed-row product with one vector, for the kernels that need it (the plain
// product, flexible CG's fused one).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace fc {

// Lanes of a warp that share a row: half a warp takes a structured mesh's 81-entry row in five
// rounds (a whole warp in three, the last mostly idle) and keeps two rows' loads in flight a warp.
constexpr int SPMV_LANES = 16;

// sum over the row's entries of val * x[idx], on every lane of the row's group: six entries a lane in
// flight (a whole 81-entry row at once: the chain is then row pointer, entries, x, whatever the
// row), the lanes' sums by a butterfly. Every lane of the warp calls it; a row with ok false is empty.
__device__ __forceinline__ double spmv_entries(int64_t e0, int64_t e1, const int32_t *__restrict__ idx,
                                               const double *__restrict__ val, const double *x, int lane) {
  constexpr int FLIGHT = 6;
  double sum = 0.0;
  for (int64_t e = e0 + lane; e < e1; e += FLIGHT * SPMV_LANES) {
    int32_t c[FLIGHT];
    double v[FLIGHT], xv[FLIGHT];
#pragma unroll
    for (int q = 0; q < FLIGHT; ++q) {
      const bool in = e + q * SPMV_LANES < e1;
      c[q] = in ? idx[e + q * SPMV_LANES] : -1;
      v[q] = in ? val[e + q * SPMV_LANES] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < FLIGHT; ++q) xv[q] = c[q] >= 0 ? x[c[q]] : 0.0;
#pragma unroll
    for (int q = 0; q < FLIGHT; ++q)
      if (c[q] >= 0) sum = fma(v[q], xv[q], sum);
  }
#pragma unroll
  for (int o = SPMV_LANES / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o, SPMV_LANES);
  return sum;
}
__device__ __forceinline__ double spmv_row(bool ok, int64_t row, const int64_t *__restrict__ ptr,
                                           const int32_t *__restrict__ idx, const double *__restrict__ val,
                                           const double *x, int lane) {
  return spmv_entries(ok ? ptr[row] : 0, ok ? ptr[row + 1] : 0, idx, val, x, lane);
}

}  // namespace fc
