// Device constants shared by the trajectory kernels: the DOP853 tables, the Chebyshev table of the
// smearing source, and the functions that read them. Each translation unit that includes this
// holds its own copy in constant memory, filled by dop853_upload().
#pragma once
#include <cuda_runtime.h>
#include "dop853_tables.h"
#include "source_table.h"

namespace rcmps {

static __constant__ double c_dop_a[256];
static __constant__ double c_dop_b[16];
static __constant__ double c_dop_c[16];
static __constant__ double c_dop_e5[16];
static __constant__ double c_dop_e3[16];
static __constant__ double c_dop_d[64];
static __constant__ double c_source[RCMPS_SOURCE_SEGMENTS * (RCMPS_SOURCE_DEGREE + 1)];

// 2|t| J(t^2) from the piecewise Chebyshev table (Clenshaw); |t| <= sqrt(40).
static __device__ double source_value(double t) {
  const double a = fabs(t);
  const double width = RCMPS_SOURCE_AMAX / RCMPS_SOURCE_SEGMENTS;
  int seg = (int)(a / width);
  if (seg > RCMPS_SOURCE_SEGMENTS - 1) seg = RCMPS_SOURCE_SEGMENTS - 1;
  const double z = 2.0 * (a - seg * width) / width - 1.0;
  const double* c = c_source + seg * (RCMPS_SOURCE_DEGREE + 1);
  double b1 = 0.0, b2 = 0.0;
  for (int j = RCMPS_SOURCE_DEGREE; j > 0; --j) {
    const double b0 = 2.0 * z * b1 - b2 + c[j];
    b2 = b1;
    b1 = b0;
  }
  return z * b1 - b2 + c[0];
}

// The next double above t (nextafter(t, +inf)) for finite t.
static __device__ __forceinline__ double next_up(double t) {
  if (t == 0.0) return 4.9406564584124654e-324;
  const long long b = __double_as_longlong(t);
  return __longlong_as_double(t > 0.0 ? b + 1 : b - 1);
}

// Fill this translation unit's tables on the current device.
static inline cudaError_t dop853_upload() {
  cudaError_t e;
  if ((e = cudaMemcpyToSymbol(c_dop_a, rcmps_dop_a, sizeof(rcmps_dop_a))) != cudaSuccess) return e;
  if ((e = cudaMemcpyToSymbol(c_dop_b, rcmps_dop_b, sizeof(rcmps_dop_b))) != cudaSuccess) return e;
  if ((e = cudaMemcpyToSymbol(c_dop_c, rcmps_dop_c, sizeof(rcmps_dop_c))) != cudaSuccess) return e;
  if ((e = cudaMemcpyToSymbol(c_dop_e5, rcmps_dop_e5, sizeof(rcmps_dop_e5))) != cudaSuccess) return e;
  if ((e = cudaMemcpyToSymbol(c_dop_e3, rcmps_dop_e3, sizeof(rcmps_dop_e3))) != cudaSuccess) return e;
  if ((e = cudaMemcpyToSymbol(c_dop_d, rcmps_dop_d, sizeof(rcmps_dop_d))) != cudaSuccess) return e;
  return cudaMemcpyToSymbol(c_source, rcmps_source_table, sizeof(rcmps_source_table));
}

}  // namespace rcmps
