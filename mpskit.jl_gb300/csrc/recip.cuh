// Reciprocal and inverse square root of an FP64 value in few dependent FP64 instructions (a scheduler
// issues one in 64 clocks): for positive values of magnitude 2^-1000 to 2^1000, good to an ulp.
#pragma once

#include "tc_ptx.cuh"

namespace gb {

// 1 / sqrt(d), d > 0: single-precision seed of the mantissa brought to [1, 4) and one cubic
// step (e = 1 - d y^2 is at most 2^-21), five dependent FP64 instructions
__device__ __forceinline__ double inv_sqrt(double d) {
  const int hi = __double2hiint(d);
  const int s = (((hi >> 20) & 0x7ff) - 1023) >> 1;
  const double m = __hiloint2double(hi - (s << 21), __double2loint(d));
  const double y = to_double(rsqrtf(to_float(m)));
  const double e = fma(-m * y, y, 1.0);
  const double r = fma(y * e, fma(0.375, e, 0.5), y);
  return __hiloint2double(__double2hiint(r) - (s << 20), __double2loint(r));
}

// 1 / d likewise
__device__ __forceinline__ double inverse(double d) {
  const int hi = __double2hiint(d);
  const int s = ((hi >> 20) & 0x7ff) - 1023;
  const double m = __hiloint2double(hi - (s << 20), __double2loint(d));
  const double y = to_double(__fdividef(1.0f, to_float(m)));
  const double e = fma(-m, y, 1.0);
  const double r = fma(y, fma(e, e, e), y);
  return __hiloint2double(__double2hiint(r) - (s << 20), __double2loint(r));
}

}  // namespace gb
