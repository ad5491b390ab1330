// Reciprocal square roots in FP64 from the FP32 one: y (1 + e / 2 + 3 e^2 / 8) with e = 1 - d y^2, Householder's
// iteration of third order for 1 / sqrt(d) (the binomial series of 1 / sqrt(1 - e) cut after the square). With e at
// most some 6e-7 the rest is below 1e-19. Five dependent FP64 operations where sqrt and a division take more
// than twenty, at some 80 cycles of latency each on this GPU.
#pragma once

namespace ttgb {

// y / sqrt(1 - e) for |e| below about 1e-6
__device__ __forceinline__ double rsqrt_corrected(double y, double e) {
  return fma(y * e, fma(e, 0.375, 0.5), y);
}

// 1 / sqrt(d) for d in the FP32 range
__device__ __forceinline__ double rsqrt_refined(double d) {
  const double y = (double)rsqrtf((float)d);
  return rsqrt_corrected(y, fma(-d * y, y, 1.0));
}

// 1 / sqrt(d) for any d, by its significand in [1, 4) where d is a normal positive number
__device__ __forceinline__ double rsqrt_full(double d) {
  const int hi = __double2hiint(d);
  if (hi < 0x00100000 || hi >= 0x7ff00000) return 1.0 / sqrt(d);   // zero, subnormal, negative, not finite
  const int e = ((hi >> 20) - 1023) & ~1;
  const double v = rsqrt_refined(__hiloint2double(hi - (e << 20), __double2loint(d)));
  return __hiloint2double(__double2hiint(v) - ((e >> 1) << 20), __double2loint(v));
}

}  // namespace ttgb
