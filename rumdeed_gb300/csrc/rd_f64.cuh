// rd_f64.cuh -- inverse cubes of distances in FP64.
//
// The FP64 pair sums are bound by this part's FP64 pipe (about two operations per
// SM and clock), and sqrt and the division of 1 / (sqrt(s) + l^2)^3 are some
// twenty of a pair's fifty operations.  Here the FP32 reciprocal root gives a seed
// y of 1 / sqrt(s), |1 - s y^2| < 1e-6, and the rest is the binomial series
//   s^{-3/2} = y^3 (1 - e)^{-3/2} = y^3 (1 + 3/2 e + 15/8 e^2 + O(e^3)),
//   e = 1 - s y^2,
// whose next term is below 2.2e-18.  y has 24 bits, so y^2 is exact and e has one
// rounding; the result has the roundings of y^3 and of the last step, where sqrt,
// the addition, two products and the division left up to six halves of an ulp.  The
// l^2 of the reference's r + l^2 (l = 1 nm, so l^2 = 1e-18 m) enters as (1 + u)^-3,
// u = l^2 / r = l^2 y (1 + e / 2 + ..): with w = 3 l^2 y the whole factor is
//   1 + (3/2 + 15/8 e - 2 w) e - w + O(w^2, e^3, w e^2).
// w stays below 1.5e-9 for the distances this path takes (2 nm on), so w from FP32
// is off by less than 2e-16 there, and w^2 terms by 1.5e-18.  Closer pairs and
// anything out of FP32's range take the plain formula.  The conversions between
// float and double, and 3/2 - 2 w, are made of integer operations on the bits: cvt
// runs on the FP64 pipe too.
//
// Measured at one chunking (chunks of 1024): forces of 6000 electrons with one image
// partner 5.43 -> 2.88 ms; a step of 1300 electrons and 960 chains 109.7 -> 55.0 ms.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

// s in [4e-18, 1e30) m^2, by the high word
__device__ __forceinline__ bool rd_cube_ok(double s) {
  const unsigned h = (unsigned)__double2hiint(s);
  return h - 0x3c527285u < 0x46293e59u - 0x3c527285u;
}

// float of a positive normal double in FP32's range, the mantissa cut off
__device__ __forceinline__ float rd_cut_float(double s) {
  return __uint_as_float(__funnelshift_l((unsigned)__double2loint(s), (unsigned)__double2hiint(s) - 0x38000000u, 3));
}
// double of a positive normal float
__device__ __forceinline__ double rd_wide(float f) {
  const unsigned b = __float_as_uint(f);
  return __hiloint2double((int)((b >> 3) + 0x38000000u), (int)(b << 29));
}

// 3/2 - d 2^-52 for 0 <= d < 2^31
__device__ __forceinline__ double rd_three_halves_less(unsigned d) {
  return __longlong_as_double(0x3ff8000000000000ll - (long long)d);
}
#define RD_2P53 9007199254740992.0f

// 1 / (sqrt(s) + L2)^3 for rd_cube_ok(s), L2x3 = 3 L2; *bare: s^{-3/2} if asked for
template <bool BARE = false>
__device__ __forceinline__ double rd_inv_cube(double s, float L2x3, double* bare = nullptr) {
  const float yf = rsqrtf(rd_cut_float(s)), wf = yf * L2x3;
  const double y = rd_wide(yf);
  const double y2 = y * y, e = fma(-s, y2, 1.0), y3 = y2 * y;
  const double c = fma(1.875, e, rd_three_halves_less(__float2uint_rz(wf * RD_2P53)));
  if (BARE) *bare = fma(y3, fma(1.875, e, 1.5) * e, y3);
  return fma(y3, fma(c, e, -rd_wide(wf)), y3);
}
// s^{-3/2} for rd_cube_ok(s)
__device__ __forceinline__ double rd_inv_cube0(double s) {
  const double y = rd_wide(rsqrtf(rd_cut_float(s)));
  const double y2 = y * y, e = fma(-s, y2, 1.0), y3 = y2 * y, c = fma(1.875, e, 1.5);
  return fma(y3, c * e, y3);
}
// the plain formula
__device__ __forceinline__ double rd_inv_cube_any(double s, double L2) {
  const double r = sqrt(s) + L2;
  return 1.0 / ((r * r) * r);
}
