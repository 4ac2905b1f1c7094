// rd_bounds.h -- rounding bounds of the planar near / far split (rd_near.cuh), as plain
// functions that a host check can evaluate too.  u = 2^-24 (5.97e-8 with a little room).
#pragma once
#include <cmath>

#include "rd_split.h"

#ifndef RD_HD
#ifdef __CUDACC__
#define RD_HD __host__ __device__ __forceinline__
#else
#define RD_HD inline
#endif
#endif

#define RD_U24 5.97e-8f
#define RD_NEAR_UNITS 250.0f   // 153 pair sum, 25 a term, 36 runs of 32 terms and lanes, 30 evaluation
#define RD_NEAR_RUN 32         // terms that a lane adds before the run joins its sum

// Units of u of |S| that the estimate at a point may be off beside the far part, for
// P panels per side and `cnt` near electrons: eight lanes add them in runs of
// RD_NEAR_RUN, so each sum takes cnt / 256 more additions.
RD_HD float rd_near_units(int P, int cnt) {
  return RD_NEAR_UNITS + 0.6f * (float)P + (float)cnt * (1.0f / (8 * RD_NEAR_RUN));
}

// The nodes' near sums: two lanes each, a run per 64 electrons.  As a factor on the
// nodes' largest magnitude, which the bound takes RD_NEAR_UNITS + .. times.
RD_HD float rd_near_node_factor(int cnt) { return 1.0f + (float)cnt * (1.0f / (2 * RD_NEAR_RUN * RD_NEAR_UNITS)); }

// Direct sums over all n electrons by nt threads, runs of eight terms (near_open).
RD_HD float rd_near_direct_units(int n, int nt) { return RD_NEAR_UNITS + (float)n / (float)(8 * nt); }

// a - 1/2 log v for v > 0 (a tip's log phi and xi^2 - eta^2), without the ulp of a large
// logarithm: v = m 2^k with m in [2/3, 4/3), k (log 2) / 2 in two parts, the first exact;
// log_m is log m.  With e = 2^-24 and log_m within 2e of itself the error is at most 1.4e +
// 2e |result|, the rounding of v included, in a difference of two results with one a.
RD_HD float rd_log_parts(float v, float* kf) {
  const int b = (int)rd_bits_of_float(v), k = (b - 0x3f2aaaab) >> 23;
  *kf = (float)k;
  return rd_float_of_bits((uint32_t)(b - k * 0x800000));
}
RD_HD float rd_less_half_log(float a, float kf, float log_m) {
  return fmaf(kf, -0.34655761719f, a) + fmaf(-0.5f, log_m, kf * -1.5973092e-5f);
}

// Guard of a decision from FP32 targets (near_decide): how far
//   df = 2 log(F_n / F_c) - (rho_n - rho_c)  and  log u
// as FP32 forms them can lie from what the same fields give in FP64, S the sum of
// their magnitudes.  With e = 2^-24, logf and log1pf within 1 ulp (2e of the result):
//   the fields rounded to floats 4e, their quotient 2e, its logarithm 2e |2 log|;
//   each rho 1.95e + 2e |rho| (mh_guard has the terms), at a tip 1.6e + e |rho| more
//   (rd_less_half_log);
//   log u 2.01e + 2e |log u|, three sums rounded.
// Planar 12.2e + 5e S, tip 15.4e + 6e S.  The guard is a sixth above the tip's.
RD_HD float rd_near_guard(float S) { return 1.06e-6f + 4.3e-7f * S; }
