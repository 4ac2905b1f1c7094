// rd_bounds.h -- rounding bounds of the planar near / far split (rd_near.cuh), as plain
// functions that a host check can evaluate too.  u = 2^-24 (5.97e-8 with a little room).
#pragma once

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
