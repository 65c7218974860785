// jitter.h - k / 10000 for the march jitter's draws k = 0 .. 1000, correctly
// rounded without a division: Markstein's final step (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor",
// IBM J. Res. Dev. 34, 1990) corrects the product with the rounded reciprocal
// by its exact remainder.  Equal to the IEEE quotient for every such k (tested
// over all of them); 3 FP64 operations instead of a division.
#pragma once
#include <math.h>

#ifndef MBR_HD
#ifdef __CUDACC__
#define MBR_HD __host__ __device__
#else
#define MBR_HD
#endif
#endif

namespace mbr {

inline MBR_HD double tenthousandths(int k) {
  const double y = 1e-4, d = double(k);
  const double q = d * y;
  return fma(fma(-10000.0, q, d), y, q);
}

}  // namespace mbr
