// The searches of the basis-state sampler (qg_extra.cu).
//
// Running sums that several threads join are not monotone in the last bit, so
// the place that a search finds may hold no weight.  Both searches end on one
// that does (where there is any): a state of zero weight is never drawn.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define QG_HD __host__ __device__ __forceinline__
#else
#define QG_HD inline
#endif

namespace qg {

// Last chunk whose prefix is at most u, or the next lower one with weight, or
// else the first with weight.  prefix[nb] is the total (0 or NaN: chunk 0).
QG_HD int64_t pick_chunk(const double* prefix, const double* sums, int64_t nb, double u) {
  int64_t lo = 0, hi = nb - 1;
  while (lo < hi) {
    const int64_t mid = (lo + hi + 1) >> 1;
    if (prefix[mid] <= u)
      lo = mid;
    else
      hi = mid - 1;
  }
  while (lo > 0 && !(sums[lo] > 0.0)) --lo;
  if (prefix[nb] > 0.0)
    while (lo < nb - 1 && !(sums[lo] > 0.0)) ++lo;
  return lo;
}

// First index with weight from the first running sum above u on, or else the
// last one with weight.  weight: a bit per index (bit x % 8 of byte x / 8).
QG_HD int pick_index(const double* cdf, const uint8_t* weight, int N, double u, int last) {
  int lo = 0, hi = N;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (cdf[mid] > u)
      hi = mid;
    else
      lo = mid + 1;
  }
  for (; lo < N; lo = (lo | 7) + 1) {
    unsigned bits = (unsigned)weight[lo >> 3] >> (lo & 7);
    for (int x = lo; bits; ++x, bits >>= 1)
      if (bits & 1) return x;
  }
  return last;
}

}  // namespace qg
