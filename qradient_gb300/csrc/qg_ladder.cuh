// The CNOT ladder as an index map, for kernels and for the host's descriptors.
#pragma once
#include <stdint.h>

namespace qg {

// Reference CNOT ladder as a basis permutation: CNOT(q, q+1) flips bit
// (n-2-q) when bit (n-1-q) is set, i.e. x ^= (x & bit_c) >> 1.  The odd-pair
// CNOTs act first, then the even pairs (state.py:235-241).  The pairs of one
// parity are disjoint, so each parity is one masked shift-xor.  The periodic
// ladder (state.py:218-219, even n) adds CNOT(n-1, 0) to the odd pairs: bit
// n-1 flips when bit 0 is set, x ^= (x & wrap) << (n - 1).
struct LadderMasks {
  uint64_t odd, even, wrap;
  int wshift;
};

__host__ __device__ __forceinline__ LadderMasks ladder_masks(int n, bool periodic) {
  LadderMasks m{0, 0, periodic ? 1ull : 0ull, n - 1};
  for (int q = 0; q + 1 < n; ++q) {
    const uint64_t b = 1ull << (n - 1 - q);
    if (q & 1)
      m.odd |= b;
    else
      m.even |= b;
  }
  return m;
}

// A(x): ladder |x> = |A(x)>
__host__ __device__ __forceinline__ uint64_t ladder_fwd(uint64_t x, const LadderMasks& m) {
  x ^= ((x & m.odd) >> 1) ^ ((x & m.wrap) << m.wshift);
  x ^= (x & m.even) >> 1;
  return x;
}
// A^{-1}(x)
__host__ __device__ __forceinline__ uint64_t ladder_inv(uint64_t x, const LadderMasks& m) {
  x ^= (x & m.even) >> 1;
  x ^= ((x & m.odd) >> 1) ^ ((x & m.wrap) << m.wshift);
  return x;
}

}  // namespace qg
