// Exchange layouts and scaling schedule of the fixed-point kernels: host code
// too (tests/test_fixed_layouts.py compiles this header with g++).
#pragma once
#include <algorithm>

#include "qg_fixed.h"

namespace qg {

// ------------------------------------------------------------ layouts
//
// A thread holds NA = 2^E amplitudes; stage s has local bits T-E(s+1)..T-Es-1
// in the thread (the last stage, where fewer remain, the r low bits filled up
// with the top ones).  The exchange buffer between stages is XOR-swizzled on
// 16-byte slots so that the eight lanes of a quarter warp hit eight bank
// groups: in every stage with eight amplitudes a thread, in all but the one
// before the last with four (two lanes to a group there).
#ifndef QG_FIX_E
#define QG_FIX_E 3
#endif
constexpr int E = QG_FIX_E, NA = 1 << E;

template <int T, int = QG_FIX_E>  // (a type of its own per translation unit's E)
struct Lay {
  static constexpr int NT = 1 << (T - E);
  __host__ __device__ static constexpr int sw(int e) { return e ^ ((e >> 3) & 7); }
  // local index of (thread 0, in-thread index c)
  __host__ __device__ static constexpr int eoff(int s, int c) {
    const int lo = T - E * (s + 1);
    if (lo >= 0) return c << lo;
    const int r = E + lo;  // low bits in the thread
    return (c & ((1 << r) - 1)) | ((c >> r) << (T + lo));
  }
  // local index of (thread tid, in-thread index 0)
  __host__ __device__ static constexpr int ebase(int s, int tid) {
    const int lo = T - E * (s + 1);
    if (lo >= 0) return (tid & ((1 << lo) - 1)) | ((tid >> lo) << (lo + E));
    return tid << (E + lo);
  }
  static constexpr int NS = (T + E - 1) / E;
};

// The scaling of a sweep, from the number of its butterfly levels alone.  h
// counts half bits of the tile's norm above 2^60: a level adds one, a phase
// product takes eight (its table is scaled by 2^60), the cost product four
// (2^62), a shift by s takes 2 s.  LIM = 5 keeps the norm, and so every
// component and every sum inside a product, below 2^62.5.  Up to nine levels
// need no shift: the tile is loaded at the B (58..62) that lets V^-1 grow to
// LIM, and the phase product makes the room that V needs.  h never falls below
// -4, so a tile's unit is at most 2^-58 of the power of two above its norm,
// 2^-57 of the norm.
inline void fix_schedule(FixDesc& d) {
  constexpr int LIM = 5;
  int m[FIX_STAGES] = {};
  int levels = 0;
  for (int s = 0; s < d.nst; ++s) {
    for (int i = 0; i < FIX_E; ++i) m[s] += ((d.code[s] >> (2 * i)) & 3) != 0;
    levels += m[s];
  }
  for (int dir = 0; dir < 2; ++dir) {
    int total = 0;  // right shifts so far
    int h;
    if (dir == 0 && d.cost == COST_INT) {
      d.B[0] = 62;
      h = 0;  // after the cost product
      total += 2;
    } else {
      const int up = levels <= LIM ? (LIM - levels) / 2 : -((levels - LIM + 1) / 2);
      d.B[dir] = (int8_t)(60 + std::max(-2, std::min(2, up)));
      h = 2 * (d.B[dir] - 60);
    }
    auto room = [&](int mm) {
      const int over = h + mm - LIM;
      const int s = over > 0 ? (over + 1) / 2 : 0;
      h += mm - 2 * s;
      total += s;
      return (int8_t)s;
    };
    d.sh_in[dir][0] = 0;
    h += m[0];
    for (int s = 1; s < d.nst; ++s) d.sh_in[dir][s] = room(m[s]);
    if (dir == 1) d.kw = (int16_t)(64 - 2 * d.B[1] - levels + 2 * total);
    h -= 8;
    total += 4;
    for (int s = d.nst - 1; s >= 0; --s) d.sh_out[dir][s] = room(m[s]);
    if (dir == 1 && d.cost == COST_INT) total += 2;
    d.kout[dir] = (int16_t)(-d.B[dir] - levels + total);
  }
}

}  // namespace qg
