// 64-bit fixed-point arithmetic of the complex128 kernels (qg_fixed.cu,
// qg_batched_fix.cu): products, butterflies, exchange layouts, phases.
#pragma once
#include <stdint.h>

#include "qg_fixed.h"
#include "qg_fixed_layout.cuh"

namespace qg {

using i64 = long long;


__device__ __forceinline__ i64 mad_wide(int a, int b, i64 c) {
  i64 d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
  return d;
}
// A launch constant that the compiler must treat as new: a branch on it inside
// the tile loop is then not unswitched (copies of the loop body per option
// overran the instruction cache).
__device__ __forceinline__ int opaque(int x) {
  asm volatile("" : "+r"(x));
  return x;
}
// x = h * 2^32 + l with l signed
struct Limbs {
  int h, l;
};
__device__ __forceinline__ Limbs limbs(i64 x) {
  const int lo = (int)x;
  return {(int)(x >> 32) - (lo >> 31), lo};
}

// (re + i im) *= (cos + i sin) 2^-(64 - b): the phase's cosine (d.x d.y) and
// sine (d.z d.w) as limbs at 2^b, the product's top 64 bits (low x low
// dropped, rounded)
template <bool CONJ>
__device__ __forceinline__ void cmul_fix(i64& re, i64& im, int4 d) {
  const Limbs r = limbs(re), i = limbs(im);
  const int sh = CONJ ? -d.z : d.z, sl = CONJ ? -d.w : d.w;
  const i64 half = 0x80000000ll;
  const i64 m = mad_wide(i.l, -sh, mad_wide(i.h, -sl, mad_wide(r.l, d.x, mad_wide(r.h, d.y, half))));
  const i64 q = mad_wide(r.l, sh, mad_wide(r.h, sl, mad_wide(i.l, d.x, mad_wide(i.h, d.y, half))));
  re = mad_wide(i.h, -sh, mad_wide(r.h, d.x, m >> 32));
  im = mad_wide(r.h, sh, mad_wide(i.h, d.x, q >> 32));
}

// V^-1 (INV) or V on the in-thread bits of a stage, times sqrt(2) per X/Y bit:
//   X: V^-1 = [[1, 1], [-1, 1]], V = [[1, -1], [1, 1]]
//   Y: V^-1 = [[1, -i], [-i, 1]], V = [[1, i], [i, 1]]
// (V Z V^-1 = 2 P).  Both are pairs of real butterflies
//   (u, v) -> (u + v, v - u)   and   (u, v) -> (u - v, u + v)
// done in place -- v -= u, u = 2 u + v -- so that the branches on the axis
// meet without register moves.
__device__ __forceinline__ void bf_a(i64& u, i64& v) {  // (u + v, v - u)
  v -= u;
  u = (u << 1) + v;
}
__device__ __forceinline__ void bf_b(i64& u, i64& v) {  // (u - v, u + v)
  u -= v;
  v = (v << 1) + u;
}
template <bool INV>
__device__ __forceinline__ void butterflies(i64* re, i64* im, int code) {
#pragma unroll
  for (int i = 0; i < E; ++i) {
    const int ty = (code >> (2 * i)) & 3;
    // warp-uniform branch around the whole unrolled block
    if (ty == 1) {
#pragma unroll
      for (int c = 0; c < NA; ++c)
        if (!((c >> i) & 1)) {
          const int e = c | (1 << i);
          if (INV)
            bf_a(re[c], re[e]), bf_a(im[c], im[e]);
          else
            bf_b(re[c], re[e]), bf_b(im[c], im[e]);
        }
    } else if (ty == 2) {
#pragma unroll
      for (int c = 0; c < NA; ++c)
        if (!((c >> i) & 1)) {
          const int e = c | (1 << i);
          if (INV)  // (a - i b, b - i a)
            bf_a(re[c], im[e]), bf_b(im[c], re[e]);
          else  // (a + i b, b + i a)
            bf_b(re[c], im[e]), bf_a(im[c], re[e]);
        }
    }
  }
}

// ------------------------------------------------------------ right shifts
//
// A shift by one bit meets a tie every other time.  All rounded up, they moved
// every component by a quarter of a unit, the same way each time, and that
// adds up where a state's amplitudes are alike: gradients by small X angles in
// the batched kernel were 3.5e-14 off (n = 14, 20 layers of angles below 0.01;
// now 9e-16, double sweeps 2.2e-15).  So half of a thread's components round
// ties up and half down, and which half is a bit of a hash of thread, tile and
// sweep: the errors are those of independent roundings again.
__device__ __forceinline__ unsigned dither_bit(int tile, int sweep) {
  unsigned x = threadIdx.x * 0x9e3779b1u + (unsigned)tile * 0x85ebca6bu + (unsigned)sweep * 0xc2b2ae35u;
  x ^= x >> 15;
  x *= 0x2c1b3c6du;
  return x >> 31;
}
__host__ __device__ constexpr bool dither_odd(int c) { return (c ^ (c >> 1) ^ (c >> 2)) & 1; }
// (x + half) >> s, 1 <= s < 32
__device__ __forceinline__ void shift_right(i64* re, i64* im, int s, unsigned dither) {
  const unsigned a = (1u << (s - 1)) - dither, b = (1u << (s - 1)) - 1 + dither;
#pragma unroll
  for (int c = 0; c < NA; ++c) {
    re[c] = (re[c] + (dither_odd(c) ? a : b)) >> s;
    im[c] = (im[c] + (dither_odd(c) ? b : a)) >> s;
  }
}

// ------------------------------------------------------------ phases
//
// A phase's error acts on the whole state, so phases are computed in 62-bit
// fixed point as well: products of ten double sines and cosines alone doubled
// a gradient's error at n = 10.  Sine and cosine: reduction by a 128-bit 2/pi
// and the Taylor series on [-pi/4, pi/4], absolute error below 2.2 * 2^-62;
// angles from 2^20 on take the double functions.

using u128 = unsigned __int128;
using i128 = __int128;

struct Unit {  // cosine and sine at 2^62
  i64 c, s;
};

__device__ __forceinline__ i64 mul62(i64 a, i64 b) { return (i64)(((i128)a * b + ((i128)1 << 61)) >> 62); }
__device__ __forceinline__ Unit mul62(Unit a, Unit b) {
  const i128 h = (i128)1 << 61;
  return Unit{(i64)(((i128)a.c * b.c - (i128)a.s * b.s + h) >> 62), (i64)(((i128)a.c * b.s + (i128)a.s * b.c + h) >> 62)};
}

// quarter turns of a >= 0 radians, a < 2^20: a (2 / pi) 2^80
__device__ __forceinline__ u128 quarter_turns(double a) {
  const int hi = __double2hiint(a), ex = hi >> 20;
  if (ex == 0) return 0;
  const uint64_t m = ((uint64_t)((hi & 0xfffff) | 0x100000) << 32) | (unsigned)__double2loint(a);  // a = m 2^(ex-1075)
  // 2 / pi = 0.a2f9836e 4e441529 fc2757d1 f534ddc0... (hexadecimal)
  const u128 top = (u128)m * 0xa2f9836e4e441529ull + (((u128)m * 0xfc2757d1f534ddc0ull) >> 64);
  const int sh = 1059 - ex;  // >= 17
  return sh < 128 ? top >> sh : (u128)0;
}

__device__ __forceinline__ Unit unit_of(u128 turns) {
  const u128 t = turns >> 16;
  const uint64_t frac = (uint64_t)t;
  const int q = (int)((uint64_t)(t >> 64) + (frac >> 63)) & 3;
  const i64 one = 1ll << 62;
  const i64 r = (i64)(((i128)(i64)frac * 0x6487ed5110b4611all) >> 64);  // times pi / 2
  const i64 z = mul62(r, r);
  i64 s = one, c = one;
#pragma unroll
  for (int k = 9; k >= 1; --k) s = one - mul62(mul62(z, (one + k * (2 * k + 1)) / (2 * k * (2 * k + 1))), s);
#pragma unroll
  for (int k = 10; k >= 1; --k) c = one - mul62(mul62(z, (one + k * (2 * k - 1)) / (2 * k * (2 * k - 1))), c);
  s = mul62(r, s);
  return q == 0 ? Unit{c, s} : q == 1 ? Unit{-s, c} : q == 2 ? Unit{-c, -s} : Unit{s, -c};
}

__device__ __forceinline__ Unit unit_angle(double a, bool& bad) {
  Unit u;
  if (fabs(a) < 0x1p20) {
    u = unit_of(quarter_turns(fabs(a)));
    if (a < 0) u.s = -u.s;
  } else {
    double sv, cv;
    sincos(a, &sv, &cv);
    if (!isfinite(cv)) {
      bad = true;
      cv = sv = 0.0;
    }
    u = Unit{__double2ll_rn(cv * 0x1p62), __double2ll_rn(sv * 0x1p62)};
  }
  return u;
}

// limbs at 2^(62 - down).  Products negate the sine's limbs, so its low limb
// is never -2^31 (which has no negative; one unit of 2^-60 apart).
__device__ __forceinline__ int4 phase_limbs(Unit u, int down) {
  const i64 h = down ? 1ll << (down - 1) : 0;
  const i64 c = (u.c + h) >> down;
  i64 s = (u.s + h) >> down;
  if ((int)s == (int)0x80000000) ++s;
  const Limbs a = limbs(c), b = limbs(s);
  return make_int4(a.h, a.l, b.h, b.l);
}

}  // namespace qg
