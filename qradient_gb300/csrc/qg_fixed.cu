// Fixed-point sweeps: the complex128 forward and adjoint sweeps in 64-bit
// integer arithmetic.
//
// Why.  GB300 has two FP64 lanes per SM and clock: a warp's double
// instruction holds the pipe 16 cycles, and a rotation (2 DFMA per amplitude
// forward, 4 backward) made the double sweeps FP64-bound at a tenth of HBM
// bandwidth.  A 64-bit integer add takes 0.55 SM cycles per warp.  So a
// rotation exp(-i theta/2 P) is applied as V D V^-1: V is the Clifford that
// maps P to Z (X: Hadamard H; Y: S H; Z: none), D the diagonal phase.  V is
// additions only.  All rotations of a sweep commute, so the tile goes through
// V^-1 on every active bit, one multiply by the product of all phases (a
// table), and V on every active bit.  The adjoint's reductions become
// diagonal too: Im<lam|P_q|psi> = sum_x s_q(x) w_x in the frame of V^-1, with
// one w_x = Im(conj(lam_x) psi_x) per amplitude for all qubits.
//
// Number format.  States stay complex128 in memory.  A tile is loaded, scaled
// by a power of two that puts its 2-norm below 2^B (B = 58..62), and rounded to
// int64; sums are exact; products keep the top 64 of 128 bits.
// The norm bounds every component at every later point, because V, D are
// unitary up to the known factor sqrt(2) per butterfly level, so right shifts
// scheduled from the level counts alone (fix_schedule) rule out overflow.
// A unit is at most 2^-57 of the tile's norm.  The typical one of 2^12
// components keeps 52 bits or more; the rounding of a whole sweep (one
// conversion, at most four shifts, one product) is below that of the double
// rotations it replaces.  Components far below the tile's norm keep fewer bits
// (relative to themselves) than double would: results are as close as the
// double sweeps' in norm, not element by element.
//
// Reference mapping (qradient, pure numpy):
//   rotations          physical_components/state.py:90-97, 142-149, 168-175
//   McClean grad_run   circuit_logic/mc_clean.py:47-78
//   QAOA grad_run      circuit_logic/qaoa.py:40-70
#include <algorithm>
#include <atomic>
#include <mutex>
#include <type_traits>

#include "qg_fixed_math.cuh"
#include "qg_sweep_common.cuh"

namespace qg {

namespace {

// From stage A's layout to stage B's.  The swizzle is linear: slot(c) is the
// thread's base XOR the image of c, of which only the low three bits meet the
// base's.  Every stage rewrites the slots it read, so one barrier per
// exchange suffices.
template <int T, int A, int B>
__device__ __forceinline__ void exchange(unsigned char* ex, i64* re, i64* im) {
  const int a = Lay<T>::sw(Lay<T>::ebase(A, threadIdx.x)) * 16, b = Lay<T>::sw(Lay<T>::ebase(B, threadIdx.x)) * 16;
#pragma unroll
  for (int c = 0; c < NA; ++c) {
    const int o = Lay<T>::sw(Lay<T>::eoff(A, c)) * 16;
    *(longlong2*)(ex + (a ^ (o & 112)) + (o & ~112)) = make_longlong2(re[c], im[c]);
  }
  __syncthreads();
#pragma unroll
  for (int c = 0; c < NA; ++c) {
    const int o = Lay<T>::sw(Lay<T>::eoff(B, c)) * 16;
    const longlong2 v = *(const longlong2*)(ex + (b ^ (o & 112)) + (o & ~112));
    re[c] = v.x;
    im[c] = v.y;
  }
}
// between the neighbouring stages s-1 and s (UP: to s)
template <int T, bool UP, int S = 1>
__device__ __forceinline__ void exchange_at(unsigned char* ex, i64* re, i64* im, int s) {
  if (S == Lay<T>::NS - 1 || s == S)
    exchange<T, UP ? S - 1 : S, UP ? S : S - 1>(ex, re, im);
  else if constexpr (S < Lay<T>::NS - 1)
    exchange_at<T, UP, S + 1>(ex, re, im, s);
}

// ------------------------------------------------------------ stages

__device__ __forceinline__ void shift_all(i64* re, i64* im, int s, unsigned dither) {
  if (s) shift_right(re, im, s, dither);
}

// V^-1 on all active bits, from stage 0's layout to the last stage's
template <int T>
__device__ __forceinline__ void to_frame(unsigned char* ex, i64* re, i64* im, const FixDesc& d, int dir,
                                         unsigned dither) {
#pragma unroll 1
  for (int s = 0;;) {
    butterflies<true>(re, im, d.code[s]);
    if (++s == opaque(d.nst)) break;
    exchange_at<T, true>(ex, re, im, s);
    shift_all(re, im, d.sh_in[dir][s], dither);
  }
}
template <int T>
__device__ __forceinline__ void from_frame(unsigned char* ex, i64* re, i64* im, const FixDesc& d, int dir,
                                           unsigned dither) {
#pragma unroll 1
  for (int s = opaque(d.nst) - 1;;) {
    shift_all(re, im, d.sh_out[dir][s], dither);
    butterflies<false>(re, im, d.code[s]);
    if (--s < 0) break;
    exchange_at<T, false>(ex, re, im, s + 1);
  }
}

// multiply by the phase table (conjugated for the inverse)
template <int T, bool CONJ>
__device__ __forceinline__ void phase_mul(i64* re, i64* im, const int4* tab, int nst) {
  const int lo = T - E * nst;
  const int skip = lo > 0 ? lo : 0;
  const int w = 1 << (T - E - skip);
  const int4* t = tab + (threadIdx.x >> skip);
#pragma unroll
  for (int c = 0; c < NA; ++c) cmul_fix<CONJ>(re[c], im[c], __ldg(t + c * w));
}

// ------------------------------------------------------------ addresses

// element offset of in-thread index c from the offsets of its bits
__device__ __forceinline__ i64 combine(const int64_t (&o)[FIX_E], int c) {
  i64 x = 0;
#pragma unroll
  for (int i = 0; i < E; ++i)
    if ((c >> i) & 1) x ^= o[i];
  return x;
}

// global index of (thread, in-thread index 0) of stage 0's layout, tile 0
template <int T>
__device__ __forceinline__ i64 thread_index(const FixDesc& d) {
  const int t = threadIdx.x;
  return (i64)(t & ((1 << d.low) - 1)) | (i64)(t >> d.low) << d.lo;
}
// global index of a tile's first element: its number's bits outside the tile
__device__ __forceinline__ i64 tile_base(const FixDesc& d, int tile) {
  const int mid = d.lo - d.low;  // outside bits below the active ones (none in sweep A: lo = low = 0)
  return (i64)(tile & ((1 << mid) - 1)) << d.low | (i64)(tile >> mid) << (d.lo + d.t - d.low);
}

__device__ __forceinline__ LadderMasks masks_of(const FixDesc& d) {
  return LadderMasks{d.odd, d.even, d.periodic ? 1ull : 0ull, d.n - 1};
}

// Load one tile of v, undoing or applying an entangler.  CNOT: the ladder is
// a GF(2)-linear map of the index, so the image of an element is the XOR of
// the images of its parts (`src`: that of tile and thread, `top` those of the
// in-thread bits).
__device__ __forceinline__ void load_tile(double2* raw, const double2* v, int ent, i64 x, i64 src,
                                          const int64_t (&top)[FIX_E], const int64_t (&ltop)[FIX_E]) {
  if (ent == ENT_CNOT) {
#pragma unroll
    for (int c = 0; c < NA; ++c) raw[c] = v[src ^ combine(ltop, c)];
  } else {
    const double2* q = v + x;
#pragma unroll
    for (int c = 0; c < NA; ++c) raw[c] = q[combine(top, c)];
    if (ent == ENT_CZ) {
#pragma unroll
      for (int c = 0; c < NA; ++c)
        if (cz_negative((uint64_t)(x ^ combine(top, c)))) raw[c] = cneg(raw[c]);
    }
  }
}

// ------------------------------------------------------------ scaling
//
// The power-of-two exponent p of a tile: its 2-norm is below 2^p.  The norm
// is summed in single precision (its relative error is far below the factor
// two that rounding up to a power of two leaves).  Outside the range where
// the squares are representable -- zero, tiny and huge tiles, infinities and
// NaN -- the tile is first multiplied by the power of two 2^q that brings its
// largest exponent to 0, and its results by 2^-q (both in two factors, which
// are always representable); a tile with a non-finite entry, or whose phases
// are not finite, has NaN results.

// 2^e, -1022 <= e <= 1023
__device__ __forceinline__ double pow2(int e) { return __hiloint2double((e + 1023) << 20, 0); }

struct Scale {
  int p;
  int q;  // 0: nothing more to do; kNaN: NaN results; else the power of two applied on load
};
constexpr int kNaN = 1 << 20;

template <int T>
struct NormShared {
  float s[2][Lay<T>::NT / 32 > 0 ? Lay<T>::NT / 32 : 1];
  int m[Lay<T>::NT / 32];
};

template <int T>
__device__ __forceinline__ Scale tile_scale(double2* v, NormShared<T>& N, int& par, bool poison) {
  constexpr int NW = Lay<T>::NT / 32;
  // from the high words alone, without a double instruction: the larger
  // component's bits become a float (exponent moved by 896, clamped below),
  // and |v|^2 <= 2 max^2
  float s = 0.f;
  int mx = 0;
#pragma unroll
  for (int c = 0; c < NA; ++c) {
    const int h = __vimax3_s32(__double2hiint(v[c].x) & 0x7fffffff, __double2hiint(v[c].y) & 0x7fffffff, 0x38000000);
    mx = max(mx, h);
    const float x = __int_as_float((h - 0x38000000) << 3);
    s = fmaf(x, x, s);
  }
  s = mx >= 0x47f00000 ? __int_as_float(0x7f800000) : 2.f * s * (1.f + 0x1p-18f);  // (truncated mantissas)
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) N.s[par][threadIdx.x >> 5] = s;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int w = 0; w < NW; ++w) tot += N.s[par][w];
  par ^= 1;
  if (tot >= 0x1p-60f && tot <= 0x1p100f && !poison) {  // the same in every thread
    const int e = (__float_as_int(tot) >> 23) - 127;
    return Scale{(e + 2) >> 1, 0};  // norm^2 < 2^(e+1)
  }
  Scale r;
  int m = 0;
#pragma unroll
  for (int c = 0; c < NA; ++c) m = __vimax3_s32(m, __double2hiint(v[c].x) & 0x7fffffff, __double2hiint(v[c].y) & 0x7fffffff);
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) N.m[threadIdx.x >> 5] = m;
  __syncthreads();
  m = 0;
  for (int w = 0; w < NW; ++w) m = max(m, N.m[w]);
  __syncthreads();  // N.m is free again
  r.p = 1 + (T + 2) / 2;  // norm <= max sqrt(2^(T+1))
  if (m >= 0x7ff00000 || poison) {
    r.q = kNaN;
#pragma unroll
    for (int c = 0; c < NA; ++c) v[c] = make_double2(0.0, 0.0);
    return r;
  }
  r.q = 1023 - (m >> 20);
  const double f0 = pow2(r.q >> 1), f1 = pow2(r.q - (r.q >> 1));
#pragma unroll
  for (int c = 0; c < NA; ++c) v[c] = make_double2(v[c].x * f0 * f1, v[c].y * f0 * f1);
  return r;
}

// x * 2^k to the nearest integer in integer instructions, |x * 2^k| < 2^62:
// half of the conversions take this form, so that the FP64 pipe (16 cycles per
// conversion) and the integer pipes share them (a half, a quarter, none: n = 20,
// L = 50 5.80, 6.05, 6.22 ms; n = 24 72.1, 72.0, 74.0).  `tie` 2 rounds ties
// up, 0 down, whatever the sign (see dither_bit).  Rounded down instead, as
// this was (n = 24 70.3 ms), every imaginary part was half a unit low, the
// same way in every sweep: gradients by small X angles 1.1e-13 off at n = 14
// and 20 layers (now 2.3e-15, double sweeps 2.2e-15), QAOA with small angles
// 2.1e-14 at n = 16 (2e-16, 4.0e-15).  All ties up: 9e-15 and 2.3e-15.
__device__ __forceinline__ i64 to_fix_int(double x, int k, unsigned tie) {
  const int hi = __double2hiint(x), sg = hi >> 31;
  // leading one at bit 61: |value| = m 2^(ex - 1084); negative values in ones'
  // complement, one less than the two's: `tie` - 1 beside it is 1 or -1
  const unsigned lo = (unsigned)__double2loint(x);
  const unsigned mh = ((__funnelshift_l(lo, (unsigned)hi, 9) & 0x1fffffffu) | 0x20000000u) ^ (unsigned)sg;
  const int r = min(1084 - k - ((hi >> 20) & 0x7ff), 63);  // 0..63 (beyond: below a quarter, as at 63)
  const i64 m = (i64)((uint64_t)mh << 32 | ((lo << 9) ^ (unsigned)sg));
  uint64_t below;  // 2^(r-1) - 1, or 0 for r < 2: a whole number then, off by two of 2^60 at most
  asm("shr.u64 %0, %1, %2;" : "=l"(below) : "l"(~0ull), "r"(65 - r));
  return (m + (i64)below + (i64)(uint64_t)tie) >> r;
}
// x * 2^k to the nearest integer; |x * 2^k| < 2^63
__device__ __forceinline__ i64 to_fix(double x, int k) {
  // the exponent field moves by k; zeros and denormals become a value below
  // one half for every k < 1022, and 7 <= k <= 91 on this path
  return __double2ll_rn(__hiloint2double(__double2hiint(x) + (k << 20), __double2loint(x)));
}
// X * 2^-k
__device__ __forceinline__ double from_fix(i64 X, int k) {
  const double v = (double)X;
  const int hi = __double2hiint(v);
  return __hiloint2double(hi ? hi - (k << 20) : 0, __double2loint(v));
}
__device__ __forceinline__ void load_fix(const double2* raw, i64* re, i64* im, const Scale& s, int B, unsigned dither) {
  const int k = B - s.p;
  const unsigned a = 2 * dither, b = 2 - a;
#pragma unroll
  for (int c = 0; c < NA; ++c) {
    re[c] = to_fix(raw[c].x, k);
    im[c] = to_fix_int(raw[c].y, k, dither_odd(c) ? a : b);
  }
}

// what undoes the slow tiles' scaling, in two factors
__device__ __forceinline__ double2 unscale(int q) {
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  return q == kNaN ? make_double2(nan, nan) : make_double2(pow2(-(q >> 1)), pow2(-(q - (q >> 1))));
}

// results of stage 0's layout to memory
__device__ __forceinline__ void store_tile(double2* out, const i64* re, const i64* im, const Scale& s, int kout,
                                           const int64_t (&top)[FIX_E]) {
  const int k = -(s.p + kout);
  if (s.q == 0) {
#pragma unroll
    for (int c = 0; c < NA; ++c) out[combine(top, c)] = make_double2(from_fix(re[c], k), from_fix(im[c], k));
  } else {
    const double2 f = unscale(s.q);
#pragma unroll
    for (int c = 0; c < NA; ++c)
      out[combine(top, c)] = make_double2(from_fix(re[c], k) * f.x * f.y, from_fix(im[c], k) * f.x * f.y);
  }
}

// Prefetch into L2 the 128-byte lines of a tile, one of eight amplitudes per
// thread, or two threads to a line (their images under the ladder share a line as well).  Backward
// only: n = 24, L = 20 28.98 -> 28.83 ms; the forward sweeps lost 3%.
template <int T>
__device__ __forceinline__ i64 line_index(const FixDesc& d) {
  const int t = threadIdx.x << E;
  return (i64)(t & ((1 << d.low) - 1)) | (i64)(t >> d.low) << d.lo;
}
__device__ __forceinline__ void prefetch_line(const double2* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// ------------------------------------------------------------ forward

// Resident warps per SM that the registers are capped for (64 and 80 a
// thread).  At these caps the sweeps of up to 11 bits spill 56-204 bytes a
// thread; with 24 and 16 warps (80 and 128 registers) nothing spills, and
// n = 24, L = 20 takes 29.6 against 28.8 ms (n = 22, L = 10 3.82 against 3.92,
// n = 18, L = 20 933 against 965 us).
constexpr int fwd_warps = 32, bwd_warps = 24;

template <int T>
__global__ void __launch_bounds__(Lay<T>::NT, fwd_warps / (Lay<T>::NT / 32))
    fix_fwd_kernel(const __grid_constant__ FixDesc d, FixPtrs p) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ NormShared<T> N;
  const i64 dep = thread_index<T>(d);
  const int ntiles = 1 << (d.n - T);
  int par = 0;
  pdl_wait();
  const bool poison = p.flags[d.sweep] != 0;
  const int4* tab = (const int4*)(p.area + d.tab);
  const int4* ctab = (const int4*)(p.area + d.ctab);
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const i64 x = tile_base(d, tile) | dep;
    const i64 src = (i64)ladder_inv((uint64_t)x, masks_of(d));
    const unsigned dither = dither_bit(tile, d.sweep);
    double2 raw[NA];
    if (opaque(d.start) == START_LOAD) {
      load_tile(raw, p.psi_in, opaque(d.pre), x, src, d.top, d.top_inv);
    } else {
#pragma unroll
      for (int c = 0; c < NA; ++c) {
        const uint64_t y = (uint64_t)(x ^ combine(d.top, c));
        const uint64_t from = opaque(d.pre) == ENT_CNOT ? (uint64_t)(src ^ combine(d.top_inv, c)) : y;
        raw[c] = make_double2(p.startp[__popcll(from)], 0.0);
        if (opaque(d.pre) == ENT_CZ && cz_negative(y)) raw[c] = cneg(raw[c]);
      }
    }
    const Scale s = tile_scale<T>(raw, N, par, poison);
    i64 re[NA], im[NA];
    load_fix(raw, re, im, s, d.B[0], dither);
    if (opaque(d.cost) == COST_INT) {
      const int32_t* ci = p.cost_i + x;
#pragma unroll
      for (int c = 0; c < NA; ++c) cmul_fix<false>(re[c], im[c], __ldg(ctab + ci[combine(d.top, c)] + d.cost_maxabs));
    }
    to_frame<T>(smem, re, im, d, 0, dither);
    phase_mul<T, false>(re, im, tab, opaque(d.nst));
    from_frame<T>(smem, re, im, d, 0, dither);
    store_tile(p.psi_out + x, re, im, s, d.kout[0], d.top);
    // The next launch may come in once every CTA has stored its last tile.
    // Triggered at the start, its CTAs waited on
    // the SMs beside this grid's, and filled a few of them when a grid is
    // smaller than the chip holds (n = 18, L = 20: 1.89 -> 1.07 ms).
    if (tile + (int)gridDim.x >= ntiles) pdl_trigger();
  }
}

// ------------------------------------------------------------ backward

// EARLY (history mode, few tiles per CTA): what a sweep does to psi needs only
// the forward pass, so a chain of backward sweeps brings the first tile's psi
// into the frame before it waits for the sweep ahead of it, which lets it in
// as it starts on its last tile (after its own wait, so that the chain is two
// deep and everything up to the sweep before the last is complete).  n = 10,
// L = 10: 248 -> 223 us; n = 15, L = 20: 590 -> 525; n = 17: 759 -> 706;
// n = 18: 1057 -> 965; n = 20: 2400 -> 2233.  Triggered before the wait,
// waiting CTAs piled up on some SMs (n = 18: 985 -> 1498).
template <int T, bool UNCOMPUTE, bool EARLY>
__global__ void __launch_bounds__(Lay<T>::NT, bwd_warps / (Lay<T>::NT / 32) > 0 ? bwd_warps / (Lay<T>::NT / 32) : 1)
    fix_bwd_kernel(const __grid_constant__ FixDesc d, FixPtrs p) {
  constexpr int NT = Lay<T>::NT, NW = NT / 32;
  extern __shared__ __align__(16) unsigned char smem[];
  longlong2* park = (longlong2*)smem + (1 << T);  // psi in the frame: [in-thread index][thread]
  __shared__ NormShared<T> N;
  const int tid = threadIdx.x;
  const i64 dep = thread_index<T>(d);
  const int ntiles = 1 << (d.n - T);
  int par = 0;
  double Tacc = 0.0, U0 = 0.0, U1 = 0.0, U2 = 0.0, gacc = 0.0;
  bool early = EARLY && d.early;
  if (!early) pdl_wait();
  const bool poison = p.flags[d.sweep] != 0;
  const int4* tab = (const int4*)(p.area + d.tab);
  const int4* ctab = (const int4*)(p.area + d.ctab);
  const i64 line = line_index<T>(d);
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const i64 x = tile_base(d, tile) | dep;
    const i64 src = (i64)ladder_fwd((uint64_t)x, masks_of(d));
    const unsigned dither = dither_bit(tile, d.sweep);
    const bool last = tile + (int)gridDim.x >= ntiles;
    if (EARLY && last && !early) pdl_trigger();
    {
      // lambda of this tile, used once psi is in the frame; psi of the next
      const i64 y = tile_base(d, tile) | line;
      prefetch_line(p.lam_in + (opaque(d.lam_undo) == ENT_CNOT ? (i64)ladder_fwd((uint64_t)y, masks_of(d)) : y));
      const int nxt = tile + gridDim.x;
      if (nxt < ntiles) {
        const i64 z = tile_base(d, nxt) | line;
        prefetch_line(p.psi_in + (opaque(d.psi_undo) == ENT_CNOT ? (i64)ladder_fwd((uint64_t)z, masks_of(d)) : z));
      }
    }
    Scale sq;
    // psi into the frame, parked there; then lambda (one copy of the code)
#pragma unroll 1
    for (int st = 0; st < 2; ++st) {
      i64 re[NA], im[NA];
      double2 raw[NA];
      if (EARLY && st == 1 && early) {
        pdl_wait();
        early = false;
        if (last) pdl_trigger();
      }
      load_tile(raw, st ? p.lam_in : p.psi_in, opaque(st ? d.lam_undo : d.psi_undo), x, src, d.top, d.top_fwd);
      if (st == (EARLY ? 1 : 0) && opaque(d.has_gslot)) {
        // gamma of the next layer's cost: sum_x C(x) Im(conj(lam) psi), before any inverse gate
        const double2* o = (EARLY ? p.psi_in : p.lam_in) + x;
        const int32_t* ci = p.cost_i + x;
#pragma unroll
        for (int c = 0; c < NA; ++c) {
          const double2 b = o[combine(d.top, c)], a = EARLY ? raw[c] : b, q = EARLY ? b : raw[c];
          gacc = fma((double)ci[combine(d.top, c)], fma(a.x, q.y, -a.y * q.x), gacc);
        }
      }
      const Scale s = tile_scale<T>(raw, N, par, poison);
      load_fix(raw, re, im, s, d.B[1], dither);
      to_frame<T>(smem, re, im, d, 1, dither);
      if (st == 0) {
#pragma unroll
        for (int c = 0; c < NA; ++c) park[c * NT + tid] = make_longlong2(re[c], im[c]);
        sq = s;
        if (!UNCOMPUTE) continue;
      } else {
        // w = Im(conj(lam) psi) = lr qi - li qr per amplitude: V its top 64 bits,
        // f the next 28; sums over the thread's amplitudes and, per in-thread
        // bit, over those with the bit set
      {
          i64 sT = 0, s0 = 0, s1 = 0, s2 = 0;
          uint32_t fT = 0, f0 = 0, f1 = 0, f2 = 0;
#pragma unroll
          for (int c = 0; c < NA; c += 2) {
            i64 V[2];
            uint32_t f[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              const longlong2 q = park[(c + k) * NT + tid];
              const Limbs lr = limbs(re[c + k]), li = limbs(im[c + k]), qr = limbs(-q.x), qi = limbs(q.y);
              const i64 m = mad_wide(li.l, qr.h, mad_wide(li.h, qr.l, mad_wide(lr.l, qi.h, mad_wide(lr.h, qi.l, 0))));
              V[k] = mad_wide(li.h, qr.h, mad_wide(lr.h, qi.h, m >> 32));
              f[k] = (uint32_t)m >> 4;
            }
            s0 += V[1];
            f0 += f[1];
            const i64 v = V[0] + V[1];
            const uint32_t g = f[0] + f[1];
            sT += v;
            fT += g;
            if (c & 2) s1 += v, f1 += g;
            if (c & 4) s2 += v, f2 += g;
          }
          // (the fraction's carry, rounded; 28 fraction bits)
          double sc = pow2(s.p + sq.p + d.kw);
          if (s.q | sq.q) {
            const double2 a = unscale(s.q), b = unscale(sq.q);
            sc = sc * a.x * b.x * a.y * b.y;
          }
          const uint32_t r = 1u << 27;
          Tacc = fma((double)(sT + (i64)(((uint64_t)fT + r) >> 28)), sc, Tacc);
          U0 = fma((double)(s0 + (i64)(((uint64_t)f0 + r) >> 28)), sc, U0);
          U1 = fma((double)(s1 + (i64)(((uint64_t)f1 + r) >> 28)), sc, U1);
          U2 = fma((double)(s2 + (i64)(((uint64_t)f2 + r) >> 28)), sc, U2);
        }
      }
      phase_mul<T, true>(re, im, tab, opaque(d.nst));
      from_frame<T>(smem, re, im, d, 1, dither);
      if (opaque(d.cost) == COST_INT) {
        const int32_t* ci = p.cost_i + x;
#pragma unroll
        for (int c = 0; c < NA; ++c) cmul_fix<true>(re[c], im[c], __ldg(ctab + ci[combine(d.top, c)] + d.cost_maxabs));
      }
      store_tile((st ? p.lam_out : p.psi_out) + x, re, im, s, d.kout[1], d.top);
      if (!EARLY && st && last) pdl_trigger();
    }
  }
  // S_j = sum_x s_j(x) w_x = T - 2 U_j over the CTA's threads
  __syncthreads();
  double* red = (double*)smem;  // [warp][active bit], then gamma
  for (int a = 0; a < d.nact; ++a) {
    const int j = T - d.nact + a;  // local bit
    // in the last stage's layout: in-thread bit, or bit of the thread index
    int cb = -1, tbit = -1;
    const int lo = T - E * d.nst;
    if (lo >= 0) {
      if (j >= lo + E)
        tbit = j - E;
      else if (j >= lo)
        cb = j - lo;
      else
        tbit = j;
    } else {
      const int r = E + lo;
      if (j < r)
        cb = j;
      else if (j >= T + lo)
        cb = j - (T + lo) + r;
      else
        tbit = j - r;
    }
    const double U = cb == 0 ? U0 : cb == 1 ? U1 : cb == 2 ? U2 : ((tid >> tbit) & 1) ? Tacc : 0.0;
    const double v = warp_sum(Tacc - 2.0 * U);
    if ((tid & 31) == 0) red[(tid >> 5) * (FIX_TMAX + 1) + a] = v;
  }
  {
    const double v = warp_sum(gacc);
    if ((tid & 31) == 0) red[(tid >> 5) * (FIX_TMAX + 1) + FIX_TMAX] = v;
  }
  __syncthreads();
  if (tid <= FIX_TMAX) {
    const int slot = tid < FIX_TMAX ? (tid < d.nact ? d.slot[tid] : -1) : (d.has_gslot ? d.gslot : -1);
    if (slot >= 0) {
      double v = 0.0;
      for (int w = 0; w < NW; ++w) v += red[w * (FIX_TMAX + 1) + tid];
      p.partials[(i64)slot * p.G + blockIdx.x] = tid == FIX_TMAX ? v * d.cost_w0 : v;
    }
  }
}

#if QG_FIX_E == 3
// ------------------------------------------------------------ phase tables
//
// One launch per run / grad_run fills the tables of every sweep (one CTA per
// sweep, persistent), so that a sweep's own start-up reads no angle and takes
// no sine: the double sweeps build their tables in every CTA.  Entry (c,
// thread) of a sweep is prod_j exp(-+ i theta_j / 2) over its active bits, in
// the order in which the sweep's threads read it.

__global__ void __launch_bounds__(256) fix_tables_kernel(const __grid_constant__ FixTables f, const double* params,
                                                         char* area) {
  __shared__ Unit one[FIX_TMAX], lo[64], hi[64];
  __shared__ int bad;
  const int tid = threadIdx.x;
  int32_t* flags = (int32_t*)(area + f.flags);
  if (blockIdx.x == 0 && tid <= f.n) {
    // start amplitudes: Ry(pi/4)^n |0> by popcount, or the uniform state
    double s8, c8;
    sincospi(0.125, &s8, &c8);
    double q = 1.0;
    for (int i = 0; i < f.n - tid; ++i) q *= c8;
    for (int i = 0; i < tid; ++i) q *= s8;
    ((double*)(area + f.startp))[tid] = f.kind == 0 ? q : exp2(-0.5 * f.n);
  }
  for (int sweep = blockIdx.x; sweep < f.nsweeps; sweep += gridDim.x) {
    const int layer = sweep / f.per_layer, s = sweep % f.per_layer;
    const int T = f.t[s], k = f.nact[s];
    if (tid == 0) bad = 0;
    __syncthreads();
    bool mybad = false;
    if (tid < k) {
      const int q = f.n - 1 - (f.lo[s] + tid);
      const double th = layer < f.ini_layers ? 0.78539816339744830962
                        : f.kind == 0        ? params[(int64_t)(layer - f.ini_layers) * f.n + q]
                                             : params[2 * layer];
      one[tid] = unit_angle(0.5 * th, mybad);
    }
    __syncthreads();
    // products over the low six and the high active bits
    if (tid < 128) {
      const int half = tid >> 6, e = tid & 63;
      Unit v{1ll << 62, 0};
      for (int j = 0; j < 6; ++j) {
        const int a = half * 6 + j;
        if (a < k) v = mul62(v, Unit{one[a].c, ((e >> j) & 1) ? one[a].s : -one[a].s});
      }
      (half ? hi : lo)[e] = v;
    }
    __syncthreads();
    const int E = f.e;
    const int nst = fix_stages(k, E), skip = fix_table_skip(T, k, E);
    const int lw = T - E - skip;
    int4* tab = (int4*)(area + f.tab0 + layer * f.layer_bytes + f.off[s]);
    for (int i = tid; i < (1 << (E + lw)); i += 256) {
      const int c = i >> lw, th = (i & ((1 << lw) - 1)) << skip;
      // local index of (th, c) in the last stage's layout
      const int low = T - E * nst, r = E + low;
      int e = low >= 0 ? (c << low) | (th & ((1 << low) - 1)) | ((th >> low) << (low + E))
                       : (c & ((1 << r) - 1)) | ((c >> r) << (T + low)) | (th << r);
      e >>= T - k;
      tab[i] = phase_limbs(mul62(lo[e & 63], hi[e >> 6]), 2);
    }
    if (f.cost == COST_INT && s == 0) {
      // exp(-i gamma w0 m), the angle rounded to double as gamma * C is
      int4* ct = (int4*)(area + f.ctab0 + layer * f.ctab_bytes);
      const double g = params[2 * layer + 1] * f.cost_w0;
      for (int m = tid; m <= f.cost_maxabs; m += 256) {
        Unit u = unit_angle(g * (double)m, mybad);
        ct[f.cost_maxabs - m] = phase_limbs(u, 0);
        u.s = -u.s;
        ct[f.cost_maxabs + m] = phase_limbs(u, 0);
      }
    }
    if (mybad) bad = 1;
    __syncthreads();
    if (tid == 0) flags[sweep] = bad;
  }
}
#endif

template <int T>
size_t fix_smem(bool bwd) {
  return ((size_t)16 << T) * (bwd ? 2 : 1);
}

template <typename F>
cudaError_t with_t(int t, F f) {
  // 4 amplitudes a thread: up to FIX_TMAX2
  if (QG_FIX_E == 2 && t > FIX_TMAX2) return cudaErrorInvalidValue;
  switch (t) {
    case 8:
      return f(std::integral_constant<int, 8>());
    case 9:
      return f(std::integral_constant<int, 9>());
    case 10:
      return f(std::integral_constant<int, 10>());
#if QG_FIX_E == 3
    case 11:
      return f(std::integral_constant<int, 11>());
    case 12:
      return f(std::integral_constant<int, 12>());
#endif
  }
  return cudaErrorInvalidValue;
}

// raise the shared-memory limits once per device
cudaError_t prepare_fix_kernels() {
  constexpr int kMaxDev = 64;
  static std::atomic<int> ready[kMaxDev];
  static std::mutex mu;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDev) return cudaErrorInvalidDevice;
  if (ready[dev].load(std::memory_order_acquire)) return cudaSuccess;
  std::lock_guard<std::mutex> lock(mu);
  for (int t = FIX_TMIN; t <= (QG_FIX_E == 3 ? FIX_TMAX : FIX_TMAX2); ++t) {
    e = with_t(t, [](auto tc) {
      constexpr int T = decltype(tc)::value;
      const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
      cudaError_t r = cudaFuncSetAttribute(fix_fwd_kernel<T>, a, (int)fix_smem<T>(false));
      if (r == cudaSuccess) r = cudaFuncSetAttribute(fix_bwd_kernel<T, false, false>, a, (int)fix_smem<T>(true));
      if (r == cudaSuccess) r = cudaFuncSetAttribute(fix_bwd_kernel<T, true, false>, a, (int)fix_smem<T>(true));
      if (r == cudaSuccess) r = cudaFuncSetAttribute(fix_bwd_kernel<T, false, true>, a, (int)fix_smem<T>(true));
      return r;
    });
    if (e != cudaSuccess) return e;
  }
  ready[dev].store(1, std::memory_order_release);
  return cudaSuccess;
}

template <typename D, typename P>
cudaError_t launch_nt(void (*kern)(D, P), int grid, int nt, size_t smem, cudaStream_t st, bool pdl, const D& d,
                      const P& p) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)nt);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, d, p);
}

}  // namespace

#define FIXFN2(f, e) f##_e##e
#define FIXFN1(f, e) FIXFN2(f, e)
#define FIXFN(f) FIXFN1(f, QG_FIX_E)

int FIXFN(fix_ctas_per_sm)(int t, bool bwd, bool uncompute) {
  int blocks = 0;
  if (prepare_fix_kernels() != cudaSuccess) {
    cudaGetLastError();
    return 1;
  }
  const cudaError_t e = with_t(t, [&](auto tc) {
    constexpr int T = decltype(tc)::value;
    const void* fn = !bwd        ? (const void*)fix_fwd_kernel<T>
                     : uncompute ? (const void*)fix_bwd_kernel<T, true, false>
                                 : (const void*)fix_bwd_kernel<T, false, false>;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, fn, Lay<T>::NT, fix_smem<T>(bwd));
  });
  if (e != cudaSuccess) {
    cudaGetLastError();
    return 1;
  }
  return blocks > 0 ? blocks : 1;
}

cudaError_t FIXFN(launch_fix_fwd)(const FixDesc& d, const FixPtrs& p, int grid, cudaStream_t st, bool pdl) {
  if (cudaError_t e = prepare_fix_kernels()) return e;
  return with_t(d.t, [&](auto tc) {
    constexpr int T = decltype(tc)::value;
    return launch_nt(fix_fwd_kernel<T>, grid, Lay<T>::NT, fix_smem<T>(false), st, pdl, d, p);
  });
}

cudaError_t FIXFN(launch_fix_bwd)(const FixDesc& d, const FixPtrs& p, bool uncompute, bool chained, int grid,
                                  cudaStream_t st, bool pdl) {
  if (cudaError_t e = prepare_fix_kernels()) return e;
  return with_t(d.t, [&](auto tc) {
    constexpr int T = decltype(tc)::value;
    return launch_nt(uncompute ? fix_bwd_kernel<T, true, false>
                     : chained ? fix_bwd_kernel<T, false, true>
                               : fix_bwd_kernel<T, false, false>,
                     grid, Lay<T>::NT, fix_smem<T>(true), st, pdl, d, p);
  });
}

#if QG_FIX_E == 3
cudaError_t launch_fix_tables(const FixTables& f, const double* params, char* area, cudaStream_t st) {
  const int grid = f.nsweeps < 1 ? 1 : f.nsweeps < 1024 ? f.nsweeps : 1024;
  fix_tables_kernel<<<grid, 256, 0, st>>>(f, params, area);
  return cudaGetLastError();
}

// 8 or 4 amplitudes a thread (qg_fixed2.cu)
int fix_ctas_per_sm_e2(int t, bool bwd, bool uncompute);
cudaError_t launch_fix_fwd_e2(const FixDesc& d, const FixPtrs& p, int grid, cudaStream_t st, bool pdl);
cudaError_t launch_fix_bwd_e2(const FixDesc& d, const FixPtrs& p, bool uncompute, bool chained, int grid,
                              cudaStream_t st, bool pdl);

int fix_ctas_per_sm(const FixDesc& d, bool bwd, bool uncompute) {
  return (d.e == 2 ? fix_ctas_per_sm_e2 : fix_ctas_per_sm_e3)(d.t, bwd, uncompute);
}
cudaError_t launch_fix_fwd(const FixDesc& d, const FixPtrs& p, int grid, cudaStream_t st, bool pdl) {
  return (d.e == 2 ? launch_fix_fwd_e2 : launch_fix_fwd_e3)(d, p, grid, st, pdl);
}
cudaError_t launch_fix_bwd(const FixDesc& d, const FixPtrs& p, bool uncompute, bool chained, int grid,
                           cudaStream_t st, bool pdl) {
  return (d.e == 2 ? launch_fix_bwd_e2 : launch_fix_bwd_e3)(d, p, uncompute, chained, grid, st, pdl);
}
#endif

}  // namespace qg
