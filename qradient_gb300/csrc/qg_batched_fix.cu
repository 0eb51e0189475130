// Batched persistent kernel in complex128, in 64-bit fixed point.
//
// Why.  The double form of this kernel (qg_batched.cu) kept the FP64 pipe
// 82% busy: 2 double instructions per amplitude and rotation forward, 6
// backward, 16 cycles of the pipe each per warp.  Here a layer of rotations
// is V D V^-1 as in the fixed-point sweeps (qg_fixed.cu): additions, one
// phase product, additions; and all gradient sums of a layer come from one
// product per amplitude.  Psi and lambda stay with their threads, eight
// amplitudes of each, for the whole circuit: in registers, of which the
// compiler spills 1.4-1.5 KB a thread (480-byte frame) at the cap of 128.
// Shared memory only carries the exchanges between layouts, the
// CNOT ladder's gather and (across a cluster) the split bits.
//
// Number format.  Rotations keep ||psi|| = 1 and ||lambda||, so one power of
// two per state scales it to int64 from start to end: no conversion per
// layer.  h counts half bits of the norm above 2^60; a
// butterfly level adds one, the phase product (phases at 2^62) takes four,
// shifts keep h <= 5 and bring it back to at least 1 before a phase product.
//
// Measured (GB300, L = 30, circuits/s, double form -> this, batches of 4096 to
// 1024 jobs): n = 10 114k -> 476k, n = 11 74k -> 269k, n = 12 41k -> 131k,
// n = 13 (2 CTAs) 18.4k -> 48.5k, n = 14 (4 CTAs) 7.8k -> 18.3k; one n = 12 job
// alone 3.57 -> 1.14 ms.  What bounds it now is instruction issue (45% active
// at the one CTA of 16 warps that 184 KB of shared memory leave room for).
#include <cooperative_groups.h>
#include <stdint.h>

#include "qg_batched.h"
#include "qg_fixed_math.cuh"

namespace cg = cooperative_groups;

namespace qg {

namespace {

constexpr int BF_UNITS = 512;    // angles of a run of layers, as unit complex numbers
constexpr int BF_CTAB = 1024;    // QAOA cost phases (|m| <= 511)
constexpr int LIM = 5;

template <int T>
struct BfSmem {
  static constexpr int NT = 1 << (T - E);
  static constexpr size_t XL = (size_t)16 << T;                 // after XP
  static constexpr size_t R = XL + ((size_t)16 << T);           // int64 sums [4][NT]
  static constexpr size_t F = R + (size_t)4 * NT * 8;           // and their 2^-28 fractions, uint32 [4][NT]
  static constexpr size_t U = F + (size_t)4 * NT * 4;           // Unit [BF_UNITS]
  static constexpr size_t CT = U + (size_t)BF_UNITS * 16;       // int4 [BF_CTAB]
  static constexpr size_t CM = CT + (size_t)BF_CTAB * 16;       // int16 costs [in-thread index][thread]
  static constexpr size_t total = CM + ((size_t)2 << T);
};

struct BfShared {
  int job, bad;
  BatchJob J;
  Unit lo[32], mid[16], dd[NA];  // phase factors of the layer: thread bits 0-4, 5.., in-thread (and split) bits
  double startP[32];             // start amplitudes by popcount
  double red[16];
  double bsum[16];
  double norm2;                  // |lambda|^2 of this block
};

// x 2^e for |e| up to 2000
__device__ __forceinline__ double pow2d(int e) { return __hiloint2double((e + 1023) << 20, 0); }
__device__ __forceinline__ double scale2(double x, int e) { return x * pow2d(e >> 1) * pow2d(e - (e >> 1)); }

__device__ __noinline__ Unit unit_call(double a, int* bad) {
  bool b = false;
  const Unit u = unit_angle(a, b);
  if (b) *bad = 1;
  return u;
}

// one stage's in-thread bits: masks of X and Y by local bit -> two-bit codes
template <int T>
__device__ __forceinline__ int stage_code(int s, unsigned mx, unsigned my) {
  int code = 0;
#pragma unroll
  for (int i = 0; i < E; ++i) {
    const int lo = T - E * (s + 1);
    const int j = lo >= 0 ? lo + i : i;
    if (lo >= 0 || i < E + lo) code |= (int)(((mx >> j) & 1) | (((my >> j) & 1) << 1)) << (2 * i);
  }
  return code;
}

__device__ __forceinline__ int levels_of(int code) { return __popc(code); }

__device__ __forceinline__ void shift_left(i64* re, i64* im, int s) {
#pragma unroll
  for (int c = 0; c < NA; ++c) {
    re[c] = re[c] << s;
    im[c] = im[c] << s;
  }
}

template <int T, int S>
__device__ __forceinline__ void put(unsigned char* ex, const i64* re, const i64* im) {
  const int a = Lay<T>::sw(Lay<T>::ebase(S, threadIdx.x)) * 16;
#pragma unroll
  for (int c = 0; c < NA; ++c) {
    const int o = Lay<T>::sw(Lay<T>::eoff(S, c)) * 16;
    *(longlong2*)(ex + (a ^ (o & 112)) + (o & ~112)) = make_longlong2(re[c], im[c]);
  }
}
template <int T, int S>
__device__ __forceinline__ void get(const unsigned char* ex, i64* re, i64* im) {
  const int a = Lay<T>::sw(Lay<T>::ebase(S, threadIdx.x)) * 16;
#pragma unroll
  for (int c = 0; c < NA; ++c) {
    const int o = Lay<T>::sw(Lay<T>::eoff(S, c)) * 16;
    const longlong2 v = *(const longlong2*)(ex + (a ^ (o & 112)) + (o & ~112));
    re[c] = v.x;
    im[c] = v.y;
  }
}
// the same with the stage known at run time
template <int T, bool PUT>
__device__ __forceinline__ void move_at(unsigned char* ex, i64* re, i64* im, int s) {
  if (s == 0)
    PUT ? put<T, 0>(ex, re, im) : get<T, 0>(ex, re, im);
  else if (s == 1)
    PUT ? put<T, 1>(ex, re, im) : get<T, 1>(ex, re, im);
  else if (Lay<T>::NS == 3 || s == 2)
    PUT ? put<T, 2>(ex, re, im) : get<T, 2>(ex, re, im);
  else
    PUT ? put<T, Lay<T>::NS - 1>(ex, re, im) : get<T, Lay<T>::NS - 1>(ex, re, im);
}

}  // namespace

// Cluster size 2^lg (lg > 0 only with CL).  A job's block has m = n - lg
// local bits; jobs with m < T run padded (the higher local bits stay zero).
template <int T, bool CL>
__global__ void __launch_bounds__(BfSmem<T>::NT, 512 / BfSmem<T>::NT) batched_fix_kernel(const BatchJob* __restrict__ jobs, int njobs,
                                                                      int* counter, int mmax, int lg) {
  constexpr int NT = BfSmem<T>::NT, NW = NT / 32, NS = Lay<T>::NS, LAST = NS - 1;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ BfShared S;
  unsigned char* XP = smem;
  unsigned char* XL = smem + BfSmem<T>::XL;
  i64* R = (i64*)(smem + BfSmem<T>::R);
  uint32_t* F = (uint32_t*)(smem + BfSmem<T>::F);
  Unit* U = (Unit*)(smem + BfSmem<T>::U);
  int4* ctab = (int4*)(smem + BfSmem<T>::CT);
  int16_t* cm = (int16_t*)(smem + BfSmem<T>::CM) + threadIdx.x;  // this thread's, stride NT
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = CL ? (int)cluster.block_rank() : 0;
  auto csync = [&]() {
    if (CL)
      cluster.sync();
    else
      __syncthreads();
  };

  // the first job number is written into the other CTAs' shared memory, which
  // may be touched only once they have started
  if (CL) cluster.sync();
  for (;;) {
    if (tid == 0 && rank == 0) {
      const int j = atomicAdd(counter, 1);
      S.job = j;
      if (CL)
        for (int r = 1; r < (1 << lg); ++r) *cluster.map_shared_rank(&S.job, r) = j;
    }
    if (tid == 0) S.bad = 0;
    csync();
    const int jid = S.job;
    if (jid >= njobs) break;
    if (tid < (int)(sizeof(BatchJob) / 4)) ((int*)&S.J)[tid] = ((const int*)(jobs + jid))[tid];
    __syncthreads();
    const BatchJob& J = S.J;
    const int n = J.n, m = n - (CL ? lg : 0), L = J.layers;
    const bool grad = J.grad != nullptr;
    const int np = J.kind == 0 ? L * n : 2 * L;
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    if (m < (CL ? 2 : 1) || m > mmax || L < 0) {
      // a job this launch cannot hold: NaN outputs, no state touched
      if (tid == 0 && rank == 0) {
        if (J.expec) *J.expec = nan;
        if (J.grad && L >= 0)
          for (int i = 0; i < np; ++i) J.grad[i] = nan;
      }
      csync();
      continue;
    }
    if (tid == 0 && rank == 0 && CL) {
      // the CTAs of a cluster add their parts
      if (J.expec) *J.expec = 0.0;
      if (grad)
        for (int i = 0; i < np; ++i) J.grad[i] = 0.0;
      if (J.term_expec)
        for (int k = 0; k < J.nterms; ++k) J.term_expec[k] = 0.0;
    }
    const int M = 1 << m;
    int hflip = 0, lrank = rank;  // see qg_batched.cu: the ladder's CNOT(0, 1) relabels 4-CTA blocks
    auto hmap = [](int t) { return t ^ ((t >> 1) & 1); };
    auto relabel = [&]() {
      if (CL && lg == 2) {
        hflip ^= 1;
        lrank = hmap(lrank);
      }
    };
    auto peer = [&](unsigned char* v, int block) -> const unsigned char* {
      return CL ? (const unsigned char*)cluster.map_shared_rank(v, lg == 2 && hflip ? hmap(block) : block) : v;
    };
    // this thread's elements in stage 0's layout: e(c) = tid | c << (T - 3);
    // those at M and above are padding
    auto elem = [&](int c) { return tid | (c << (T - E)); };
    auto global_of = [&](int e) { return ((uint32_t)lrank << m) | (uint32_t)(e & (M - 1)); };

    i64 pr[NA], pi[NA], lr[NA], li[NA];
    int h = 0;    // half bits of the norm above 2^60
    int sp = 60;  // psi = X 2^-sp, lambda = X 2^(pl - sp)
    int pl = 0;

    // ---- start state: Ry(pi/4)^n |0..0> or |+..+>
    if (tid <= n) {
      double c8, s8;
      sincospi(0.125, &s8, &c8);
      double q = 1.0;
      for (int i = 0; i < n - tid; ++i) q *= c8;
      for (int i = 0; i < tid; ++i) q *= s8;
      S.startP[tid] = J.kind == 0 ? q : exp2(-0.5 * n);
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < NA; ++c) {
      pr[c] = elem(c) < M ? __double2ll_rn(S.startP[__popc(global_of(elem(c)))] * 0x1p60) : 0;
      pi[c] = lr[c] = li[c] = 0;
    }
    // QAOA: the integer cost of this thread's elements
    if (J.kind == 1) {
#pragma unroll 1
      for (int c = 0; c < NA; ++c) {
        const uint32_t x = global_of(elem(c));
        int v = 0;
        for (int k = 0; k < J.cost_nterms; ++k) {
          const qg_cost_term t = J.cost[k];
          int s = (int)((x >> t.b0) & 1);
          if (t.b1 >= 0) s ^= (int)((x >> t.b1) & 1);
          v += s ? -t.c : t.c;
        }
        cm[c * NT] = (int16_t)v;
      }
    }

    bool swapped = false;  // split bits exchanged with in-thread ones in this layer's frame

    // ---- angles of a run of layers as unit complex numbers in shared memory
    const int per = J.kind == 0 ? n : 1;
    const int run = BF_UNITS / per;  // layers per fill
    int ubase = -1;
    auto need_units = [&](int i, bool down) {  // the same decision in every thread
      if (ubase >= 0 && i >= ubase && i < ubase + run) return;
      ubase = down ? (i - run + 1 > 0 ? i - run + 1 : 0) : i;
      __syncthreads();  // the previous run's readers are done
#pragma unroll 1
      for (int k = tid; k < run * per && ubase + k / per < L; k += NT)
        U[k] = unit_call(0.5 * (J.kind == 0 ? J.params[(int64_t)ubase * n + k] : J.params[2 * (ubase + k)]), &S.bad);
      __syncthreads();
    };
    // Phase factors of layer i, by the first 56 threads; read after two exchanges.
    auto build_phases = [&](int i) {
      constexpr int lo_last = T - E * NS;  // <= 0: low in-thread bits are [0, r), thread bits follow
      constexpr int r = E + lo_last;
      if (tid < 32 + 16 + NA) {
        const Unit* u = U + (i - ubase) * per;
        auto unit = [&](int j, int one) {  // exp(-+ i theta / 2) of local or split bit j
          const Unit v = u[J.kind == 0 ? n - 1 - j : 0];
          return Unit{v.c, one ? v.s : -v.s};
        };
        Unit p{1ll << 62, 0};
        if (tid < 48) {
          const int first = tid < 32 ? 0 : 5, cnt = tid < 32 ? 5 : T - E - 5, e = tid < 32 ? tid : tid - 32;
#pragma unroll 1
          for (int k = 0; k < cnt; ++k) {
            const int j = r + first + k;
            if (j < m) p = mul62(p, unit(j, (e >> k) & 1));
          }
          if (tid < 32)
            S.lo[e] = p;
          else if (e < (1 << (T - E - 5)))
            S.mid[e] = p;
        } else {
          const int c = tid - 48;
#pragma unroll 1
          for (int k = 0; k < E; ++k) {
            const int j = k < r ? k : T - E + k;  // top bits fill a short last stage
            const bool out = CL && swapped && k < lg;
            if (j < m) p = mul62(p, unit(j, ((out ? lrank : c) >> k) & 1));
            if (CL && k < lg) p = mul62(p, unit(m + k, ((out ? c : lrank) >> k) & 1));
          }
          S.dd[c] = p;
        }
      }
    };
    // exp(-i gamma w0 m) of layer i (QAOA), visible after a barrier
    auto build_costs = [&](int i) {
      const double g = J.params[2 * i + 1] * J.cost_w0;
      __syncthreads();
#pragma unroll 1
      for (int k = tid; k <= J.cost_maxabs; k += NT) {
        Unit u = unit_call(g * (double)k, &S.bad);
        ctab[J.cost_maxabs - k] = phase_limbs(u, 0);
        u.s = -u.s;
        ctab[J.cost_maxabs + k] = phase_limbs(u, 0);
      }
      __syncthreads();
    };

    // masks of the layer's X and Y rotations by bit, one axis per lane
    unsigned mx = 0, my = 0;
    auto load_axes = [&](int i) {
      const int q = n - 1 - lane;
      const int ax = J.kind == 1 ? 0 : q >= 0 ? (int)J.axes[i * n + q] : 2;
      mx = __ballot_sync(0xffffffffu, q >= 0 && ax == 0);
      my = __ballot_sync(0xffffffffu, q >= 0 && ax == 1);
    };

    // ---- the CNOT ladder as a gather, (E v)[y] = v[A^-1 y] (inverse: v[A y]);
    // linear, so an element's source slot is the XOR of its parts'
    auto entangle = [&](bool inv, bool both) {
      if (J.entangler == 0) return;
      if (J.entangler == 2) {
#pragma unroll
        for (int c = 0; c < NA; ++c) {
          const uint32_t x = global_of(elem(c));
          if (__popc(x & (x >> 1)) & 1) {
            pr[c] = -pr[c];
            pi[c] = -pi[c];
            if (both) lr[c] = -lr[c], li[c] = -li[c];
          }
        }
        return;
      }
      if (J.entangler == 1) relabel();
      // CNOT(q, q+1): odd q have control bits n-2, n-4, .., even q n-1, n-3, ..
      const uint32_t all = (1u << n) - 2u, alt = n & 1 ? 0xaaaaaaaau : 0x55555555u;
      const uint32_t odd = all & alt, even = all & ~alt;
      const int wrap = J.entangler == 3 ? n - 1 : 31;  // (bit 31 is never set: n <= 15)
      auto image = [&](uint32_t x) {
        if (!inv) x ^= (x & even) >> 1;
        x ^= ((x & odd) >> 1) ^ ((J.entangler == 3 ? x & 1u : 0u) << wrap);
        if (inv) x ^= (x & even) >> 1;
        return x;
      };
      auto local = [&](int e) {  // padding maps to itself
        return (int)(image((uint32_t)(e & (M - 1))) & (uint32_t)(M - 1)) | (e & ~(M - 1));
      };
      const int base = local(tid) ^ (int)(image((uint32_t)lrank << m) & (uint32_t)(M - 1));
      int step[E];
#pragma unroll
      for (int k = 0; k < E; ++k) step[k] = local(1 << (T - E + k));
      put<T, 0>(XP, pr, pi);
      if (both) put<T, 0>(XL, lr, li);
      __syncthreads();
#pragma unroll
      for (int c = 0; c < NA; ++c) {
        int e = base;
#pragma unroll
        for (int k = 0; k < E; ++k)
          if ((c >> k) & 1) e ^= step[k];
        // padding elements keep their (zero) value: the block's own bits must not move them
        if (elem(c) >= M) e = elem(c);
        const int o = Lay<T>::sw(e) * 16;
        const longlong2 v = *(const longlong2*)(XP + o);
        pr[c] = v.x;
        pi[c] = v.y;
        if (both) {
          const longlong2 w = *(const longlong2*)(XL + o);
          lr[c] = w.x;
          li[c] = w.y;
        }
      }
      __syncthreads();  // the next exchange rewrites slots that others read here
    };

    unsigned dither = 0;  // of the step
    // shift so that mm more levels fit
    auto room = [&](int mm, bool both) {
      const int over = h + mm - LIM;
      const int s = over > 0 ? (over + 1) / 2 : 0;
      if (s) {
        shift_right(pr, pi, s, dither);
        if (both) shift_right(lr, li, s, dither);
        h -= 2 * s;
        sp -= s;
      }
      h += mm;
    };
    // Split bits: the last stage's first lg in-thread bits change places with
    // them across the cluster, so that a thread holds all blocks' values of
    // its remaining elements and the rotations become in-thread ones: half
    // (lg = 1) or three quarters of a block travel each way.  (Reading the
    // partners' whole blocks and keeping one's own half of each pair moved
    // two to four times as much and ran n = 14 jobs at 11.3k circuits/s.)
    // In: every CTA puts its block into its own slots, the others read their
    // share.  Out: a thread writes straight into the slots it read -- nobody
    // else reads those -- and every CTA collects its own block.
    auto swap_in = [&](auto lgc, bool both) {
      constexpr int LG = decltype(lgc)::value, CS = 1 << LG;
      put<T, LAST>(XP, pr, pi);
      if (both) put<T, LAST>(XL, lr, li);
      cluster.sync();
      int mine = Lay<T>::sw(Lay<T>::ebase(LAST, tid)) * 16;  // in-thread bits [0, LG) = this block's number
#pragma unroll
      for (int k = 0; k < LG; ++k)
        if ((lrank >> k) & 1) mine ^= Lay<T>::sw(Lay<T>::eoff(LAST, 1 << k)) * 16;
#pragma unroll
      for (int b = 0; b < CS; ++b) {
        const unsigned char* x = peer(XP, b);
        const unsigned char* y = peer(XL, b);
#pragma unroll
        for (int c = 0; c < NA; c += CS) {
          const int at = mine ^ (Lay<T>::sw(Lay<T>::eoff(LAST, c)) * 16);
          const longlong2 v = *(const longlong2*)(x + at);
          pr[c + b] = v.x;
          pi[c + b] = v.y;
          if (both) {
            const longlong2 w = *(const longlong2*)(y + at);
            lr[c + b] = w.x;
            li[c + b] = w.y;
          }
        }
      }
    };
    auto swap_out = [&](auto lgc, bool both) {
      constexpr int LG = decltype(lgc)::value, CS = 1 << LG;
      int mine = Lay<T>::sw(Lay<T>::ebase(LAST, tid)) * 16;
#pragma unroll
      for (int k = 0; k < LG; ++k)
        if ((lrank >> k) & 1) mine ^= Lay<T>::sw(Lay<T>::eoff(LAST, 1 << k)) * 16;
#pragma unroll
      for (int b = 0; b < CS; ++b) {
        unsigned char* x = const_cast<unsigned char*>(peer(XP, b));
        unsigned char* y = const_cast<unsigned char*>(peer(XL, b));
#pragma unroll
        for (int c = 0; c < NA; c += CS) {
          const int at = mine ^ (Lay<T>::sw(Lay<T>::eoff(LAST, c)) * 16);
          *(longlong2*)(x + at) = make_longlong2(pr[c + b], pi[c + b]);
          if (both) *(longlong2*)(y + at) = make_longlong2(lr[c + b], li[c + b]);
        }
      }
      cluster.sync();
      get<T, LAST>(XP, pr, pi);
      if (both) get<T, LAST>(XL, lr, li);
    };
    auto split_code = [&]() {
      int code = 0;
      for (int k = 0; k < lg; ++k) code |= (int)(((mx >> (m + k)) & 1) | ((my >> (m + k)) & 1) << 1) << (2 * k);
      return code;
    };
    auto to_frame = [&](bool both) {
#pragma unroll 1
      for (int s = 0;;) {
        const int code = stage_code<T>(s, mx & (M - 1), my & (M - 1));
        room(levels_of(code), both);
        butterflies<true>(pr, pi, code);
        if (both) butterflies<true>(lr, li, code);
        if (++s == NS) break;
        move_at<T, true>(XP, pr, pi, s - 1);
        if (both) move_at<T, true>(XL, lr, li, s - 1);
        __syncthreads();
        move_at<T, false>(XP, pr, pi, s);
        if (both) move_at<T, false>(XL, lr, li, s);
      }
      if (CL && swapped) {
        const int code = split_code();
        room(levels_of(code), both);
        if (lg == 1)
          swap_in(std::integral_constant<int, 1>(), both);
        else
          swap_in(std::integral_constant<int, 2>(), both);
        butterflies<true>(pr, pi, code);
        if (both) butterflies<true>(lr, li, code);
      }
    };
    auto from_frame = [&](bool both, auto after_first) {
      if (CL && swapped) {
        const int code = split_code();
        room(levels_of(code), both);
        butterflies<false>(pr, pi, code);
        if (both) butterflies<false>(lr, li, code);
        if (lg == 1)
          swap_out(std::integral_constant<int, 1>(), both);
        else
          swap_out(std::integral_constant<int, 2>(), both);
      }
#pragma unroll 1
      for (int s = NS - 1;;) {
        const int code = stage_code<T>(s, mx & (M - 1), my & (M - 1));
        room(levels_of(code), both);
        butterflies<false>(pr, pi, code);
        if (both) butterflies<false>(lr, li, code);
        if (--s < 0) break;
        move_at<T, true>(XP, pr, pi, s + 1);
        if (both) move_at<T, true>(XL, lr, li, s + 1);
        __syncthreads();
        if (s == NS - 2) after_first();
        move_at<T, false>(XP, pr, pi, s);
        if (both) move_at<T, false>(XL, lr, li, s);
      }
    };
    // keep at least one half bit after the phase product's four
    auto lift = [&](bool both) {
      const int s = h < LIM - 1 ? (LIM - h) / 2 : 0;
      if (s) {
        shift_left(pr, pi, s);
        if (both) shift_left(lr, li, s);
        h += 2 * s;
        sp += s;
      }
    };
    // this thread's phase of in-thread index c, at 2^62
    Unit pt;
    auto phase_of = [&](int c) {
      Unit d = pt;
      cmul_fix<false>(d.c, d.s, phase_limbs(S.dd[c], 0));
      return phase_limbs(Unit{d.c << 2, d.s << 2}, 0);
    };
    const bool live = Lay<T>::ebase(LAST, tid) < M;  // padding threads of the last stage have nothing to multiply
    auto load_pt = [&]() { pt = mul62(S.lo[tid & 31], S.mid[tid >> 5]); };
          // block sum in a fixed order; a cluster's CTAs add theirs
          auto emit = [&](double val, double* out, double factor) {
    #pragma unroll
            for (int o = 16; o > 0; o >>= 1) val += __shfl_down_sync(0xffffffffu, val, o);
            if (lane == 0) S.red[warp] = val;
            __syncthreads();
            if (tid == 0) {
              double tot = 0.0;
              for (int w = 0; w < NW; ++w) tot += S.red[w];
              tot *= factor;
              if (S.bad) tot = nan;
              if (CL)
                atomicAdd(out, tot);
              else
                *out = tot;
            }
            __syncthreads();
          };
    // ---- observable: lam = O psi and E = Re<psi|lam>, in double; psi in
    // stage 0's slots of XP for the X / Y terms' partners
    auto observe = [&]() {
      double2* P = (double2*)XP;
      __syncthreads();
      const double k = pow2d(-sp);
      double2 v[NA];
#pragma unroll
      for (int c = 0; c < NA; ++c) {
        v[c] = make_double2((double)pr[c] * k, (double)pi[c] * k);
        P[Lay<T>::sw(elem(c))] = v[c];
      }
      csync();
      const bool costonly = J.kind == 1 && grad;
      double2 l[NA];
#pragma unroll
      for (int c = 0; c < NA; ++c) l[c] = make_double2(0.0, 0.0);
      auto partner = [&](uint32_t x) -> double2 {
        const int slot = Lay<T>::sw((int)(x & (uint32_t)(M - 1)));
        if (CL && (int)(x >> m) != lrank) return ((const double2*)peer(XP, (int)(x >> m)))[slot];
        return P[slot];
      };
      if (costonly) {
#pragma unroll
        for (int c = 0; c < NA; ++c) {
          const double d = J.cost_w0 * (double)cm[c * NT];
          l[c] = make_double2(d * v[c].x, d * v[c].y);
        }
      } else {
        // runs of equal weights: signs counted in integers, one multiply per run
        int cnt[NA];
        double dv[NA];
#pragma unroll
        for (int c = 0; c < NA; ++c) cnt[c] = 0, dv[c] = 0.0;
        double rw = 0.0;
        auto flush = [&]() {
#pragma unroll
          for (int c = 0; c < NA; ++c) {
            dv[c] = fma(rw, (double)cnt[c], dv[c]);
            cnt[c] = 0;
          }
        };
        for (int t = 0; t < J.nterms; ++t) {
          const BatchTerm tm = J.terms[t];
          const uint32_t b0 = 1u << (n - 1 - tm.q0);
          if (tm.kind >= 2) {
            if (tm.w != rw) {
              flush();
              rw = tm.w;
            }
            const uint32_t mask = b0 | (tm.kind == 3 ? 1u << (n - 1 - tm.q1) : 0u);
#pragma unroll
            for (int c = 0; c < NA; ++c) cnt[c] += 1 - 2 * (__popc(global_of(elem(c)) & mask) & 1);
          } else {
#pragma unroll
            for (int c = 0; c < NA; ++c) {
              const uint32_t x = global_of(elem(c));
              const double2 u = elem(c) < M ? partner(x ^ b0) : make_double2(0.0, 0.0);
              if (tm.kind == 0) {
                l[c].x = fma(tm.w, u.x, l[c].x);
                l[c].y = fma(tm.w, u.y, l[c].y);
              } else {
                const double sg = (x & b0) ? tm.w : -tm.w;
                l[c].x = fma(-sg, u.y, l[c].x);
                l[c].y = fma(sg, u.x, l[c].y);
              }
            }
          }
        }
        flush();
#pragma unroll
        for (int c = 0; c < NA; ++c) {
          l[c].x = fma(dv[c], v[c].x, l[c].x);
          l[c].y = fma(dv[c], v[c].y, l[c].y);
        }
      }
      double e = 0.0;
#pragma unroll
      for (int c = 0; c < NA; ++c)
        if (elem(c) < M) e = fma(v[c].x, l[c].x, fma(v[c].y, l[c].y, e));
      emit(e, J.expec, 1.0);
      if (J.term_expec) {
        // <P_k> of every term (observable.py:82-177, base.py:22-46)
        for (int t = 0; t < J.nterms; ++t) {
          const BatchTerm tm = J.terms[t];
          const uint32_t b0 = 1u << (n - 1 - tm.q0);
          const uint32_t mask = b0 | (tm.kind == 3 ? 1u << (n - 1 - tm.q1) : 0u);
          double acc = 0.0;
#pragma unroll
          for (int c = 0; c < NA; ++c) {
            if (elem(c) >= M) continue;
            const uint32_t x = global_of(elem(c));
            if (tm.kind >= 2) {
              const double p2 = fma(v[c].x, v[c].x, v[c].y * v[c].y);
              acc += (__popc(x & mask) & 1) ? -p2 : p2;
            } else {
              const double2 u = partner(x ^ b0);
              if (tm.kind == 0)
                acc += fma(v[c].x, u.x, v[c].y * u.y);
              else
                acc += ((x & b0) ? 1.0 : -1.0) * fma(-v[c].x, u.y, v[c].y * u.x);
            }
          }
          emit(acc, J.term_expec + t, 1.0);
        }
      }
      csync();  // every partner has been read

      if (grad) {
        // lambda to fixed point at psi's h: ||lambda|| < 2^pl.  (The largest
        // component first, so that the squares stay representable.)
        double big = 0.0;
#pragma unroll
        for (int c = 0; c < NA; ++c)
          if (elem(c) < M) big = fmax(big, fmax(fabs(l[c].x), fabs(l[c].y)));
        auto block_max = [&](double x) {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) x = fmax(x, __shfl_xor_sync(0xffffffffu, x, o));
          if (lane == 0) S.red[warp] = x;
          __syncthreads();
          x = 0.0;
          for (int w = 0; w < NW; ++w) x = fmax(x, S.red[w]);
          __syncthreads();
          return x;
        };
        auto over_cluster = [&](double x, auto op) {  // the same value in every CTA
          if (!CL) return x;
          if (tid == 0) S.norm2 = x;
          cluster.sync();
          x = S.norm2;
          double r = *cluster.map_shared_rank(&S.norm2, 0);
          for (int k = 1; k < (1 << lg); ++k) r = op(r, *cluster.map_shared_rank(&S.norm2, k));
          cluster.sync();
          return r;
        };
        big = over_cluster(block_max(big), [](double a, double b) { return fmax(a, b); });
        const int e0 = big > 0.0 && isfinite(big) ? ilogb(big) : 0;
        double q = 0.0;
#pragma unroll
        for (int c = 0; c < NA; ++c)
          if (elem(c) < M) {
            const double x = scale2(l[c].x, -e0), y = scale2(l[c].y, -e0);
            q = fma(x, x, fma(y, y, q));
          }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
        if (lane == 0) S.red[warp] = q;
        __syncthreads();
        q = 0.0;
        for (int w = 0; w < NW; ++w) q += S.red[w];
        __syncthreads();
        q = over_cluster(q, [](double a, double b) { return a + b; });
        // lambda with a NaN or an infinity (a non-finite weight, or finite ones
        // whose sum overflows): fixed point has none to carry on, so the job's
        // gradient is set to NaN (`big` drops NaN, the squares keep them)
        if (tid == 0 && !isfinite(q)) S.bad = 1;
        pl = e0 + (q > 0.0 && isfinite(q) ? (ilogb(q) + 2) >> 1 : 0);  // norm^2 < 2^(ilogb + 1)
#pragma unroll
        for (int c = 0; c < NA; ++c) {
          lr[c] = __double2ll_rn(scale2(l[c].x, sp - pl));
          li[c] = __double2ll_rn(scale2(l[c].y, sp - pl));
        }
      }
    };

    // ---- the layers forward, the observable, the layers backward: one loop,
    // so that there is one copy of the code
#pragma unroll 1
    for (int step = 0; step <= (grad ? 2 * L : L); ++step) {
      const bool back = step > L, mid = step == L;
      const int i = back ? 2 * L - step : step;
      dither = dither_bit(rank, step);
      if (!mid) {
        need_units(i, back);
        load_axes(i);
        swapped = CL && ((mx | my) >> m) != 0;
      }
      // what lies before this layer's rotations: the entangler (or, after
      // them, the previous layer's), or the QAOA cost phase
      if (J.kind == 0) {
        const bool here = J.placement == 0 ? (back ? i < L - 1 : !mid) : (back || step > 0);
        if (here) entangle(back, back);
      } else if (back ? i < L - 1 : !mid) {
        build_costs(back ? i + 1 : i);
        lift(back);
#pragma unroll
        for (int c = 0; c < NA; ++c) {
          int4 d = ctab[cm[c * NT] + J.cost_maxabs];
          if (back) d.z = -d.z, d.w = -d.w;
          cmul_fix<false>(pr[c], pi[c], d);
          if (back) cmul_fix<false>(lr[c], li[c], d);
        }
        h -= 4;
        sp -= 2;
      }
      if (mid) {
        observe();
        continue;
      }
      build_phases(i);
      const int levels = __popc(mx | my);
      to_frame(back);
      int wexp = 0;
      if (back) {
        // w = Im(conj(lam) psi): its sum over the thread's amplitudes, and over
        // those with each in-thread bit set (as in qg_fixed.cu)
        i64 sT = 0, s0 = 0, s1 = 0, s2 = 0;
        uint32_t fT = 0, f0 = 0, f1 = 0, f2 = 0;
        if (live) {
#pragma unroll
          for (int c = 0; c < NA; c += 2) {
            i64 V[2];
            uint32_t f[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              const Limbs ar = limbs(lr[c + k]), ai = limbs(li[c + k]), qr = limbs(-pr[c + k]), qi = limbs(pi[c + k]);
              // (a job keeps one scale, and gradients fall with 2^(-n/2): the low
              // x low products count here)
              const i64 ll = mad_wide(ai.l, qr.l, 0) >> 32;
              const i64 l2 = mad_wide(ar.l, qi.l, 0) >> 32;
              const i64 mm = mad_wide(ai.l, qr.h, mad_wide(ai.h, qr.l, mad_wide(ar.l, qi.h, mad_wide(ar.h, qi.l, ll + l2))));
              V[k] = mad_wide(ai.h, qr.h, mad_wide(ar.h, qi.h, mm >> 32));
              f[k] = (uint32_t)mm >> 4;
            }
            s0 += V[1];
            f0 += f[1];
            const i64 w = V[0] + V[1];
            const uint32_t g = f[0] + f[1];
            sT += w;
            fT += g;
            if (c & 2) s1 += w, f1 += g;
            if (c & 4) s2 += w, f2 += g;
          }
        }
        R[tid] = sT, F[tid] = fT;
        R[NT + tid] = s0, F[NT + tid] = f0;
        R[2 * NT + tid] = s1, F[2 * NT + tid] = f1;
        R[3 * NT + tid] = s2, F[3 * NT + tid] = f2;
        // w = V 2^64 / (2^sl 2^sp 2^levels), with the frame's scales
        wexp = 64 - sp - (sp - pl) - levels;
      }
      // the layer's sums, once they are visible: one bit per warp
      auto sums = [&]() {
        constexpr int r = E + (T - E * NS);
        const int nb = m + (CL ? lg : 0);
        for (int j = warp; j < nb; j += NW) {
          // in-thread bit (a split bit is one when swapped), bit of the block's
          // number (a swapped-out local bit, a split bit otherwise), or thread bit
          int cb = j >= m ? (swapped ? j - m : -1) : j < r ? j : j >= T - E + r ? j - (T - E) : -1;
          int rb = j >= m && !swapped ? j - m : -1;
          if (CL && swapped && j < m && cb >= 0 && cb < lg) rb = cb, cb = -1;
          const int tb = j - r;
          i64 acc = 0, frac = 0;  // exact sums
          for (int t = lane; t < NT; t += 32) {
            i64 v = R[t], f = (i64)F[t];
            if (cb >= 0) {
              v -= 2 * R[(cb + 1) * NT + t];
              f -= 2 * (i64)F[(cb + 1) * NT + t];
            } else if (rb < 0 && ((t >> tb) & 1)) {
              v = -v;
              f = -f;
            }
            acc += v;
            frac += f;
          }
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            acc += __shfl_down_sync(0xffffffffu, acc, o);
            frac += __shfl_down_sync(0xffffffffu, frac, o);
          }
          if (lane == 0) {
            double g = scale2(fma((double)frac, 0x1p-28, (double)acc), wexp);
            if (rb >= 0 && ((lrank >> rb) & 1)) g = -g;
            if (S.bad) g = nan;
            if (J.kind == 1)
              S.bsum[j] = g;
            else if (CL)
              atomicAdd(&J.grad[i * n + n - 1 - j], g);
            else
              J.grad[i * n + n - 1 - j] = g;
          }
        }
      };
      lift(back);
      if (live) {
        load_pt();
#pragma unroll
        for (int c = 0; c < NA; ++c) {
          int4 d = phase_of(c);
          if (back) d.z = -d.z, d.w = -d.w;
          cmul_fix<false>(pr[c], pi[c], d);
          if (back) cmul_fix<false>(lr[c], li[c], d);
        }
      }
      h -= 4;
      sp -= 2;
      from_frame(back, [&]() {
        if (back) sums();
      });
      sp += levels;  // V V^-1 = 2 per rotation
      if (back && J.kind == 1) {
        // gamma before the cost phase (qaoa.py:65-68), and beta's sum over the qubits
        const double a = pow2d(-sp);
        double g = 0.0;
#pragma unroll
        for (int c = 0; c < NA; ++c) {
          const double w = fma((double)lr[c] * a, (double)pi[c] * a, -((double)li[c] * a) * ((double)pr[c] * a));
          g = fma((double)cm[c * NT], w, g);
        }
        if (tid == 0) {
          double b = 0.0;
          for (int j = 0; j < n; ++j) b += S.bsum[j];
          if (CL)
            atomicAdd(&J.grad[2 * i], b);
          else
            J.grad[2 * i] = b;
        }
        emit(scale2(g, pl), J.grad + 2 * i + 1, 2.0 * J.cost_w0);
      }
    }
    csync();
  }
}

template <int T, bool CL>
static cudaError_t launch_fix_one(const BatchJob* jobs, int njobs, int* counter, int mmax, int lg, cudaStream_t st,
                                  int* grid_out) {
  constexpr int NT = BfSmem<T>::NT;
  const size_t smem = BfSmem<T>::total;
  auto kern = batched_fix_kernel<T, CL>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, NT, smem);
  if (e != cudaSuccess) return e;
  if (per < 1) return cudaErrorInvalidConfiguration;
  const int cs = 1 << lg;
  int units = sms * per / cs;
  if (units > njobs) units = njobs;
  if (units < 1) units = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(units * cs);
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (CL) {
    // clusters co-resident at once (a cluster's CTAs share one GPC)
    int nc = 0;
    if (cudaOccupancyMaxActiveClusters(&nc, kern, &cfg) == cudaSuccess && nc > 0 && nc < units) {
      units = nc;
      cfg.gridDim = dim3(units * cs);
    }
    cudaGetLastError();
  }
  *grid_out = units;
  e = cudaLaunchKernelEx(&cfg, kern, jobs, njobs, counter, mmax, lg);
  if (e != cudaSuccess) return e;
  return cudaGetLastError();
}

cudaError_t launch_batched_fix(int cluster, const BatchJob* jobs, int njobs, int* counter, int mmax, cudaStream_t st,
                               int* grid_out) {
  const int lg = cluster == 4 ? 2 : cluster - 1;
  // the smallest tile that holds the launch's largest block
  switch (mmax <= 9 ? 9 : mmax) {
    case 9:
      return lg ? launch_fix_one<9, true>(jobs, njobs, counter, mmax, lg, st, grid_out)
                : launch_fix_one<9, false>(jobs, njobs, counter, mmax, lg, st, grid_out);
    case 10:
      return lg ? launch_fix_one<10, true>(jobs, njobs, counter, mmax, lg, st, grid_out)
                : launch_fix_one<10, false>(jobs, njobs, counter, mmax, lg, st, grid_out);
    case 11:
      return lg ? launch_fix_one<11, true>(jobs, njobs, counter, mmax, lg, st, grid_out)
                : launch_fix_one<11, false>(jobs, njobs, counter, mmax, lg, st, grid_out);
    case 12:
      return lg ? launch_fix_one<12, true>(jobs, njobs, counter, mmax, lg, st, grid_out)
                : launch_fix_one<12, false>(jobs, njobs, counter, mmax, lg, st, grid_out);
  }
  return cudaErrorInvalidValue;
}

}  // namespace qg
