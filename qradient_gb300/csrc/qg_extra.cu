// Cost tables and the shot sampler.
#include <stdint.h>

#include "qg_draw.cuh"
#include "qg_extra.h"
#include "qg_philox.cuh"

namespace qg {

// ------------------------------------------------------------ cost tables
//
// Integer diagonal m(x) = sum_k c_k s_k(x) over Z / ZZ terms with integer
// coefficients c_k, s_k(x) = +1 when the term's bits have even parity (z = +1
// for bit 0), state.py:273-292.  For MaxCut every c_k = 1.

__global__ void int_cost_kernel(int n, const __grid_constant__ IntTermList L, int32_t* table) {
  const int64_t N = (int64_t)1 << n;
  for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < N; x += (int64_t)gridDim.x * blockDim.x) {
    int32_t m = 0;
    for (int k = 0; k < L.nterms; ++k) {
      const IntTerm tk = L.t[k];
      int s = (int)((x >> tk.b0) & 1);
      if (tk.b1 >= 0) s ^= (int)((x >> tk.b1) & 1);
      m += s ? -tk.c : tk.c;
    }
    table[x] = m;
  }
}

// Real diagonal C(x) = sum_k w_k s_k(x) for weights without a common integer base.
__global__ void real_cost_kernel(int n, const __grid_constant__ RealTermList L, double* table) {
  const int64_t N = (int64_t)1 << n;
  for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < N; x += (int64_t)gridDim.x * blockDim.x) {
    double c = 0.0;
    for (int k = 0; k < L.nterms; ++k) {
      const RealTerm tk = L.t[k];
      int s = (int)((x >> tk.b0) & 1);
      if (tk.b1 >= 0) s ^= (int)((x >> tk.b1) & 1);
      c += s ? -tk.w : tk.w;
    }
    table[x] = c;
  }
}

cudaError_t launch_int_cost(int n, const IntTermList& terms, int32_t* table, int grid, cudaStream_t st) {
  int_cost_kernel<<<grid, 256, 0, st>>>(n, terms, table);
  return cudaGetLastError();
}

cudaError_t launch_real_cost(int n, const RealTermList& terms, double* table, int grid, cudaStream_t st) {
  real_cost_kernel<<<grid, 256, 0, st>>>(n, terms, table);
  return cudaGetLastError();
}

// ------------------------------------------------------------ sampler
//
// Inverse-CDF sampling of basis states from |psi|^2 (qaoa.py:196-198 draws
// with scipy.stats.rv_discrete).  Chunk sums, one exclusive scan over the
// chunk sums, then one CTA per shot: binary search over the chunks, sums of
// the chunk's segments (one per thread), and a walk inside one segment.  Uniforms come from Philox4x32-10 (Salmon,
// Moraes, Dror, Shaw, "Parallel random numbers: as easy as 1, 2, 3", SC'11),
// counter = shot index + offset, key = seed.

template <typename C>
__global__ void chunk_sum_kernel(const C* psi, int64_t N, double* sums) {
  __shared__ double red[32];
  const int64_t b0 = (int64_t)blockIdx.x * SAMPLE_CHUNK;
  double acc = 0.0;
  for (int i = threadIdx.x; i < SAMPLE_CHUNK; i += blockDim.x) {
    const int64_t x = b0 + i;
    if (x < N) {
      const C v = psi[x];
      acc = fma((double)v.x, (double)v.x, fma((double)v.y, (double)v.y, acc));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
    sums[blockIdx.x] = s;
  }
}

// Inclusive scan over the lanes of a warp.
__device__ __forceinline__ double warp_scan(double v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += u;
  }
  return v;
}

// Exclusive scan of nb chunk sums by one block (sequential per thread
// segment, then a scan of segment totals by shuffles); prefix[nb] = total.
__global__ void __launch_bounds__(1024) scan_kernel(const double* sums, int64_t nb, double* prefix) {
  __shared__ double wtot[32];
  const int T = blockDim.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t per = (nb + T - 1) / T;
  const int64_t lo = threadIdx.x * per, hi = lo + per < nb ? lo + per : nb;
  double s = 0.0;
  for (int64_t i = lo; i < hi; ++i) s += sums[i];
  const double inc = warp_scan(s);
  if (lane == 31) wtot[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    const double v = wtot[lane], w = warp_scan(v);
    if (lane == 31) prefix[nb] = w;
    wtot[lane] = w - v;
  }
  __syncthreads();
  double run = wtot[warp] + (inc - s);
  for (int64_t i = lo; i < hi; ++i) {
    prefix[i] = run;
    run += sums[i];
  }
}

// One CTA per shot (grid-stride), 128 threads with a segment of 32 amplitudes
// of the chunk each.  One thread per shot walked up to 4096 amplitudes, each
// a dependent load and FP64 add: sampling 100 shots at n = 20 took 1376 us,
// now 39 (100,000 shots: 5.5 -> 2.9 ms; the FP64 work per shot, two
// operations per amplitude of one chunk, is no larger than a warp's 32 walks
// took).
constexpr int DRAW_THREADS = 128, DRAW_SEG = SAMPLE_CHUNK / DRAW_THREADS;

template <typename C>
__global__ void __launch_bounds__(DRAW_THREADS) draw_kernel(const C* psi, int64_t N, const double* sums, const double* prefix,
                                                            int64_t nb, int64_t nshots, uint64_t seed, uint64_t offset,
                                                            int64_t* out) {
  __shared__ double seg[DRAW_THREADS];      // running sum before each segment
  __shared__ double wtot[DRAW_THREADS / 32];
  __shared__ int first, last;               // the segment holding u; the last one with weight
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double total = prefix[nb];
  for (int64_t s = blockIdx.x; s < nshots; s += gridDim.x) {
    const uint64_t ctr = (uint64_t)s + offset;
    uint32_t c[4] = {(uint32_t)ctr, (uint32_t)(ctr >> 32), 0u, 0u};
    philox4x32_10(c, (uint32_t)seed, (uint32_t)(seed >> 32));
    const double u = u01_from(c[0], c[1]) * total;
    const int64_t lo = pick_chunk(prefix, sums, nb, u);  // the same in every thread
    const int64_t x0 = lo * SAMPLE_CHUNK, mine = x0 + tid * DRAW_SEG;
    double sum = 0.0;
    if (mine < N) {
      const int64_t len = N - mine < DRAW_SEG ? N - mine : DRAW_SEG;
#pragma unroll 8
      for (int i = 0; i < (int)len; ++i) {
        const C v = psi[mine + i];
        sum = fma((double)v.x, (double)v.x, fma((double)v.y, (double)v.y, sum));
      }
    }
    if (tid == 0) first = DRAW_THREADS, last = -1;
    const double inc = warp_scan(sum);
    if (lane == 31) wtot[warp] = inc;
    __syncthreads();
    double run = prefix[lo] + (inc - sum);
    for (int w = 0; w < warp; ++w) run += wtot[w];
    seg[tid] = run;
    if (sum > 0.0) {
      atomicMax(&last, tid);
      if (run + sum > u) atomicMin(&first, tid);
    }
    __syncthreads();
    if (tid == 0) {
      // first amplitude with weight whose running sum exceeds u; where the
      // rounding of the sums leaves none, the chunk's last one with weight
      int64_t pick = -1, last_nz = -1;
      for (int g = first < DRAW_THREADS ? first : last; g >= 0 && g <= last && pick < 0; ++g) {
        double r = seg[g];
        const int64_t y0 = x0 + g * DRAW_SEG;
        const int len = N - y0 < DRAW_SEG ? (int)(N - y0) : DRAW_SEG;
        double pr[DRAW_SEG];
#pragma unroll
        for (int i = 0; i < DRAW_SEG; ++i) {
          pr[i] = 0.0;
          if (i < len) {
            const C v = psi[y0 + i];
            pr[i] = fma((double)v.x, (double)v.x, (double)v.y * (double)v.y);
          }
        }
#pragma unroll
        for (int i = 0; i < DRAW_SEG; ++i) {
          r += pr[i];
          if (pr[i] > 0.0) {
            last_nz = y0 + i;
            if (r > u && pick < 0) pick = y0 + i;
          }
        }
      }
      out[s] = pick >= 0 ? pick : (last_nz >= 0 ? last_nz : x0);
    }
    __syncthreads();  // seg, first and last are rewritten for the next shot
  }
}

// States of one chunk (n <= 12): every CTA builds the running sums of the
// whole state in shared memory and its threads search them, one shot each.
// A CTA per shot would read the chunk again for every shot: 100,000 shots at
// n = 8 took 1.65 ms that way (0.41 with a walk per thread, now 0.04), at
// n = 12 2.7 ms (5.4 and 0.04).
constexpr int CDF_THREADS = 512, CDF_SEG = SAMPLE_CHUNK / CDF_THREADS;
static_assert(CDF_SEG == 8, "a byte of weight bits per thread");

template <typename C>
__global__ void __launch_bounds__(CDF_THREADS) draw_cdf_kernel(const C* psi, int N, const double* prefix,
                                                               int64_t nshots, uint64_t seed, uint64_t offset,
                                                               int64_t* out) {
  __shared__ double cdf[SAMPLE_CHUNK];
  __shared__ double wtot[CDF_THREADS / 32];
  __shared__ uint8_t weight[CDF_THREADS];  // bit i of a byte: its thread's i-th amplitude has weight
  __shared__ int last_nz;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) last_nz = 0;
  double pr[CDF_SEG];
  double sum = 0.0;
  int nz = -1;
  unsigned bits = 0;
#pragma unroll
  for (int i = 0; i < CDF_SEG; ++i) {
    const int x = tid * CDF_SEG + i;
    pr[i] = 0.0;
    if (x < N) {
      const C v = psi[x];
      pr[i] = fma((double)v.x, (double)v.x, (double)v.y * (double)v.y);
      if (pr[i] > 0.0) nz = x, bits |= 1u << i;
    }
    sum += pr[i];
  }
  const double inc = warp_scan(sum);
  if (lane == 31) wtot[warp] = inc;
  __syncthreads();
  double run = inc - sum;
  for (int w = 0; w < warp; ++w) run += wtot[w];
#pragma unroll
  for (int i = 0; i < CDF_SEG; ++i) {
    run += pr[i];
    cdf[tid * CDF_SEG + i] = run;
  }
  weight[tid] = (uint8_t)bits;
  if (nz >= 0) atomicMax(&last_nz, nz);
  __syncthreads();
  const double total = prefix[1];
  for (int64_t s = (int64_t)blockIdx.x * CDF_THREADS + tid; s < nshots; s += (int64_t)gridDim.x * CDF_THREADS) {
    const uint64_t ctr = (uint64_t)s + offset;
    uint32_t c[4] = {(uint32_t)ctr, (uint32_t)(ctr >> 32), 0u, 0u};
    philox4x32_10(c, (uint32_t)seed, (uint32_t)(seed >> 32));
    const double u = u01_from(c[0], c[1]) * total;
    out[s] = pick_index(cdf, weight, N, u, last_nz);
  }
}

template <typename C>
cudaError_t launch_sample(int n, const C* psi, int64_t nshots, uint64_t seed, uint64_t offset, double* ws,
                          int64_t* out, cudaStream_t st) {
  const int64_t N = (int64_t)1 << n;
  const int64_t nb = (N + SAMPLE_CHUNK - 1) / SAMPLE_CHUNK;
  double* sums = ws;
  double* prefix = ws + nb;
  chunk_sum_kernel<C><<<(unsigned)nb, 256, 0, st>>>(psi, N, sums);
  scan_kernel<<<1, 1024, 0, st>>>(sums, nb, prefix);
  if (nshots > 0 && nb == 1) {
    const int64_t want = (nshots + CDF_THREADS - 1) / CDF_THREADS;
    draw_cdf_kernel<C><<<(unsigned)(want < 256 ? want : 256), CDF_THREADS, 0, st>>>(psi, (int)N, prefix, nshots, seed,
                                                                                    offset, out);
  } else if (nshots > 0)
    draw_kernel<C><<<(unsigned)(nshots < 65536 ? nshots : 65536), DRAW_THREADS, 0, st>>>(psi, N, sums, prefix, nb,
                                                                                         nshots, seed, offset, out);
  return cudaGetLastError();
}

template cudaError_t launch_sample<double2>(int, const double2*, int64_t, uint64_t, uint64_t, double*, int64_t*,
                                            cudaStream_t);
template cudaError_t launch_sample<float2>(int, const float2*, int64_t, uint64_t, uint64_t, double*, int64_t*,
                                           cudaStream_t);

}  // namespace qg
