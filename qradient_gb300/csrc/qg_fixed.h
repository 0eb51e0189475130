// Fixed-point sweeps of the complex128 path (qg_fixed.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "qg_internal.cuh"

namespace qg {

constexpr int FIX_TMIN = 8, FIX_TMAX = 12;  // tile bits with an instantiation
// A thread holds 2^FIX_E amplitudes.  With 16 instead of 8 a layer has fewer
// exchanges, but twice the registers halve the resident warps and the code no
// longer fits the instruction cache: n = 24, L = 20 31.3 against 28.9 ms.
// With 4 a circuit of few tiles has twice the warps to hide the latency of
// dependent instructions behind (see build_fixed, which chooses); those are
// the instantiations of up to FIX_TMAX2 tile bits in qg_fixed2.cu.
constexpr int FIX_E = 3, FIX_TMAX2 = 10;
constexpr int FIX_STAGES = (FIX_TMAX + 1) / 2;

// One sweep: every rotation on the tile's active bits (its top `nact` local
// bits), each as V D V^-1 with V the Clifford that turns the rotation's Pauli
// into Z.  Bits are handled in stages of e local bits from the top.
struct FixDesc {
  int32_t n, t, nact, nst;  // qubits, tile bits, active bits, stages
  int32_t e;                // in-thread bits: FIX_E or 2
  // The tile's local bits: [0, low) are the same global bits, [low, t) the
  // active ones, global [lo, lo + t - low).  Element offsets of the top
  // FIX_E local bits, and their images under the CNOT ladder and its inverse.
  int32_t low, lo;
  int64_t top[FIX_E], top_fwd[FIX_E], top_inv[FIX_E];
  uint64_t odd, even;       // ladder masks
  uint8_t code[FIX_STAGES];          // per stage, two bits per in-thread bit: 0 none (Z or inactive), 1 X, 2 Y
  // scaling of the fixed-point tile (see fix_schedule): log2 bound of the
  // loaded norm, right shifts before each stage of V^-1 and of V, and the
  // exponents of the results relative to the tile's
  int8_t B[2];
  int8_t sh_in[2][FIX_STAGES], sh_out[2][FIX_STAGES];
  int16_t kout[2];  // stored value = X * 2^(p + kout)  (p: the tile's norm exponent)
  int16_t kw;       // w = Xl Xq 2^-64 * 2^(pl + pq + kw)
  int8_t start, pre, lam_undo, psi_undo, periodic;
  int8_t cost, has_gslot;
  int8_t early;             // backward, chained: the launch before this one is a chained backward sweep
  int32_t cost_maxabs, gslot;
  double cost_w0;
  int32_t slot[FIX_TMAX];  // gradient slot per active bit (from the lowest), -1 none
  int32_t sweep;           // index into the flags
  int64_t tab, ctab;       // byte offsets of the phase tables in the table area
};

// What the table kernel needs of a whole circuit.
struct FixTables {
  int32_t e;                                  // in-thread bits of every sweep
  int32_t n, nsweeps, per_layer, ini_layers;  // ini_layers: leading layers of fixed Ry(pi/4)
  int32_t kind, nparams;                      // 0 McClean, 1 QAOA
  int32_t t[QMAX], nact[QMAX], lo[QMAX];      // per sweep of a layer: tile bits, active bits, lowest active bit
  int64_t off[QMAX];                          // table offset of each sweep inside a layer
  int64_t layer_bytes, tab0, ctab0, ctab_bytes, startp, flags;
  int32_t cost_maxabs, cost;
  double cost_w0;
};

struct FixPtrs {
  const double2* psi_in;
  double2* psi_out;
  const double2* lam_in;
  double2* lam_out;
  const char* area;  // table area
  const int32_t* cost_i;
  double* partials;
  const int32_t* flags;
  const double* startp;
  int32_t G;
};

__host__ __device__ inline int fix_stages(int nact, int e) { return nact <= 0 ? 1 : (nact + e - 1) / e; }
// Phase-table entries of a sweep: [in-thread index][thread index of the last
// stage's layout without its low bits, which are inactive unless that stage
// reaches the lowest bits].
__host__ __device__ inline int fix_table_skip(int t, int nact, int e) {
  const int lo = t - e * fix_stages(nact, e);
  return lo > 0 ? lo : 0;
}
inline int64_t fix_table_entries(int t, int nact, int e) { return (int64_t)1 << (t - fix_table_skip(t, nact, e)); }

int fix_ctas_per_sm(const FixDesc& d, bool bwd, bool uncompute);
cudaError_t launch_fix_tables(const FixTables& ft, const double* params, char* area, cudaStream_t st);
cudaError_t launch_fix_fwd(const FixDesc& d, const FixPtrs& p, int grid, cudaStream_t st, bool pdl);
// chained: history mode, every backward sweep of the call is launched so, and d.early is
// set on all but the first
cudaError_t launch_fix_bwd(const FixDesc& d, const FixPtrs& p, bool uncompute, bool chained, int grid,
                           cudaStream_t st, bool pdl);

}  // namespace qg
