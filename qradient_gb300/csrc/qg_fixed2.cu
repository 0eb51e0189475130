// The fixed-point sweeps with four amplitudes a thread instead of eight, for
// states of few tiles (build_fixed in qg_capi.cu chooses).
#define QG_FIX_E 2
#include "qg_fixed.cu"
