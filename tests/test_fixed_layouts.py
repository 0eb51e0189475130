"""The exchange layouts and the scaling schedule of the fixed-point kernels, as
the library compiles them (csrc/qg_fixed_layout.cuh, built for the host), for
eight and for four amplitudes a thread and every tile size.

Norms: h counts half bits above 2^60 of the power of two that bounds a tile's
norm.  At no point does h exceed 5 (every component and partial product stays
inside 63 bits) or fall below -4, so the unit of a tile is at most 2^-58 of
that power of two, 2^-57 of the norm itself."""
import ctypes
import itertools

import pytest

from host_build import compile_host

SOURCE = """
#define QG_FIX_E %d
#include "qg_fixed_layout.cuh"
using namespace qg;
static_assert(E == QG_FIX_E && FIX_STAGES == 6, "");
template <int T>
static void lay(int* ns, int* eoff, int* ebase, int* slot) {
  using L = Lay<T>;
  *ns = L::NS;
  for (int s = 0; s < L::NS; ++s) {
    for (int c = 0; c < NA; ++c) *eoff++ = L::eoff(s, c);
    for (int t = 0; t < L::NT; ++t) *ebase++ = L::ebase(s, t);
  }
  for (int e = 0; e < (1 << T); ++e) slot[e] = L::sw(e);
}
extern "C" void layout(int t, int* ns, int* eoff, int* ebase, int* slot) {
  t == 8 ? lay<8>(ns, eoff, ebase, slot) : t == 9 ? lay<9>(ns, eoff, ebase, slot)
  : t == 10 ? lay<10>(ns, eoff, ebase, slot) : t == 11 ? lay<11>(ns, eoff, ebase, slot)
                                             : lay<12>(ns, eoff, ebase, slot);
}
extern "C" void schedule(int nst, const int* codes, int cost, int* B, int* in, int* out, int* kout, int* kw) {
  FixDesc d;
  memset(&d, 0, sizeof d);
  d.nst = nst;
  d.e = E;
  d.cost = cost ? COST_INT : COST_NONE;
  for (int s = 0; s < nst; ++s) d.code[s] = (uint8_t)codes[s];
  fix_schedule(d);
  for (int k = 0; k < 2; ++k) {
    B[k] = d.B[k];
    kout[k] = d.kout[k];
    for (int s = 0; s < nst; ++s) in[k * nst + s] = d.sh_in[k][s], out[k * nst + s] = d.sh_out[k][s];
  }
  *kw = d.kw;
}
"""


@pytest.fixture(scope="module")
def libs(tmp_path_factory):
    d = tmp_path_factory.mktemp("fixed")
    return {e: compile_host("#include <cstring>\n" + SOURCE % e, d, "fixed%d" % e) for e in (2, 3)}


def _layout(lib, e, T):
    stages = (T + e - 1) // e
    ns, nt = ctypes.c_int(), 1 << (T - e)
    eoff, ebase = (ctypes.c_int * (stages << e))(), (ctypes.c_int * (stages * nt))()
    slot = (ctypes.c_int * (1 << T))()
    lib.layout(T, ctypes.byref(ns), eoff, ebase, slot)
    assert ns.value == stages
    return ([list(eoff[s << e: (s + 1) << e]) for s in range(stages)],
            [list(ebase[s * nt: (s + 1) * nt]) for s in range(stages)], list(slot))


@pytest.mark.parametrize("e,T", [(3, t) for t in range(8, 13)] + [(2, t) for t in range(8, 11)])
def test_layouts_cover_the_tile(libs, e, T):
    eoff, ebase, slot = _layout(libs[e], e, T)
    assert sorted(slot) == list(range(1 << T))
    for s in range(len(eoff)):
        assert sorted(b | c for b in ebase[s] for c in eoff[s]) == list(range(1 << T))
        for c in eoff[s]:
            o = slot[c]
            for b in ebase[s]:
                assert b & c == 0
                # the kernels' split of a slot: only the low three bits of the offset meet the base
                assert (slot[b] ^ (o & 7)) + (o & ~7) == slot[b | c]


def _ways(T, eoff, ebase, slot, s):
    """Most lanes of a quarter warp on one of the eight 16-byte bank groups."""
    worst = 0
    for c in eoff[s]:
        for q in range(0, len(ebase[s]), 8):
            groups = [slot[b | c] & 7 for b in ebase[s][q:q + 8]]
            worst = max(worst, max(groups.count(g) for g in groups))
    return worst


@pytest.mark.parametrize("T", range(8, 13))
def test_eight_amplitudes_meet_no_bank_conflict(libs, T):
    lay = _layout(libs[3], 3, T)
    assert [_ways(T, *lay, s) for s in range(len(lay[0]))] == [1] * len(lay[0])


@pytest.mark.parametrize("T,ways", [(8, [1, 1, 2, 1]), (9, [1, 1, 1, 2, 1]), (10, [1, 1, 1, 2, 1])])
def test_four_amplitudes_meet_one_two_way_conflict(libs, T, ways):
    lay = _layout(libs[2], 2, T)
    assert [_ways(T, *lay, s) for s in range(len(lay[0]))] == ways


@pytest.mark.parametrize("e,most", [(3, 12), (2, 10)])
@pytest.mark.parametrize("cost", [0, 1])
def test_norms_stay_in_range(libs, e, most, cost):
    lib = libs[e]
    low = 5
    for nst in range(1, (most + e - 1) // e + 1):
        for m in itertools.product(range(e + 1), repeat=nst):
            # (the sweep that takes a QAOA layer's cost phase turns every bit of its tile, 8 or more)
            if sum(m) > most or (cost and sum(m) < 8):
                continue
            I = lambda k: (ctypes.c_int * k)()  # noqa: E731
            # `levels` X or Y bits in each stage, Z or none in the others
            codes = (ctypes.c_int * nst)(*[sum((1 + i % 2) << (2 * i) for i in range(k)) for k in m])
            B, sin, sout, kout, kw = I(2), I(2 * nst), I(2 * nst), I(2), ctypes.c_int()
            lib.schedule(nst, codes, cost, B, sin, sout, kout, ctypes.byref(kw))
            for back in (0, 1):
                assert 58 <= B[back] <= 62
                h, total = 2 * (B[back] - 60), 0
                if cost and not back:
                    h, total = h - 4, total + 2
                seen = [h]

                def stage(shift, levels):
                    nonlocal h, total
                    assert 0 <= shift < 32
                    h -= 2 * shift
                    total += shift
                    if shift:
                        seen.append(h)
                    h += levels
                    seen.append(h)

                for s in range(nst):
                    stage(sin[back * nst + s], m[s])
                if back:
                    assert kw.value == 64 - 2 * B[1] - sum(m) + 2 * total
                h, total = h - 8, total + 4
                seen.append(h)
                for s in reversed(range(nst)):
                    stage(sout[back * nst + s], m[s])
                if cost and back:
                    h, total = h - 4, total + 2
                    seen.append(h)
                assert kout[back] == -B[back] - sum(m) + total
                assert max(seen) <= 5, (m, back, seen)
                low = min(low, min(seen))
    assert low == -4
