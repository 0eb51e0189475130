"""The sampler's searches (csrc/qg_draw.cuh, compiled for the host) against a
plain walk, and on running sums that are not monotone in the last bit, as
sums joined over threads are: a state or chunk of zero weight is never
returned while there is one with weight."""
import ctypes

import numpy as np
import pytest

from host_build import compile_host

SOURCE = """
#include "qg_draw.cuh"
extern "C" int64_t chunk(const double* prefix, const double* sums, int64_t nb, double u) {
  return qg::pick_chunk(prefix, sums, nb, u);
}
extern "C" int index(const double* cdf, const uint8_t* weight, int N, double u, int last) {
  return qg::pick_index(cdf, weight, N, u, last);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    L = compile_host(SOURCE, tmp_path_factory.mktemp("draw"), "draw")
    P, D = ctypes.c_void_p, ctypes.c_double
    L.chunk.argtypes, L.chunk.restype = [P, P, ctypes.c_int64, D], ctypes.c_int64
    L.index.argtypes, L.index.restype = [P, P, ctypes.c_int, D, ctypes.c_int], ctypes.c_int
    return L


def _index(lib, cdf, pr, u):
    bits = np.packbits((pr > 0).astype(np.uint8), bitorder="little")
    nz = np.nonzero(pr > 0)[0]
    return lib.index(cdf.ctypes.data, bits.ctypes.data, len(cdf), u, int(nz[-1]) if nz.size else 0)


def _chunk(lib, prefix, sums, u):
    return lib.chunk(prefix.ctypes.data, sums.ctypes.data, len(sums), u)


def _ulp_steps(x, k):
    for _ in range(abs(k)):
        x = np.nextafter(x, np.inf if k > 0 else -np.inf)
    return x


@pytest.mark.parametrize("N", [2, 8, 24, 4096])
@pytest.mark.parametrize("density", [1.0, 0.2, 0.01])
def test_index_equals_the_walk(lib, N, density):
    rng = np.random.default_rng(N)
    pr = rng.random(N) * (rng.random(N) < density)
    pr[rng.integers(N)] = 0.5
    cdf = np.cumsum(pr)
    for u in np.concatenate([rng.random(200) * cdf[-1], cdf[:50], [0.0, cdf[-1]]]):
        above = np.nonzero((cdf > u) & (pr > 0))[0]
        assert _index(lib, cdf, pr, u) == (above[0] if above.size else np.nonzero(pr > 0)[0][-1])


@pytest.mark.parametrize("seed", range(20))
def test_index_has_weight_whatever_the_last_bits(lib, seed):
    """Segments of eight whose bases are off by a few units in the last place."""
    rng = np.random.default_rng(seed)
    N = 256
    pr = rng.random(N) * np.repeat(rng.random(N // 8) < 0.3, 8)
    pr[3] = 0.25
    cdf = np.cumsum(pr)
    for s in range(1, N // 8):
        cdf[8 * s: 8 * s + 8] = [_ulp_steps(x, int(k)) for x, k in zip(cdf[8 * s: 8 * s + 8], [rng.integers(-3, 4)] * 8)]
    for x in cdf:
        for k in range(-4, 5):
            assert pr[_index(lib, cdf, pr, _ulp_steps(x, k))] > 0


def test_index_without_weight(lib):
    z = np.zeros(16)
    assert _index(lib, z, z, 0.0) == 0
    nan = np.full(16, np.nan)
    assert _index(lib, nan, z, float("nan")) == 0


@pytest.mark.parametrize("seed", range(20))
def test_chunk_has_weight_whatever_the_last_bits(lib, seed):
    rng = np.random.default_rng(seed)
    nb = 64
    sums = rng.random(nb) * (rng.random(nb) < 0.4)
    sums[rng.integers(nb)] = 0.3
    exact = np.concatenate([[0.0], np.cumsum(sums)])
    prefix = np.array([_ulp_steps(x, int(rng.integers(-3, 4))) if x else x for x in exact])
    for c, x in enumerate(prefix[:-1]):
        for k in range(-4, 5):
            assert sums[_chunk(lib, prefix, sums, _ulp_steps(x, k))] > 0
        if sums[c] > 0:  # well inside a chunk: that chunk
            assert _chunk(lib, prefix, sums, exact[c] + 0.5 * sums[c]) == c


def test_chunk_without_weight(lib):
    z, nan = np.zeros(8), np.full(8, np.nan)
    assert _chunk(lib, np.zeros(9), z, 0.0) == 0
    assert _chunk(lib, np.full(9, np.nan), nan, float("nan")) == 0
