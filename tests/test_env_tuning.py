"""QG_TILE_BITS_C128 and QG_CTAS_PER_SM set what qg_set_tuning sets, for
handles without a setting of their own, on the fixed-point sweeps as on the
double ones.  The history workspace shows it: a state per sweep, a table per
tile, a partial sum per CTA and gradient slot."""
import ctypes

import pytest

from test_lib_abi import _create

import numpy as np


def _bytes(n, L, tile=0, ctas=0, flags=0, op=1):
    from qradient_gb300 import _lib

    lib = _lib.load()
    st, h = _create(n, L, np.zeros((L, n)))
    assert st == 0
    assert lib.qg_set_tuning(h, 0, tile, ctas, flags) == 0
    b = ctypes.c_size_t()
    assert lib.qg_workspace_size(h, 0, op, ctypes.byref(b)) == 0
    lib.qg_destroy(h)
    return b.value


@pytest.mark.parametrize("n", [8, 13, 20, 24])
@pytest.mark.parametrize("tile", [6, 8, 9, 10, 11, 12])
def test_tile_bits_from_the_environment(monkeypatch, n, tile):
    default, want, other = _bytes(n, 3), _bytes(n, 3, tile), _bytes(n, 3, 10)
    monkeypatch.setenv("QG_TILE_BITS_C128", str(tile))
    assert _bytes(n, 3) == want
    assert _bytes(n, 3, 10) == other  # a handle's own setting comes first
    monkeypatch.setenv("QG_TILE_BITS_C128", "0")
    assert _bytes(n, 3) == default


@pytest.mark.gpu
@pytest.mark.parametrize("flags", [1, 2])
def test_ctas_per_sm_from_the_environment(monkeypatch, flags):
    default, want = _bytes(24, 3, flags=flags), _bytes(24, 3, ctas=1, flags=flags)
    assert want < default
    monkeypatch.setenv("QG_CTAS_PER_SM", "1")
    assert _bytes(24, 3, flags=flags) == want
