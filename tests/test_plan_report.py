"""qg_get_plan reports the sweeps that run: the fixed-point layouts of complex128
handles, the double sweeps where a setting asks for them, complex64's.  A
history holds one state per sweep, which ties the report to the workspace."""
import ctypes

import numpy as np
import pytest

from test_lib_abi import _create


class _Nat:
    def __init__(self, h):
        self._h = h


def _plan(h, dtype, op):
    from qradient_gb300 import tuning

    return tuning.get_plan(_Nat(h), dtype, op)


@pytest.mark.parametrize("n,history,uncompute", [
    (8, [8], [8]), (10, [10], [10]), (11, [8, 8], [8, 8]), (17, [9, 9], [9, 9]), (18, [10, 10], [10, 10]),
    (20, [11, 11], [11, 11]), (24, [10, 10, 10], [10, 10, 10]), (28, [12, 11, 11], [10, 10, 10, 10])])
def test_default_complex128_layouts(n, history, uncompute):
    from qradient_gb300 import _lib

    L = 3
    st, h = _create(n, L, np.zeros((L, n)))
    assert st == 0
    for op, want in ((_lib.QG_OP_GRAD_HISTORY, history), (_lib.QG_OP_GRAD_UNCOMPUTE, uncompute)):
        p = _plan(h, 0, op)
        assert p["fixed_point"] and [t for t, _ in p["sweeps"]] == want
        assert sum(k for _, k in p["sweeps"]) == n and p["ctas_per_sm"] >= 1
    b = ctypes.c_size_t()
    lib = _lib.load()
    assert lib.qg_workspace_size(h, 0, _lib.QG_OP_GRAD_HISTORY, ctypes.byref(b)) == 0
    # lambda (two buffers: the CNOT ladder) and a state per sweep of the L layers and the start's layer
    states = 2 + (L + 1) * len(history)
    assert states <= b.value / (16 * 2 ** n) < states + 1 or n < 18
    lib.qg_destroy(h)


@pytest.mark.parametrize("tile,flags,dtype,fixed,sweeps", [
    (9, 0, 0, True, [9, 9, 9]), (12, 1, 0, True, [12, 12]), (7, 0, 0, False, [7, 7, 7, 7, 7]),
    (0, 2, 0, False, [12, 11]), (11, 2, 0, False, [11, 11, 11]), (0, 0, 1, False, [12, 12]), (13, 0, 1, False, [13, 13])])
def test_settings(tile, flags, dtype, fixed, sweeps):
    from qradient_gb300 import _lib

    lib = _lib.load()
    st, h = _create(20, 2, np.zeros((2, 20)))
    assert st == 0
    assert lib.qg_set_tuning(h, dtype, tile, 0, flags) == 0
    for op in (0, 1, 2):
        p = _plan(h, dtype, op)
        assert p["fixed_point"] == fixed and [t for t, _ in p["sweeps"]] == sweeps
        assert sum(k for _, k in p["sweeps"]) == 20
    lib.qg_destroy(h)


def test_small_circuits_and_bad_arguments():
    from qradient_gb300 import _lib

    lib = _lib.load()
    st, h = _create(5, 1, np.zeros((1, 5)))
    assert st == 0
    assert _plan(h, 0, 0) == {"fixed_point": False, "sweeps": [(5, 5)], "ctas_per_sm": 1}
    a, b = ctypes.c_int(), ctypes.c_int()
    assert lib.qg_get_plan(h, 0, 1, ctypes.byref(a), ctypes.byref(b), None, None, None) == 0
    for dtype, op in ((2, 0), (0, 3), (0, -1)):
        assert lib.qg_get_plan(h, dtype, op, ctypes.byref(a), ctypes.byref(b), None, None, None) == _lib.QG_ERR_INVALID
    assert lib.qg_get_plan(h, 0, 0, None, ctypes.byref(b), None, None, None) == _lib.QG_ERR_INVALID
    lib.qg_destroy(h)
