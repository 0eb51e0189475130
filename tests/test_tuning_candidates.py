"""The autotuner's candidates hold every uniform layout that the library picks
by itself."""
import numpy as np
import pytest

from test_lib_abi import _create
from test_plan_report import _plan


@pytest.mark.parametrize("n", range(8, 31))
def test_default_depths_are_candidates(n):
    from qradient_gb300 import _lib, tuning

    st, h = _create(n, 1, np.zeros((1, n)))
    assert st == 0
    for op in (_lib.QG_OP_GRAD_HISTORY, _lib.QG_OP_GRAD_UNCOMPUTE):
        tiles = {t for t, _ in _plan(h, _lib.QG_C128, op)["sweeps"]}
        if len(tiles) == 1:
            assert (tiles.pop(), 0, _lib.QG_TUNE_FWD_PIPELINED) in tuning.sweep_candidates(_lib.QG_C128, n)
    _lib.load().qg_destroy(h)


def test_candidates_are_settings_the_library_takes():
    from qradient_gb300 import _lib, tuning

    lib = _lib.load()
    for dtype in (_lib.QG_C128, _lib.QG_C64):
        for n in (3, 8, 13, 18, 19, 24):
            st, h = _create(n, 1, np.zeros((1, n)))
            cand = tuning.sweep_candidates(dtype, n)
            assert st == 0 and cand[0] == (0, 0, 0) and len(set(cand)) == len(cand)
            assert all(lib.qg_set_tuning(h, dtype, *c) == 0 for c in cand)
            lib.qg_destroy(h)
