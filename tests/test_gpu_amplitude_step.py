"""What the fixed-point sweeps keep of an amplitude far below its tile's norm,
as include/qgrad.h says: an error of a few 2^-57 of the norm per sweep (four
roundings of at most one unit), and every digit on a handle set to the double
sweeps.  QAOA layers of angle zero leave the state as it is."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 9, 12, 13, 18])
def test_small_amplitudes(n):
    from qradient_gb300 import Qaoa, _lib, tuning

    zz = np.full((n, n), None)
    zz[0, 1] = 1.0
    rng = np.random.default_rng(n)
    p, N = 2, 2 ** n
    small = rng.normal(size=N) + 1j * rng.normal(size=N)
    start = np.where(np.arange(N) % 256 == 37, 1.0, 1e-18 * small).astype(np.complex128)
    start /= np.linalg.norm(start)
    for flags in (0, _lib.QG_TUNE_FWD_PLAIN):
        c = Qaoa(n, {"zz": zz}, p)
        c.set_tuning(0, 0, flags)
        c.run_expec_val(np.zeros(p), np.zeros(p), ini_state=start)
        plan = tuning.get_plan(c.native(), c._dtype_code, _lib.QG_OP_RUN)
        out = c.state.tensor.cpu().numpy()
        if flags:
            assert np.max(abs(out - start) / abs(start)) <= 1e-15
        else:
            assert plan["fixed_point"]
            sweeps = p * len(plan["sweeps"])
            # (a tile of t bits holds 2^(t-8) amplitudes of one size)
            norm = abs(start[37]) * 2.0 ** ((max(t for t, _ in plan["sweeps"]) - 8) / 2)
            assert np.max(abs(out - start)) <= sweeps * 4 * 2.0 ** -57 * norm * 2 ** 0.5
