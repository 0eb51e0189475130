"""Sweeps that wait on one another across launches: deep circuits at sizes
where several grids fit on the chip at once, repeated, in complex64 and (four
and eight amplitudes a thread) complex128.  Repeats are equal bit for bit;
against the oracle 1e-12 normwise (complex128) and single-precision rounding
in the worst case (complex64): 2^-24 of the observable's norm per operation,
4 (n + 2) a layer."""
import numpy as np
import pytest

from conftest import obs_dict, rel_err
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,L", [(8, 30), (9, 20), (10, 20), (12, 20), (14, 12), (16, 10), (17, 10), (18, 10)])
@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("mode", ["history", "uncompute"])
def test_repeats(n, L, dtype, mode):
    from qradient_gb300 import McClean

    rng = np.random.default_rng(n)
    axes, angles = rng.integers(0, 3, (L, n)), rng.uniform(0, 2 * np.pi, (L, n))
    kind, q0, q1, w = [3] * (n - 1) + [1], list(range(n - 1)) + [2], list(range(1, n)) + [2], [1.0] * (n - 1) + [0.5]
    E0, g0 = O.mcclean_grad(n, axes, angles, O.Terms(kind, q0, q1, w), entangler=1, placement=0)
    c = McClean(n, obs_dict(n, np.array(kind), np.array(q0), np.array(q1), np.array(w)), L, axes=axes, angles=angles,
                grad_mode=mode, dtype=dtype)
    E, g = c.grad_run()
    E, g = float(E), np.array(g)
    if dtype == "complex128":
        assert abs(E - E0) <= 1e-12 * max(1.0, abs(E0)) and rel_err(g, g0) <= 1e-12
    else:
        tol = np.sum(w) * 2.0 ** -24 * 4 * L * (n + 2)
        assert abs(E - E0) <= tol and np.max(np.abs(g - g0)) <= tol
    for _ in range(10):
        E2, g2 = c.grad_run()
        assert E2 == E and np.array_equal(g2, g)
    assert abs(c.run_expec_val() - E) <= (1e-12 if dtype == "complex128" else 2.0 ** -24 * n) * max(1.0, abs(E))
