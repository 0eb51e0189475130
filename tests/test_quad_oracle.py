"""The extended-precision oracle against the double one: the same circuits agree
to double rounding, and what is exact in the extended form stays exact."""
import numpy as np
import pytest

from oracle import oracle as O
from oracle import quad as Q


@pytest.mark.parametrize("n,L,ent,place", [(3, 2, 1, 0), (6, 4, 2, 1), (8, 3, 3, 0), (9, 5, 0, 0)])
def test_mcclean(n, L, ent, place):
    rng = np.random.default_rng(n)
    axes, angles = rng.integers(0, 3, (L, n)), rng.uniform(-6, 6, (L, n))
    t = O.Terms([3, 0, 1, 2], [0, 0, 1, n - 1], [1, 0, 1, n - 1], [1.0, 0.5, -0.25, 0.75])
    E0, g0 = O.mcclean_grad(n, axes, angles, t, entangler=ent, placement=place)
    for unc in (False, True):
        E, g = Q.mcclean(n, axes, angles, t, entangler=ent, placement=place, uncompute=unc)
        assert g.dtype == np.longdouble and abs(E - E0) <= 1e-14 and np.max(np.abs(g - g0)) <= 1e-13
    _, s0 = O.mcclean_run(n, axes, angles, t, entangler=ent, placement=place, want_state=True)
    _, s = Q.mcclean(n, axes, angles, t, entangler=ent, placement=place, grad=False)
    assert np.max(np.abs(s - s0)) <= 1e-14
    assert abs(np.sum(s.real ** 2 + s.imag ** 2) - 1) <= 64 * L * n * 2.0 ** -Q.BITS


def test_qaoa():
    rng = np.random.default_rng(3)
    n, p = 8, 3
    t = O.Terms([3] * n, list(range(n - 1)) + [0], list(range(1, n)) + [n - 1], [1.0] * n)
    b, g = rng.uniform(0, 3, p), rng.uniform(0, 3, p)
    E0, g0 = O.qaoa_grad(n, b, g, t)
    E, gr = Q.qaoa(n, b, g, t)
    assert abs(E - E0) <= 1e-13 and np.max(np.abs(gr - g0)) <= 1e-12
