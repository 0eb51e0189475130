"""Backward sweeps that start on psi before the sweep ahead has finished
(history mode, at most four tiles a CTA) against the oracle and against
themselves: deep circuits, so that a sweep that read lambda too early would
show, at one CTA, a part of the chip, one tile and several tiles a CTA, with
sweeps of different grids in one chain.  Tolerance: 1e-12 normwise, as in the
other complex128 tests; repeats are equal bit for bit."""
import numpy as np
import pytest

from conftest import obs_dict, rel_err
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,L,ent,place", [(8, 40, "cz", "before"), (9, 40, "cnot", "before"), (12, 30, "cz", "after"), (13, 30, "cnot", "after"),
                                           (17, 20, "cnot", "before"), (19, 10, None, "before"),
                                           (20, 8, "cnot_periodic", "before"), (21, 5, "cnot", "before")])
def test_mcclean(n, L, ent, place):
    from qradient_gb300 import McClean

    rng = np.random.default_rng(n)
    axes, angles = rng.integers(0, 3, (L, n)), rng.uniform(0, 2 * np.pi, (L, n))
    kind, q0, q1, w = [3] * (n - 1) + [0], list(range(n - 1)) + [1], list(range(1, n)) + [1], [1.0] * (n - 1) + [0.5]
    E0, g0 = O.mcclean_grad(n, axes, angles, O.Terms(kind, q0, q1, w),
                            entangler={"cnot": 1, "cz": 2, "cnot_periodic": 3, None: 0}[ent],
                            placement=1 if place == "after" else 0)
    c = McClean(n, obs_dict(n, np.array(kind), np.array(q0), np.array(q1), np.array(w)), L, axes=axes, angles=angles,
                entangler=ent, placement=place, grad_mode="history")
    E, g = c.grad_run()
    E, g = float(E), np.array(g)
    assert abs(E - E0) <= 1e-12 * max(1.0, abs(E0)) and rel_err(g, g0) <= 1e-12
    for _ in range(20):
        E2, g2 = c.grad_run()
        assert E2 == E and np.array_equal(g2, g)


@pytest.mark.parametrize("n,p", [(10, 12), (14, 10), (18, 6), (21, 2)])
def test_qaoa(n, p):
    """With the cost's own sum, which needs both states as they were loaded."""
    from qradient_gb300 import Qaoa
    from qradient_gb300.optimization_problems import MaxCut, random_regular_edges

    rng = np.random.default_rng(n)
    edges = random_regular_edges(3, n - n % 2, n)
    betas, gammas = rng.uniform(-1, 4, p), rng.uniform(-1, 4, p)
    E0, g0 = O.qaoa_grad(n, betas, gammas, O.Terms([3] * len(edges), edges[:, 0], edges[:, 1], [1.0] * len(edges)))
    q = Qaoa(n, MaxCut(n, edge_set=edges).to_observable(), p, grad_mode="history")
    E, g = q.grad_run(betas, gammas)
    E, g = float(E), np.array(g)
    assert abs(E - E0) <= 1e-12 * max(1.0, abs(E0)) and rel_err(g, g0) <= 1e-12
    for _ in range(20):
        E2, g2 = q.grad_run(betas, gammas)
        assert E2 == E and np.array_equal(g2, g)
