"""The observable pass's own ordering of diagonal terms and its integer sums
for a single weight, against the oracle: one weight that no power of two
divides, runs of equal weights, all weights different; one term, and more
terms than the kernel has threads.  Tolerances: 1e-12 (complex128) and 2^-24
of the sum of the weights times the operations of one layer and the terms
(complex64, worst case)."""
import numpy as np
import pytest

from conftest import obs_dict
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,terms", [(4, 1), (9, 45), (10, 7), (12, 78), (13, 20), (16, 136), (24, 300)])
@pytest.mark.parametrize("weights", ["one", "runs", "all"])
def test_orders(n, terms, weights):
    from qradient_gb300 import McClean

    rng = np.random.default_rng(n)
    pairs = [(i, i) for i in range(n)] + [(i, j) for i in range(n) for j in range(i + 1, n)]
    pick = [pairs[i] for i in rng.permutation(len(pairs))[:terms]]
    kind = [2 if a == b else 3 for a, b in pick]
    q0, q1 = [a for a, _ in pick], [b for _, b in pick]
    w = {"one": np.full(terms, 0.37), "runs": rng.choice([0.37, -1.0, 0.2], terms),
         "all": rng.uniform(-1, 1, terms)}[weights]
    axes, angles = rng.integers(0, 3, (1, n)), rng.uniform(0, 6, (1, n))
    E0, g0 = O.mcclean_grad(n, axes, angles, O.Terms(kind, q0, q1, list(w)), entangler=1, placement=0)
    obs = obs_dict(n, np.array(kind), np.array(q0), np.array(q1), np.array(w))
    for dtype, tol in (("complex128", 1e-12), ("complex64", 2.0 ** -24 * (4 * (n + 2) + terms))):
        c = McClean(n, obs, 1, axes=axes, angles=angles, dtype=dtype)
        E, g = c.grad_run()
        scale = max(1.0, np.sum(np.abs(w)))
        assert abs(E - E0) <= tol * scale and np.max(np.abs(g - g0)) <= tol * scale, (dtype, n)
        assert abs(c.run_expec_val() - E0) <= tol * scale
