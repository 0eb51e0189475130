"""complex128 batches whose lambda = O psi is not finite: NaN and infinite
weights, and finite ones whose sum overflows, in one CTA and in clusters.  E
is not finite and the whole gradient of that job is NaN, as for a circuit run
alone; the batch's other jobs keep their results (1e-12 normwise, as in the
other complex128 tests)."""
import numpy as np
import pytest

from conftest import obs_dict, rel_err
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# X on the last and the first qubit, Z on the first, ZZ on the first two: on
# |x_0 x_1> = 00 both diagonal terms add, so two weights of 1.5e308 overflow
KIND, Q0, Q1 = [3, 2, 0, 0], [0, 0, -1, 0], [1, 0, -1, 0]
WEIGHTS = [[np.nan, 0.5, -0.75, 0.25], [1.0, np.inf, -0.75, 0.25], [1.0, 0.5, -np.inf, 0.25], [1.0, 0.5, 0.25, np.nan],
           [1.5e308, 1.5e308, 0.25, 0.25]]


def _case(n, w, seed):
    from qradient_gb300 import McClean

    rng = np.random.default_rng(seed)
    L = 3
    axes, angles = rng.integers(0, 3, (L, n)), rng.uniform(-7, 7, (L, n))
    q0, q1 = [q % n for q in Q0], [q % n for q in Q1]
    c = McClean(n, obs_dict(n, np.array(KIND), np.array(q0), np.array(q1), np.array(w)), L, axes=axes, angles=angles)
    return c, axes, angles, O.Terms(KIND, q0, q1, w)


@pytest.mark.parametrize("weights", range(len(WEIGHTS)))
@pytest.mark.parametrize("cluster_from", [13, 5])
def test_gradient_is_nan_for_its_job_only(weights, cluster_from):
    from qradient_gb300.batched import Batch

    sizes = (4, 9, 12, 13, 14)
    for bad in range(len(sizes)):
        b = Batch(dtype="complex128", use_graph=False, cluster_from=cluster_from)
        cases = [_case(n, WEIGHTS[weights] if k == bad else [1.0, 0.5, -0.75, 0.25], n) for k, n in enumerate(sizes)]
        for case in cases:
            b.add(case[0])
        E, G = b.grad()
        for k, (c, axes, angles, terms) in enumerate(cases):
            g = G[k].cpu().numpy()
            if k == bad:
                assert not np.isfinite(float(E[k])), c.qnum
                assert np.all(np.isnan(g)), c.qnum
            else:
                E0, g0 = O.mcclean_grad(c.qnum, axes, angles, terms, entangler=1, placement=0)
                assert abs(float(E[k]) - E0) <= 1e-12 and rel_err(g.reshape(g0.shape), g0) <= 1e-12, c.qnum


def test_qaoa_cost_that_overflows():
    """beta and gamma entries both: 1.5e308 on every edge of a triangle."""
    from qradient_gb300 import Qaoa
    from qradient_gb300.batched import Batch

    for n in (6, 13, 14):
        zz = np.full((n, n), None)
        zz[0, 1] = zz[0, 2] = zz[1, 2] = 1.5e308
        good = np.full((n, n), None)
        good[0, 1] = good[0, 2] = good[1, 2] = 1.5
        b = Batch(dtype="complex128", use_graph=False)
        p = np.array([[0.3, 1e-308], [0.2, 2e-308]])
        b.add(Qaoa(n, {"zz": zz}, 2), params=p)
        b.add(Qaoa(n, {"zz": good}, 2), params=np.array([[0.3, 0.4], [0.2, 0.1]]))
        E, G = b.grad()
        assert not np.isfinite(float(E[0])) and np.all(np.isnan(G[0].cpu().numpy())), n
        assert np.isfinite(float(E[1])) and np.all(np.isfinite(G[1].cpu().numpy())), n
