"""Batched cluster kernels, many short launches in a row: the first CTA of a
cluster hands job numbers to the others as they start.  Every launch gives the
oracle's values (1e-12 normwise in complex128, 1e-4 in complex64, as in the
other batched tests)."""
import numpy as np
import pytest

from conftest import obs_dict, rel_err
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,sizes,tol", [("complex128", (5, 13, 14), 1e-12), ("complex64", (5, 14, 15), 1e-4)])
def test_short_launches(dtype, sizes, tol):
    import torch

    from qradient_gb300 import McClean
    from qradient_gb300.batched import Batch

    kind, q0, q1, w = [3, 0], [0, 1], [1, 1], [1.0, 0.5]
    cases = []
    for n in sizes:
        rng = np.random.default_rng(n)
        axes, angles = rng.integers(0, 3, (1, n)), rng.uniform(-3, 3, (1, n))
        c = McClean(n, obs_dict(n, np.array(kind), np.array(q0), np.array(q1), np.array(w)), 1, axes=axes,
                    angles=angles, dtype=dtype)
        cases.append((c, O.mcclean_grad(n, axes, angles, O.Terms(kind, q0, q1, w), entangler=1, placement=0)))
    b = Batch(dtype=dtype, use_graph=False, cluster_from=5)
    for c, _ in cases * 20:
        b.add(c)
    b.finalize()
    out = []
    for _ in range(40):
        E, _ = b.execute()
        out.append((E.clone(), b.grads_flat.clone()))
    torch.cuda.synchronize()
    for E, G in out:
        E, G, off = E.cpu().numpy(), G.cpu().numpy(), 0
        for k, (c, (E0, g0)) in enumerate(cases * 20):
            assert abs(E[k] - E0) <= tol, c.qnum
            assert rel_err(G[off: off + g0.size].reshape(g0.shape), g0) <= tol, c.qnum
            off += g0.size
