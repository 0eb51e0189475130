"""complex128 calls whose workspace has no room for the fixed-point sweeps'
phase tables: the double sweeps run instead of a refusal, and a workspace too
small for those as well is refused.  Tolerance: 1e-12 normwise, as in the
other complex128 tests."""
import numpy as np
import pytest

from conftest import obs_dict, rel_err
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ent", [(9, "cnot"), (12, "cz"), (13, "cnot"), (20, None)])
def test_small_workspace(n, ent):
    import torch

    from qradient_gb300 import McClean, _lib, _native

    L, rng = 3, np.random.default_rng(n)
    axes, angles = rng.integers(0, 3, (L, n)), rng.uniform(0, 6, (L, n))
    kind, q0, q1, w = [3] * (n - 1), list(range(n - 1)), list(range(1, n)), [1.0] * (n - 1)
    E0, g0 = O.mcclean_grad(n, axes, angles, O.Terms(kind, q0, q1, w), entangler={"cnot": 1, "cz": 2, None: 0}[ent],
                            placement=0)
    c = McClean(n, obs_dict(n, np.array(kind), np.array(q0), np.array(q1), np.array(w)), L, axes=axes, angles=angles,
                entangler=ent)
    nat, dev = c.native(), torch.device("cuda")
    op = _lib.QG_OP_GRAD_UNCOMPUTE
    need = nat.workspace_bytes(_lib.QG_C128, op)
    params = torch.tensor(angles.reshape(-1), dtype=torch.float64, device=dev)
    for size in (need, need - 512):
        ws = torch.empty(size, dtype=torch.uint8, device=dev)
        E, g = nat.grad(params, _lib.QG_C128, dev, op, workspace=ws)[:2]
        assert abs(float(E) - E0) <= 1e-12 * max(1.0, abs(E0)), size
        assert rel_err(g.cpu().numpy().reshape(L, n), g0) <= 1e-12, size
    with pytest.raises(Exception):
        nat.grad(params, _lib.QG_C128, dev, op, workspace=torch.empty(need // 4, dtype=torch.uint8, device=dev))
