"""complex128 calls whose workspace holds the double sweeps' layout but not the
fixed-point sweeps' phase tables run the double sweeps.  Both kinds of sweep
are deterministic and round differently, so the bits tell which ran: with
exactly the workspace of a handle that is set to the double sweeps the results
differ from the fixed-point ones and repeat.  Less than that is refused.  And
a circuit for qg_grad_noalloc whose tables alone exceed the fixed scratch."""
import ctypes

import numpy as np
import pytest

from conftest import obs_dict, rel_err
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _case(n, L, ent, seed):
    from qradient_gb300 import McClean

    rng = np.random.default_rng(seed)
    axes, angles = rng.integers(0, 3, (L, n)), rng.uniform(0, 6, (L, n))
    kind, q0, q1, w = [3] * (n - 1), list(range(n - 1)), list(range(1, n)), [1.0] * (n - 1)
    c = McClean(n, obs_dict(n, np.array(kind), np.array(q0), np.array(q1), np.array(w)), L, axes=axes, angles=angles,
                entangler=ent)
    ref = O.mcclean_grad(n, axes, angles, O.Terms(kind, q0, q1, w), entangler={"cnot": 1, "cz": 2, None: 0}[ent],
                         placement=0)
    return c, angles, ref


@pytest.mark.parametrize("n,ent", [(9, "cnot"), (12, "cz"), (13, "cnot"), (20, None)])
@pytest.mark.parametrize("ini", [False, True])
def test_double_sweeps_without_room_for_tables(n, ent, ini):
    import torch

    from qradient_gb300 import _lib

    lib, dev, op = _lib.load(), torch.device("cuda"), _lib.QG_OP_GRAD_UNCOMPUTE
    c, angles, (E0, g0) = _case(n, 3, ent, n)
    plain, _, _ = _case(n, 3, ent, n)
    plain.set_tuning(0, 0, _lib.QG_TUNE_FWD_PLAIN)
    nat, pnat = c.native(), plain.native()
    size = pnat.workspace_bytes(_lib.QG_C128, op)
    assert size < nat.workspace_bytes(_lib.QG_C128, op)
    params = torch.tensor(angles.reshape(-1), dtype=torch.float64, device=dev)
    state = None
    if ini:  # |0..0>, the default start, as a caller's state
        state = torch.zeros(2 ** n, dtype=torch.complex128, device=dev)
        state[0] = 1.0

    def grad(x, nbytes):
        ws = torch.empty(nbytes, dtype=torch.uint8, device=dev)
        E, g = x.grad(params, _lib.QG_C128, dev, op, workspace=ws, ini_state=state)[:2]
        return float(E), g.cpu().numpy().reshape(g0.shape)

    Ep, gp = grad(pnat, size)
    Ef, gf = grad(nat, nat.workspace_bytes(_lib.QG_C128, op))
    E, g = grad(nat, size)
    assert np.array_equal(gf, grad(nat, nat.workspace_bytes(_lib.QG_C128, op))[1])
    assert np.array_equal(g, grad(nat, size)[1])
    for e, x in ((Ep, gp), (Ef, gf), (E, g)):
        assert abs(e - E0) <= 1e-12 * max(1.0, abs(E0)) and rel_err(x, g0) <= 1e-12
    assert not np.array_equal(g, gf)
    if ini:  # (without a start state the layout has one layer fewer to hold)
        ws = torch.empty(size - 256, dtype=torch.uint8, device=dev)
        e, out = torch.empty(1, dtype=torch.float64, device=dev), torch.empty(3 * n, dtype=torch.float64, device=dev)
        p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
        st = lib.qg_grad(nat._h, _lib.QG_C128, op, p(params), p(state), p(ws), ws.numel(), p(e), p(out), None)
        assert st == _lib.QG_ERR_WORKSPACE


def test_noalloc_deep_circuit():
    """n = 8: 4 KB of tables per layer, 17 MB in all.  Tolerance: each of the
    4,200 layers applies up to 8 rotations and a ladder to states of norm 1, a
    few roundings of 2^-53 each; both sides together stay below
    4,200 * 8 * 4 * 2^-53 = 1.5e-11 of the largest weight's share."""
    import torch

    from qradient_gb300 import _lib

    n, L = 8, 4200
    c, angles, (E0, g0) = _case(n, L, "cnot", 3)
    nat, dev = c.native(), torch.device("cuda")
    need = nat.workspace_bytes(_lib.QG_C128, _lib.QG_OP_GRAD_UNCOMPUTE)
    assert need > 16 << 20
    params = torch.tensor(angles.reshape(-1), dtype=torch.float64, device=dev)
    e, g = torch.empty(1, dtype=torch.float64, device=dev), torch.empty(L * n, dtype=torch.float64, device=dev)
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    torch.cuda.synchronize()
    _lib.check(_lib.load().qg_grad_noalloc(nat._h, _lib.QG_C128, p(params), None, p(e), p(g), None))
    torch.cuda.synchronize()
    assert abs(float(e) - E0) <= 1.5e-11 * (n - 1)
    assert np.max(np.abs(g.cpu().numpy().reshape(g0.shape) - g0)) <= 1.5e-11 * (n - 1)
    # a workspace with room for the tables: the fixed-point sweeps, other bits
    _, gf = nat.grad(params, _lib.QG_C128, dev, _lib.QG_OP_GRAD_UNCOMPUTE)[:2]
    assert not torch.equal(gf, g)
