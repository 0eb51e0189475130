"""complex128 results against the oracle in extended precision, beside those of
the double sweeps: random circuits, and ones whose amplitudes are alike (small
angles, one axis, one angle per layer, uniform states), where a rounding that
always goes one way adds up instead of averaging out.  The sweeps in history
and uncompute form and the batched kernel in one CTA and on clusters.

The measure is the rms over a few circuits of the gradient error's norm.  Two
terms bound it:

* four times the double sweeps': both are sums of a few hundred independent
  roundings, two such means scatter by less than two, and a fixed-point
  rounding is the smaller one;
* the fixed step, which does not shrink with a small component: a sweep
  rounds every component of psi and lambda about four times to a unit of at
  most 2^-57 of its tile's norm, 2^-(n-t)/2 of the state's.  Independent
  roundings of rms 0.29 units move an entry Im<lambda|P|psi> by at most
  |lambda| 2^-57 2^(-(n-t)/2) 0.29 sqrt(4 * 4 m) over the m sweeps of the
  circuit, forward and backward (batched kernel: t = n).

(Rounding imaginary parts down on load, and ties up in the right shifts, was
up to a hundred times further off.)"""
import numpy as np
import pytest

from conftest import obs_dict
from oracle import oracle as O
from oracle import quad as Q

pytestmark = pytest.mark.gpu

# kind, n, layers, axis (None: random), largest angle (negative: one per layer), circuits
CASES = [("mc", 10, 10, None, 6.28, 4), ("mc", 14, 10, None, 6.28, 3), ("mc", 14, 20, 0, 0.01, 3),
         ("mc", 14, 20, 1, 0.01, 3), ("mc", 14, 20, None, 0.01, 3), ("mc", 9, 20, 0, 0.01, 3),
         ("mc", 14, 10, 0, -0.01, 3), ("mc", 14, 10, 0, -3.0, 3), ("mc", 10, 40, None, 0.01, 3),
         ("mc", 16, 6, 0, 0.01, 2), ("qa", 10, 3, None, 3.14, 4), ("qa", 14, 4, None, 3.14, 3),
         ("qa", 14, 10, None, 0.01, 3), ("qa", 13, 6, None, 0.3, 3), ("qa", 16, 10, None, 0.01, 2)]


def _inputs(case, seed):
    kind, n, L, axis, scale, _ = case
    rng = np.random.default_rng([n, L, seed, int(abs(scale) * 100), 0 if axis is None else axis + 1])
    if kind == "mc":
        axes = rng.integers(0, 3, (L, n)) if axis is None else np.full((L, n), axis)
        angles = rng.uniform(0, scale, (L, n)) if scale > 0 else np.repeat(rng.uniform(0, -scale, (L, 1)), n, 1)
        return axes, angles, O.Terms([3] * (n - 1), list(range(n - 1)), list(range(1, n)), [1.0] * (n - 1))
    e = {(i, (i + 1) % n) for i in range(n)} | ({(i, i + n // 2) for i in range(n // 2)} if n % 2 == 0 else set())
    e = sorted((min(a, b), max(a, b)) for a, b in e)
    return (rng.uniform(0, scale, L), rng.uniform(0, scale, L),
            O.Terms([3] * len(e), [a for a, _ in e], [b for _, b in e], [1.0] * len(e)))


class _Errors:
    """Per form of the gradient: error norms and the step's share, per circuit."""

    def __init__(self):
        self.e, self.s = {}, {}

    def note(self, name, g, g0, step=0.0):
        d = (np.asarray(g).reshape(g0.shape) - g0).astype(np.longdouble)
        self.e.setdefault(name, []).append(float(np.sqrt(np.sum(d * d))))
        self.s.setdefault(name, []).append(step * np.sqrt(g0.size))

    def check(self):
        rms = lambda v: float(np.sqrt(np.mean(np.square(v))))  # noqa: E731
        for name, e in self.e.items():
            assert rms(e) <= 4 * rms(self.e["double"]) + rms(self.s[name]), (name, self.e, self.s)


def _step(lam, n, t, sweeps):
    return lam * 2.0 ** (-57 - (n - t) / 2) * 0.29 * np.sqrt(16 * sweeps)


def _circuit(case, a, b, t, mode, flags):
    """A circuit of the case's kind and the arguments of its grad_run."""
    from qradient_gb300 import McClean, Qaoa

    kind, n, L = case[:3]
    od = obs_dict(n, t.kind, t.q0, t.q1, t.w)
    c = McClean(n, od, L, axes=a, angles=b, grad_mode=mode) if kind == "mc" else Qaoa(n, od, L, grad_mode=mode)
    c.set_tuning(0, 0, flags)
    return c, () if kind == "mc" else (a, b)


def _exact(case, a, b, t):
    """Gradient and |O psi| from the extended oracle."""
    kind, n = case[:2]
    oracle = Q.mcclean if kind == "mc" else Q.qaoa
    x = np.arange(2 ** n)
    diag = sum(1 - 2.0 * (((x >> (n - 1 - i)) ^ (x >> (n - 1 - j))) & 1) for i, j in zip(t.q0, t.q1))
    state = abs(oracle(n, a, b, t, grad=False)[1])
    return oracle(n, a, b, t)[1], float(np.sqrt(np.sum((diag * state) ** 2)))


@pytest.mark.parametrize("case", [c for c in CASES if c[1] <= 14], ids=lambda c: "-".join(map(str, c[:5])))
def test_batched_gradient_error(case):
    from qradient_gb300 import _lib
    from qradient_gb300.batched import Batch

    kind, n, L, _, _, count = case
    errors = _Errors()
    for seed in range(count):
        a, b, t = _inputs(case, seed)
        g0, lam = _exact(case, a, b, t)
        c, args = _circuit(case, a, b, t, "history", _lib.QG_TUNE_FWD_PLAIN)
        errors.note("double", c.grad_run(*args)[1], g0)
        for first in (13, 11):
            batch = Batch(dtype="complex128", use_graph=False, cluster_from=first)
            batch.add(c, params=(b if kind == "mc" else np.stack([a, b], 1)).reshape(-1))
            errors.note("batch from %d" % first, batch.grad()[1][0].cpu().numpy(), g0, _step(lam, n, n, L))
    errors.check()


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(map(str, c[:5])))
def test_sweep_gradient_error(case):
    from qradient_gb300 import _lib, tuning

    n, L, count = case[1], case[2], case[5]
    errors = _Errors()
    for seed in range(count):
        a, b, t = _inputs(case, seed)
        g0, lam = _exact(case, a, b, t)
        for name, mode, op, flags in (("double", "history", _lib.QG_OP_GRAD_HISTORY, _lib.QG_TUNE_FWD_PLAIN),
                                      ("history", "history", _lib.QG_OP_GRAD_HISTORY, 0),
                                      ("uncompute", "uncompute", _lib.QG_OP_GRAD_UNCOMPUTE, 0)):
            c, args = _circuit(case, a, b, t, mode, flags)
            plan = tuning.get_plan(c.native(), c._dtype_code, op)
            assert plan["fixed_point"] == (name != "double")
            errors.note(name, c.grad_run(*args)[1], g0,
                        _step(lam, n, max(t for t, _ in plan["sweeps"]), L * len(plan["sweeps"])))
    errors.check()
