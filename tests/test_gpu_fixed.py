"""The fixed-point complex128 sweeps (qg_fixed.cu) against the oracle.

One case per sweep layout the default rule takes (single tile, two sweeps of
8..12-bit tiles, three sweeps), every tuned tile size with a remainder, and
the states whose tiles leave the usual range: zero tiles, tiny, huge and
non-finite amplitudes.  Tolerance: the oracle's own double rounding, 1e-12
normwise, as in the other complex128 tests (a tile's fixed-point step is
2^-53 of its norm or less)."""
import numpy as np
import pytest

from conftest import obs_dict, rel_err
from oracle import oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-12
ENT = {"cnot": 1, "cz": 2, "cnot_periodic": 3, None: 0}


def _terms(n):
    kind, q0, q1, w = [3] * (n - 1), list(range(n - 1)), list(range(1, n)), [1.0] * (n - 1)
    for k, q, v in ((0, 0, 0.5), (1, n - 1, -0.25), (2, n // 2, 0.75), (0, n // 2, -1.0)):
        kind.append(k), q0.append(q), q1.append(q), w.append(v)
    return kind, q0, q1, w


def _check(n, L, ent="cnot", place="before", seed=0, axes=None, ini=None, tile=0, scale=1.0):
    from qradient_gb300 import McClean

    rng = np.random.default_rng(100 * n + seed)
    axes = rng.integers(0, 3, (L, n)) if axes is None else np.full((L, n), axes)
    angles = rng.uniform(-2 * np.pi, 4 * np.pi, (L, n))
    kind, q0, q1, w = _terms(n)
    E0, g0 = O.mcclean_grad(n, axes, angles, O.Terms(kind, q0, q1, w), entangler=ENT[ent],
                            placement=1 if place == "after" else 0, ini=ini)
    E0, g0 = E0 * scale ** 2, g0 * scale ** 2
    start = None if ini is None else ini * scale
    for mode in ("history", "uncompute"):
        c = McClean(n, obs_dict(n, np.array(kind), np.array(q0), np.array(q1), np.array(w)), L, axes=axes,
                    angles=angles, entangler=ent, placement=place, grad_mode=mode)
        if tile:
            c.set_tuning(tile, 0, 0)
        E, g = c.grad_run(ini_state=start)
        big = np.max(np.abs(g0))
        assert abs(E - E0) <= TOL * max(scale ** 2, abs(E0)), (n, mode)
        assert np.max(np.abs(g - g0)) <= TOL * max(big, 1e-3 * scale ** 2), (n, mode)
    assert abs(c.run_expec_val(ini_state=start) - E0) <= TOL * max(scale ** 2, abs(E0))


@pytest.mark.parametrize("n", [8, 9, 10, 11, 12, 13, 16, 17, 18, 19, 20, 21, 22])
def test_default_layouts(n):
    _check(n, 3 if n < 18 else 2, ("cnot", "cz", None)[n % 3], ("before", "after")[n % 2])


@pytest.mark.parametrize("tile,n", [(8, 8), (8, 11), (8, 15), (9, 9), (9, 14), (9, 16), (10, 17), (10, 19), (11, 15), (11, 20), (12, 13), (12, 21)])
def test_tuned_tiles(tile, n):
    _check(n, 2, "cnot" if n % 2 else "cnot_periodic", "before", seed=tile, tile=tile)


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_one_axis(axis):
    """Every bit a butterfly level (X, Y), or none (Z)."""
    for n in (8, 9, 11, 12, 13, 19):
        _check(n, 2, "cnot", "after", axes=axis)


@pytest.mark.parametrize("scale", [1.0, 1e-12, 1e-40, 1e-130, 1e12, 1e40, 1e130])
def test_start_state_magnitudes(scale):
    """Random and basis states from tiny to huge: the squares leave single
    precision's range from about 1e-9 and 1e15 on."""
    rng = np.random.default_rng(3)
    for n in (10, 13):
        v = rng.normal(size=2 ** n) + 1j * rng.normal(size=2 ** n)
        _check(n, 2, ini=v / np.linalg.norm(v), scale=scale)
        b = np.zeros(2 ** n, dtype=complex)
        b[5] = 1j
        _check(n, 1, ini=b, scale=scale)


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_non_finite_inputs_stay_visible(bad):
    from qradient_gb300 import McClean

    n, L = 13, 2
    rng = np.random.default_rng(1)
    axes, angles = rng.integers(0, 2, (L, n)), rng.uniform(0, 6, (L, n))
    zz = np.full((n, n), None)
    zz[0, 1] = 1.0
    c = McClean(n, {"zz": zz}, L, axes=axes, angles=angles)
    v = np.full(2 ** n, 2.0 ** (-n / 2), dtype=complex)
    v[77] = bad
    E, g = c.grad_run(ini_state=v)
    assert np.isnan(E) and np.all(np.isnan(g))
    angles = angles.copy()
    angles[1, 3] = bad
    c.angles = angles
    E, g = c.grad_run()
    assert np.isnan(E) and np.all(np.isnan(g))


def test_qaoa_layouts_and_start_state():
    from qradient_gb300 import Qaoa
    from qradient_gb300.optimization_problems import MaxCut, random_regular_edges

    for n, p, mode in ((10, 1, "history"), (12, 3, "uncompute"), (14, 2, "history"), (18, 2, "uncompute"),
                       (20, 2, "history"), (22, 1, "uncompute")):
        rng = np.random.default_rng(n)
        edges = random_regular_edges(3, n, n)
        betas, gammas = rng.uniform(-1, 4, p), rng.uniform(-1, 4, p)
        t = O.Terms([3] * len(edges), edges[:, 0], edges[:, 1], [1.0] * len(edges))
        q = Qaoa(n, MaxCut(n, edge_set=edges).to_observable(), p, grad_mode=mode)
        E0, g0 = O.qaoa_grad(n, betas, gammas, t)
        E, g = q.grad_run(betas, gammas)
        assert abs(E - E0) <= TOL * max(1.0, abs(E0)) and rel_err(g, g0) <= TOL, (n, mode)
        assert abs(q.run_expec_val(betas, gammas) - E0) <= TOL * max(1.0, abs(E0))
