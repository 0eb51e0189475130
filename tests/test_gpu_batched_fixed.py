"""The fixed-point complex128 batched kernel (qg_batched_fix.cu) against the
oracle at its edges: every block size padded and full, clusters, the split
bits with and without rotations on them, layers of one axis (norm growth and
none), runs of layers longer than one fill of the angle table, observables of
extreme weight, non-finite angles.  1e-12 normwise, as the other complex128
tests."""
import ctypes

import numpy as np
import pytest

from conftest import obs_dict, rel_err
from oracle import oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-12
ENT = {"cnot": 1, "cz": 2, "cnot_periodic": 3, None: 0}


def _case(n, L, ent, place, seed, axes=None, wscale=1.0):
    from qradient_gb300 import McClean

    rng = np.random.default_rng(seed)
    axes = rng.integers(0, 3, (L, n)) if axes is None else np.full((L, n), axes)
    angles = rng.uniform(-7, 7, (L, n))
    kind, q0, q1, w = [3, 2, 0, 1], [0, 0, n - 1, 0], [1, 0, n - 1, 0], [1.0, 0.5, -0.75, 0.25]
    w = [wscale * x for x in w]
    c = McClean(n, obs_dict(n, np.array(kind), np.array(q0), np.array(q1), np.array(w)), L, axes=axes, angles=angles,
                entangler=ent, placement=place)
    E0, g0 = O.mcclean_grad(n, axes, angles, O.Terms(kind, q0, q1, w), entangler=ENT[ent],
                            placement=1 if place == "after" else 0)
    return c, E0, g0


def _run(cases, **kw):
    from qradient_gb300.batched import Batch

    b = Batch(dtype="complex128", **kw)
    for c, _, _ in cases:
        b.add(c)
    E, G = b.grad()
    E = E.cpu().numpy()
    for k, (c, E0, g0) in enumerate(cases):
        scale = max(abs(E0), np.max(np.abs(g0)), 1e-300)
        assert abs(E[k] - E0) <= TOL * scale, (k, c.qnum)
        assert np.max(np.abs(G[k].cpu().numpy().reshape(g0.shape) - g0)) <= TOL * scale, (k, c.qnum)


@pytest.mark.parametrize("cluster_from", [13, 11, 5])
def test_all_sizes_and_clusters(cluster_from):
    cases = []
    for n in range(2, 15):
        ent = ("cnot", "cz", None, "cnot_periodic")[n % 4]
        if ent == "cnot_periodic" and n % 2:
            ent = "cnot"
        cases.append(_case(n, 3, ent, ("before", "after")[n % 2], n))
        cases.append(_case(n, 2, "cnot", ("after", "before")[n % 2], 50 + n))
    _run(cases, cluster_from=cluster_from)


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_layers_of_one_axis(axis):
    """n rotation levels per layer (right shifts), or none (left shifts)."""
    _run([_case(n, 12, "cnot", "before", n, axes=axis) for n in (4, 9, 10, 11, 12, 13, 14)])


def test_long_circuits_refill_the_angles():
    _run([_case(3, 400, "cnot", "before", 1), _case(12, 60, "cz", "after", 2), _case(14, 45, "cnot", "after", 3),
          _case(9, 120, "cnot", "before", 4)])


@pytest.mark.parametrize("wscale", [1e-200, 1e-20, 1e20, 1e200])
def test_extreme_weights(wscale):
    _run([_case(n, 3, "cnot", "before", n, wscale=wscale) for n in (6, 12, 13, 14)])


def test_non_finite_angles_give_nan_for_their_job_only():
    from qradient_gb300.batched import Batch

    cases = [_case(n, 3, "cnot", "before", n) for n in (8, 12, 13, 14)]
    for bad in range(len(cases)):
        b = Batch(dtype="complex128", use_graph=False)
        for k, (c, _, _) in enumerate(cases):
            a = np.array(c.angles)
            if k == bad:
                a[1, 2] = np.nan if bad % 2 else np.inf
            b.add(c, params=a)
        E, G = b.grad()
        for k, (c, E0, g0) in enumerate(cases):
            g = G[k].cpu().numpy()
            if k == bad:
                assert np.isnan(float(E[k])) and np.all(np.isnan(g))
            else:
                assert rel_err(g.reshape(g0.shape), g0) <= TOL


def test_small_jobs_in_a_launch_of_large_blocks():
    """qg_batch_launch with max_qubits above the jobs' sizes: padded blocks."""
    import torch

    from qradient_gb300 import _lib, _native
    from qradient_gb300.batched import Batch

    cases = [_case(n, 4, "cnot", "before", n) for n in (3, 7, 9)]
    b = Batch(dtype="complex128", use_graph=False)
    for c, _, _ in cases:
        b.add(c)
    b.finalize()
    for maxq, cluster in ((12, 1), (11, 1), (13, 2), (14, 4)):
        for cl, jobs, nj, _, ws in b._groups:
            b.grads_flat.zero_()
            _lib.check(_lib.load().qg_batch_launch(0, _native.ptr(jobs), nj, maxq, cluster, _native.ptr(ws), ws.numel(),
                                                   _native.stream_handle(b.device)))
        torch.cuda.synchronize()
        for k, (c, E0, g0) in enumerate(cases):
            if cluster == 4 and c.qnum < 4:
                continue
            assert abs(float(b.expec[k]) - E0) <= TOL
            assert rel_err(b.grads[k].cpu().numpy().reshape(g0.shape), g0) <= TOL, (maxq, cluster, c.qnum)
