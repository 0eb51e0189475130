"""The tuning cache on disk: a choice is applied only by the kernels that it was
timed with, and per gradient mode."""
import json

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _circ(n, mode, dtype="complex128"):
    from qradient_gb300 import McClean

    zz = np.full((n, n), None)
    zz[0, 1] = 1.0
    rng = np.random.default_rng(n)
    return McClean(n, {"zz": zz}, 6, axes=rng.integers(0, 3, (6, n)), angles=rng.uniform(0, 6, (6, n)), dtype=dtype,
                   grad_mode=mode)


@pytest.fixture
def cache(tmp_path, monkeypatch):
    p = tmp_path / "tune.json"
    monkeypatch.setenv("QG_TUNING_CACHE", str(p))
    return p


def _forget(tuning, p):
    tuning._MEM.pop(str(p), None)


def test_choice_of_other_kernels_is_not_applied(cache, monkeypatch):
    from qradient_gb300 import _lib, tuning

    tuning.tune_circuit(_circ(9, "history"), reps=1)
    now = json.load(open(cache))
    (key,) = now
    stale = {"tile_bits": 6, "ctas_per_sm": 1, "flags": _lib.QG_TUNE_FWD_PLAIN, "ms": 0.1, "timings": []}
    old = {key.replace(tuning.kernel_tag() + "|", ""): stale, key.replace(tuning.kernel_tag(), "k0123456789ab"): stale}
    assert len(old) == 2 and key not in old
    cache.write_text(json.dumps(old))
    _forget(tuning, cache)
    c = _circ(9, "history")
    r = tuning.tune_circuit(c, reps=1)
    assert len(r["timings"]) == len(tuning.sweep_candidates(c._dtype_code, 9))
    assert set(json.load(open(cache))) == set(old) | {key}
    # and with the right tag the entry is
    cache.write_text(json.dumps({key: stale}))
    _forget(tuning, cache)
    c = _circ(9, "history")
    assert tuning.tune_circuit(c) == stale
    assert not tuning.get_plan(c.native(), c._dtype_code, _lib.QG_OP_GRAD_HISTORY)["fixed_point"]


def test_gradient_modes_have_entries_of_their_own(cache):
    from qradient_gb300 import tuning

    for op, mode in (("grad", "history"), ("grad", "uncompute"), ("run", "history"), ("run", "uncompute")):
        tuning.tune_circuit(_circ(8, mode), op=op, reps=1)
    assert sorted(k.rsplit("|", 1)[1] for k in json.load(open(cache))) == ["grad-history", "grad-uncompute", "run"]


def test_batch_entry_of_other_kernels_is_not_applied(cache):
    from qradient_gb300 import tuning
    from qradient_gb300.batched import Batch

    def batch():
        b = Batch(dtype="complex128", use_graph=False)
        for _ in range(4):
            b.add(_circ(12, "auto"))
        b.finalize()
        return b

    tuning.tune_batch(batch(), reps=1)
    (key,) = json.load(open(cache))
    stale = {"cluster_from": 12, "ms": 0.1, "timings": []}
    cache.write_text(json.dumps({key.replace(tuning.kernel_tag() + "|", ""): stale}))
    _forget(tuning, cache)
    assert tuning.tune_batch(batch(), reps=1)["timings"]
    cache.write_text(json.dumps({key: stale}))
    _forget(tuning, cache)
    assert tuning.tune_batch(batch(), reps=1) == stale
