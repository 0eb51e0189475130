"""The streams of a batch's launch groups: the same ones in every launch,
held by one batch at a time, none of them from torch's pool (where a server's
request streams and a user's come from), returned when the batch goes."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(dtype, sizes, **kw):
    from qradient_gb300 import McClean
    from qradient_gb300.batched import Batch

    b = Batch(dtype=dtype, use_graph=False, **kw)
    for n in sizes:
        zz = np.full((n, n), None)
        zz[0, 1] = 1.0
        rng = np.random.default_rng(n)
        b.add(McClean(n, {"zz": zz}, 2, axes=rng.integers(0, 3, (2, n)), angles=rng.uniform(0, 6, (2, n)), dtype=dtype))
    b.finalize()
    return b


def _handles(monkeypatch, call):
    """Handles of the streams that the batch launches of `call` go to."""
    from qradient_gb300 import _native

    seen, orig = [], _native.stream_handle

    def record(device):
        h = orig(device)
        seen.append(h.value or 0)
        return h

    monkeypatch.setattr(_native, "stream_handle", record)
    call()
    monkeypatch.setattr(_native, "stream_handle", orig)
    return seen


def _pool():
    import torch

    return {torch.cuda.Stream().cuda_stream for _ in range(64)}


@pytest.mark.parametrize("dtype,sizes", [("complex128", (8, 10, 11, 12, 13, 14)), ("complex64", (9, 14, 15))])
def test_groups_keep_their_streams(monkeypatch, dtype, sizes):
    import torch

    pool, main = _pool(), torch.cuda.Stream()
    a, b = _batch(dtype, sizes), _batch(dtype, sizes)
    used = {}
    with torch.cuda.stream(main):
        for name, x in (("a", a), ("b", b), ("a", a), ("b", b)):
            for _ in range(20):
                h = _handles(monkeypatch, x.execute)
                assert len(set(h)) == len(h) == len(sizes)
                assert used.setdefault(name, h) == h
                assert main.cuda_stream in h and not (set(h) - {main.cuda_stream}) & pool
    assert set(used["a"]) & set(used["b"]) == {main.cuda_stream}
    torch.cuda.synchronize()


def test_streams_are_returned_and_bounded(monkeypatch):
    import torch

    from qradient_gb300 import batched

    first = set()
    for _ in range(50):
        b = _batch("complex128", (8, 10, 11, 12))
        first |= {st.cuda_stream for st in b._side}
        b.execute()
        torch.cuda.synchronize()
        del b
        gc.collect()
    assert len(first) <= 20  # reused, not made anew for every batch
    many = [_batch("complex128", (8, 10, 11, 12)) for _ in range(20)]
    assert len({st.cuda_stream for b in many for st in b._side}) == 60
    del many
    gc.collect()
    keep = _batch("complex128", (8, 10))
    assert all(len(f) <= batched._SideStreams.KEEP for f in batched._side_streams._free.values())
    keep.execute()
    torch.cuda.synchronize()


def test_launch_that_raises_leaves_the_streams_joined(monkeypatch):
    """A group's launch raises after others went out: the current stream still
    waits for them, and the batch runs again."""
    import torch

    from qradient_gb300 import _lib

    b = _batch("complex128", (8, 10, 11, 12))
    E0 = b.execute()[0].cpu().numpy().copy()
    orig, calls = _lib.check, []

    def check(status):
        calls.append(status)
        if len(calls) == 3:
            raise RuntimeError("injected")
        return orig(status)

    monkeypatch.setattr(_lib, "check", check)
    with pytest.raises(RuntimeError, match="injected"):
        b.execute()
    monkeypatch.setattr(_lib, "check", orig)
    torch.cuda.current_stream().synchronize()
    assert all(st.query() for st in b._side)
    assert np.array_equal(b.execute()[0].cpu().numpy(), E0)
