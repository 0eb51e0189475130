"""bench.py's count of the library's own kernels in a grad_run against the
profiler's list of what was launched."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dtype", [(9, "complex128"), (13, "complex128"), (6, "complex128"), (13, "complex64")])
def test_count_matches_the_profiler(n, dtype):
    import ctypes

    import torch
    from torch.profiler import ProfilerActivity, profile

    import bench
    from qradient_gb300 import McClean, _lib, tuning

    lib, steps, L = _lib.load(), 3, 4
    zz = np.full((n, n), None)
    zz[0, 1] = 1.0
    c = McClean(n, {"zz": zz}, L, axes=np.zeros((L, n), dtype=int), angles=np.zeros((L, n)), dtype=dtype,
                grad_mode="history")
    a = torch.zeros(L * n, dtype=torch.float64, device="cuda")
    c.grad_run_tensors(a)
    torch.cuda.synchronize()
    for _ in range(2):  # (a process's first profile may come back without kernels)
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            for _ in range(steps):
                c.grad_run_tensors(a)
            torch.cuda.synchronize()
    seen = sum(e.count for e in prof.key_averages() if "qg::" in e.key)
    if not seen:
        pytest.skip("the profiler lists no kernels here")
    lib.qg_profile_enable(1)
    for _ in range(steps):
        c.grad_run_tensors(a)
    torch.cuda.synchronize()
    counted = 0
    for cls in (0, 1, 2):
        ms, cnt = ctypes.c_double(0), ctypes.c_int(0)
        _lib.check(lib.qg_profile_collect(cls, ctypes.byref(ms), ctypes.byref(cnt)))
        counted += cnt.value
    lib.qg_profile_enable(0)
    plan = tuning.get_plan(c.native(), c._dtype_code, _lib.QG_OP_GRAD_HISTORY)
    assert bench.own_launches(steps, counted, plan["fixed_point"]) == seen
