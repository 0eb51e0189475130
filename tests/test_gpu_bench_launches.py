"""bench.py's count of the library's own kernels in a grad_run against the
kernel nodes of the call captured in a CUDA graph."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _kernel_nodes(graph):
    drv, P = ctypes.CDLL("libcuda.so.1"), ctypes.c_void_p
    count = ctypes.c_size_t()
    assert drv.cuGraphGetNodes(P(graph), None, ctypes.byref(count)) == 0
    nodes = (P * count.value)()
    assert drv.cuGraphGetNodes(P(graph), nodes, ctypes.byref(count)) == 0
    kernels, kind = 0, ctypes.c_int()
    for node in nodes:
        assert drv.cuGraphNodeGetType(P(node), ctypes.byref(kind)) == 0
        kernels += kind.value == 0  # CU_GRAPH_NODE_TYPE_KERNEL
    return kernels


@pytest.mark.parametrize("n,dtype", [(9, "complex128"), (13, "complex128"), (6, "complex128"), (13, "complex64")])
def test_count_matches_the_graph(n, dtype):
    import torch

    import bench
    from qradient_gb300 import McClean, _lib, tuning

    lib, steps, L = _lib.load(), 3, 4
    zz = np.full((n, n), None)
    zz[0, 1] = 1.0
    c = McClean(n, {"zz": zz}, L, axes=np.zeros((L, n), dtype=int), angles=np.zeros((L, n)), dtype=dtype,
                grad_mode="history")
    a = torch.zeros(L * n, dtype=torch.float64, device="cuda")
    out = (torch.empty(1, dtype=torch.float64, device="cuda"), torch.empty(L * n, dtype=torch.float64, device="cuda"))
    c.grad_run_tensors(a, out=out)
    torch.cuda.synchronize()
    try:
        g = torch.cuda.CUDAGraph(keep_graph=True)
    except TypeError:
        pytest.skip("this torch keeps no captured graph")
    with torch.cuda.graph(g):
        for _ in range(steps):
            c.grad_run_tensors(a, out=out)
    seen = _kernel_nodes(g.raw_cuda_graph())
    lib.qg_profile_enable(1)
    for _ in range(steps):
        c.grad_run_tensors(a, out=out)
    torch.cuda.synchronize()
    counted = 0
    for cls in (0, 1, 2):
        ms, cnt = ctypes.c_double(0), ctypes.c_int(0)
        _lib.check(lib.qg_profile_collect(cls, ctypes.byref(ms), ctypes.byref(cnt)))
        counted += cnt.value
    lib.qg_profile_enable(0)
    plan = tuning.get_plan(c.native(), c._dtype_code, _lib.QG_OP_GRAD_HISTORY)
    assert bench.own_launches(steps, counted, plan["fixed_point"]) == seen
