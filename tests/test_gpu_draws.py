"""Basis-state draws against a sequential numpy walk over the same uniforms,
at the edges of the two draw kernels: one amplitude chunk or less (n <= 12),
several chunks, states with long empty stretches, more shots than threads."""
import numpy as np
import pytest

from test_sampling import _u01, philox4x32_10

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(1, 7), (4, 600), (11, 300), (12, 1100), (13, 130), (16, 300)])
@pytest.mark.parametrize("sparse", [False, True])
def test_draws_are_the_inverse_cdf_of_the_stream(n, k, sparse):
    import torch

    from qradient_gb300.circuit_logic.qaoa import sample_state

    rng = np.random.default_rng(n)
    v = rng.normal(size=2 ** n) + 1j * rng.normal(size=2 ** n)
    if sparse and n > 1:  # (at n = 1 nothing would be left of the state)
        v[rng.random(2 ** n) < 0.97] = 0.0
        v[2 ** n // 3] = 1.0
        v[-(2 ** n // 4):] = 0.0
    v /= np.linalg.norm(v)
    got = sample_state(torch.as_tensor(v, device="cuda"), k, seed=99, offset=5).cpu().numpy()
    p = np.abs(v) ** 2
    cdf = np.cumsum(p)
    assert np.all(p[got] > 0.0)
    for s in range(k):
        c = philox4x32_10([s + 5, 0, 0, 0], [99, 0])
        u = _u01(c[0], c[1]) * cdf[-1]
        want = int(np.searchsorted(cdf, u, side="right"))
        # the running sums differ by rounding: n additions of 2^-53 at most
        assert got[s] == want or abs(cdf[min(got[s], want)] - u) <= 2.0 ** (n - 53), (s, got[s], want)
