"""Waits that run out in the FP32 same-spin products: a call either reports PQ_TIMEOUT or has the numbers of an undisturbed
one (within the order of the atomic sums of its other kernels), so no warp goes on where some of its lanes have given up,
and the next call is correct."""
import ctypes

import pytest

from cases import synthetic_fci
from test_gpu_sigma_path import _make

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SIGMA_RTOL_FP32 = 2e-5


@pytest.mark.parametrize("n,a,b", [(11, 5, 5), (12, 6, 6), (13, 6, 5)])
def test_timeout_or_the_same_numbers(n, a, b):
    from polyquant_gb300 import _lib

    L = _lib.load()
    g = _make(synthetic_fci(n, a, b, seed=n))
    X = torch.randn(4, g.N_dets, device="cuda", dtype=torch.float64).t()
    S64 = g.sigma(X)
    bound = SIGMA_RTOL_FP32 * S64.abs().max()
    try:
        for budget in (1, 100, 300, 700, 1000, 2000, 3000, 5000, 10000, 30000, 100000):
            L.pq_debug_set_sigma_wait_budget(ctypes.c_longlong(budget), ctypes.c_longlong(0))
            try:
                S = g.sigma(X, precision=_lib.PQ_FP32)
            except _lib.PQError as e:
                assert e.status == _lib.PQ_TIMEOUT
            else:
                assert budget > 1 and (S - S64).abs().max() <= bound
    finally:
        L.pq_debug_set_sigma_wait_budget(0, 0)
    assert (g.sigma(X, precision=_lib.PQ_FP32) - S64).abs().max() <= bound
    g.close()
