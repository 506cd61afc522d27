"""Waits that run out in the FP64 tensor-core sigma: every role gives up within its budget, the gate tells, the element
kernel behind computes the result, and the next call on the same handle is the digit products' again.  A budget of one
cycle stops a kernel at its first pending wait, longer ones at some later point (or not at all, where the pipeline is
faster), so that CTAs start while others of the launch have already raised the gate."""
import ctypes

import pytest

from cases import synthetic_ep, synthetic_fci
from test_gpu_sigma_path import _make, path

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-13


def _expire(monkeypatch, p, budgets):
    from polyquant_gb300 import _lib

    L = _lib.load()
    g = _make(p)
    monkeypatch.setenv("PQ_SIGMA64_GATHER", "1")
    r = _make(p)
    monkeypatch.delenv("PQ_SIGMA64_GATHER")
    X = torch.randn(3, g.N_dets, device="cuda", dtype=torch.float64).t()
    R = r.sigma(X)
    scale = TOL * R.abs().amax(0)
    try:
        for same, opposite in budgets:
            L.pq_debug_set_sigma_wait_budget(ctypes.c_longlong(same), ctypes.c_longlong(opposite))
            S = g.sigma(X)
            where, gate = path(g)
            assert where == _lib.PQ_PATH_TENSOR and gate in (0, 2)
            assert gate == 2 or (same, opposite) not in ((1, 0), (0, 1))
            assert ((S - R).abs().amax(0) <= scale).all()
    finally:
        L.pq_debug_set_sigma_wait_budget(0, 0)
    S = g.sigma(X)
    assert path(g) == (_lib.PQ_PATH_TENSOR, 0)
    assert ((S - R).abs().amax(0) <= scale).all()
    g.close()
    r.close()


def test_pair_matrices(monkeypatch):
    _expire(monkeypatch, synthetic_ep(60, 1, 1, 40, 1, 0, seed=1), [(b, 0) for b in (1, 300, 1000, 3000, 10000, 30000)])


def test_same_spin_products(monkeypatch):
    _expire(monkeypatch, synthetic_fci(12, 6, 6, seed=2), [(b, 0) for b in (1, 300, 1000, 3000, 10000, 30000)])


@pytest.mark.parametrize("n,a,b", [(12, 6, 6), (12, 6, 3), (13, 8, 2), (17, 2, 4)])
def test_opposite_spin_kernel(monkeypatch, n, a, b):
    """Its three gather warps give up at different stages: the gathers that some have issued and others have not are
    waited for before the CTA leaves."""
    _expire(monkeypatch, synthetic_fci(n, a, b, seed=3), [(0, w) for w in (1, 100, 300, 700, 1000, 2000, 3000, 10000, 30000)])
