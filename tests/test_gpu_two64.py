"""FP64 sigma of small two-species product spaces by pair matrices on the tensor cores (ci_two64.cu) against the
element kernel (PQ_SIGMA64_GATHER, read when a handle is created) and the oracle: two to four lists of more than one
string, unrestricted spins, partly filled tiles and chunks, split and whole K ranges, caller-chosen strings, non-finite
input.  The element kernel's rounding of some 10^3 terms: 1e-13 of the column's largest value."""
import ctypes

import numpy as np
import pytest

import oracle as O
from cases import synthetic_en, synthetic_ep

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-13


@pytest.fixture(autouse=True)
def every_size(monkeypatch):
    """Small spaces too: the size rule keeps them on the element kernel otherwise."""
    monkeypatch.setenv("PQ_TWO64_ALWAYS", "1")


def _pair(monkeypatch, p, **kw):
    from polyquant_gb300.detset import POLYQUANT_DETSET

    def make():
        return POLYQUANT_DETSET(p.n_orb, p.n_alpha, p.n_beta, p.h1, p.eri, p.ex_level, restricted=p.restricted,
                                charge=p.charge, max_collective_excitation_level=p.max_collective, **kw)

    g = make()
    monkeypatch.setenv("PQ_SIGMA64_GATHER", "1")
    r = make()
    monkeypatch.delenv("PQ_SIGMA64_GATHER")
    return g, r


def _check(g, r, X):
    S, R = g.sigma(X), r.sigma(X)
    assert ((S - R).abs().amax(0) <= TOL * R.abs().amax(0)).all()


@pytest.mark.parametrize("args", [(5, 1, 0, 4, 1, 0), (12, 1, 1, 7, 1, 0), (33, 1, 1, 9, 1, 0), (6, 2, 1, 5, 1, 1),
                                  (6, 2, 2, 4, 1, 1), (8, 2, 2, 6, 1, 0), (60, 1, 1, 40, 1, 0), (40, 1, 0, 40, 1, 1)])
def test_against_the_element_kernel(monkeypatch, args):
    p = synthetic_ep(*args, seed=sum(args))
    g, r = _pair(monkeypatch, p)
    gen = torch.Generator(device="cuda").manual_seed(1)
    for k in (1, 2, 3, 4, 6):
        X = torch.randn(k, g.N_dets, device="cuda", dtype=torch.float64, generator=gen).t()
        _check(g, r, X)
    f = torch.tensor([1e-150, 1.0, 1e100, 1e-5], device="cuda", dtype=torch.float64)
    _check(g, r, X[:, :4] * f)
    _check(g, r, X[:, :2] * torch.pow(10.0, -12.0 * torch.rand(g.N_dets, 1, device="cuda", dtype=torch.float64)))
    H = X[:, :2].cpu().numpy()
    want = r.sigma(X[:, :2]).cpu().numpy()
    assert np.abs(g.sigma(H) - want).max() <= TOL * np.abs(want).max()


@pytest.mark.parametrize("make", [lambda: synthetic_ep(6, 2, 1, 5, 1, 1, seed=4), lambda: synthetic_en(6, 2, 1, 5, 1, 1, seed=5),
                                  lambda: synthetic_ep(6, 2, 2, 5, 1, 0, seed=6, max_coll=2)])
def test_against_the_oracle(monkeypatch, make):
    p = make()
    g, r = _pair(monkeypatch, p)
    ref = O.Detset(p)
    X = np.random.default_rng(1).standard_normal((g.N_dets, 3))
    want = ref.sigma(X)
    S = g.sigma(torch.from_numpy(X).cuda()).cpu().numpy()
    assert np.abs(S - want).max() <= TOL * np.abs(want).max()


def test_selected_strings_shift_and_non_finite(monkeypatch):
    from polyquant_gb300 import _lib

    p = synthetic_ep(9, 2, 2, 7, 1, 0, seed=8)
    rng = np.random.default_rng(3)
    pairs = np.array([(1 << i) | (1 << j) for i in range(9) for j in range(i)], dtype=np.uint64)
    lists = [[rng.permutation(pairs)[:20], rng.permutation(pairs)[:11]], [np.array([1, 4, 16, 64], dtype=np.uint64),
                                                                         np.array([0], dtype=np.uint64)]]
    g, r = _pair(monkeypatch, p, selected_strings=lists)
    assert g.N_dets == 880
    X = torch.randn(3, 880, device="cuda", dtype=torch.float64).t()
    _check(g, r, X)
    L = _lib.load()
    for k in (1, 2, 3, 4):
        Z = torch.randn(880, k, device="cuda", dtype=torch.float64)
        out = []
        for h in (g, r):
            Y = torch.empty_like(Z)
            assert L.pq_ci_sigma_interleaved(h._h, ctypes.c_void_p(Z.data_ptr()), ctypes.c_void_p(Y.data_ptr()), k,
                                             _lib.PQ_FP64, ctypes.c_double(2.5)) == _lib.PQ_OK
            torch.cuda.synchronize()
            out.append(Y)
        assert ((out[0] - out[1]).abs().amax(0) <= TOL * out[1].abs().amax(0)).all()
    x = X[:, 0].clone()
    x[5] = float("nan")
    S, R = g.sigma(x), r.sigma(x)
    assert torch.equal(torch.isnan(S), torch.isnan(R)) and torch.equal(S.nan_to_num(), R.nan_to_num())
