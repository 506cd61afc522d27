"""FP64 full-CI sigma by digit products on the tensor cores (ci_sigma64.cu) against the element-by-element kernel
(PQ_SIGMA64_GATHER, read when a handle is created): tiles that are partly filled in either string list, one to three
pair passes, unequal and unrestricted spins, caller-chosen string lists, every number of columns, columns of very
different size, and non-finite input.  The reference rounds some 10^3 terms at 2^-53 of the diagonal term: 1e-13 of
the column's largest value."""
import ctypes

import numpy as np
import pytest

import oracle as O
from cases import synthetic_fci, synthetic_unrestricted

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-13


def _pair(monkeypatch, p, **kw):
    from polyquant_gb300.detset import POLYQUANT_DETSET

    def make():
        return POLYQUANT_DETSET(p.n_orb, p.n_alpha, p.n_beta, p.h1, p.eri, p.ex_level, restricted=p.restricted,
                                charge=p.charge, **kw)

    g = make()
    monkeypatch.setenv("PQ_SIGMA64_GATHER", "1")
    r = make()
    monkeypatch.delenv("PQ_SIGMA64_GATHER")
    return g, r


def _check(g, r, X):
    S, R = g.sigma(X), r.sigma(X)
    assert ((S - R).abs().amax(0) <= TOL * R.abs().amax(0)).all()


@pytest.mark.parametrize("n,a,b,restricted", [(10, 5, 5, True), (11, 5, 4, True), (12, 6, 3, True), (13, 2, 8, True),
                                             (13, 8, 2, True), (15, 3, 3, True), (17, 2, 4, True), (10, 4, 6, False),
                                             (11, 5, 5, False)])
def test_against_the_element_kernel(monkeypatch, n, a, b, restricted):
    p = synthetic_fci(n, a, b, seed=90 + n) if restricted else synthetic_unrestricted(n, a, b, seed=91)
    g, r = _pair(monkeypatch, p)
    gen = torch.Generator(device="cuda").manual_seed(n)
    for k in (1, 2, 3, 4, 5):
        X = torch.randn(k, g.N_dets, device="cuda", dtype=torch.float64, generator=gen).t()
        _check(g, r, X)
    # columns of different size, and entries that spread over decades
    f = torch.tensor([1e-150, 1.0, 1e100, 1e-5], device="cuda", dtype=torch.float64)
    _check(g, r, X[:, :4] * f)
    _check(g, r, X[:, :2] * torch.pow(10.0, -12.0 * torch.rand(g.N_dets, 1, device="cuda", dtype=torch.float64)))
    _check(g, r, torch.ones_like(X[:, :1]))
    assert not g.sigma(torch.zeros_like(X[:, :2])).any().item()
    # host buffers, pinned (in place) and pageable
    H = X[:, :2].cpu()
    want = r.sigma(X[:, :2]).cpu().numpy()
    assert np.abs(g.sigma(H.numpy()) - want).max() <= TOL * np.abs(want).max()
    g.close()
    r.close()


def test_rows_against_the_oracle(monkeypatch):
    p = synthetic_fci(11, 5, 5, seed=99)
    g, r = _pair(monkeypatch, p)
    X = np.random.default_rng(1).standard_normal((g.N_dets, 2))
    rows = np.random.default_rng(2).choice(g.N_dets, size=500, replace=False)
    ref = O.Detset(p, check_addressing=False).sigma_rows(X, rows)
    S = g.sigma(torch.from_numpy(X).cuda()).cpu().numpy()[rows]
    assert np.abs(S - ref).max() <= TOL * np.abs(ref).max()


def test_unit_vector_and_selected_strings(monkeypatch):
    from itertools import combinations

    p = synthetic_fci(12, 4, 4, seed=98)
    rng = np.random.default_rng(3)
    strings = np.array([sum(1 << o for o in c) for c in combinations(range(12), 4)], dtype=np.uint64)
    lists = [rng.permutation(strings)[:300], rng.permutation(strings)[:150]]
    g, r = _pair(monkeypatch, p, selected_strings=[lists])
    assert g.N_dets == 45000
    X = torch.randn(3, g.N_dets, device="cuda", dtype=torch.float64).t()
    _check(g, r, X)
    e = torch.zeros(g.N_dets, device="cuda", dtype=torch.float64)
    e[12345] = 1.0
    S = g.sigma(e).cpu().numpy()
    I = rng.choice(g.N_dets, 200)
    assert np.abs(S[I] - g.elements(I, np.full(200, 12345))).max() <= 1e-13 * np.abs(S).max()


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_non_finite_input_takes_the_element_kernel(monkeypatch, bad):
    p = synthetic_fci(10, 5, 5, seed=97)
    g, r = _pair(monkeypatch, p)
    X = torch.randn(g.N_dets, device="cuda", dtype=torch.float64)
    X[777] = bad
    S, R = g.sigma(X), r.sigma(X)
    assert torch.equal(torch.isnan(S), torch.isnan(R)) and torch.equal(S.nan_to_num(), R.nan_to_num())
    _check(g, r, torch.randn(2, g.N_dets, device="cuda", dtype=torch.float64).t())


def test_overlapping_buffers(monkeypatch):
    from polyquant_gb300 import _lib

    p = synthetic_fci(10, 5, 5, seed=96)
    g, r = _pair(monkeypatch, p)
    X = torch.randn(2, g.N_dets, device="cuda", dtype=torch.float64)
    want = r.sigma(X.t())
    st = _lib.load().pq_ci_sigma(g._h, ctypes.c_void_p(X.data_ptr()), g.N_dets, 2, ctypes.c_void_p(X.data_ptr()), g.N_dets,
                                 _lib.PQ_FP64)
    torch.cuda.synchronize()
    assert st == _lib.PQ_OK and torch.equal(X.t(), want)


def test_interleaved_vectors_and_shift(monkeypatch):
    """The native-layout entry point: widths 1, 2, 4 with a diagonal shift; three interleaved vectors stay refused."""
    from polyquant_gb300 import _lib

    p = synthetic_fci(10, 5, 5, seed=95)
    g, r = _pair(monkeypatch, p)
    L = _lib.load()
    for k in (1, 2, 3, 4):
        X = torch.randn(g.N_dets, k, device="cuda", dtype=torch.float64)
        out = []
        for h in (g, r):
            Y = torch.empty_like(X)
            st = L.pq_ci_sigma_interleaved(h._h, ctypes.c_void_p(X.data_ptr()), ctypes.c_void_p(Y.data_ptr()), k, _lib.PQ_FP64,
                                           ctypes.c_double(-3.25))
            torch.cuda.synchronize()
            assert st == (_lib.PQ_ERR_ARG if k == 3 else _lib.PQ_OK)
            out.append(Y)
        if k != 3:
            assert ((out[0] - out[1]).abs().amax(0) <= TOL * out[1].abs().amax(0)).all()
            want = r.sigma(X) + 3.25 * X
            assert ((out[0] - want).abs().amax(0) <= TOL * want.abs().amax(0)).all()
