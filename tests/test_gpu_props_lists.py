"""<S^2> and the 1-RDM of one-species spaces from the lists by orbital pair, where their tiles and limits can go wrong:
rows of unequal length, unequal spins, an empty spin, more states than one pass, row tiles of every size.  Sums of
at most 1e6 FP64 terms of unit vectors against the oracle: 1e-12 (the oracle drops products below 1e-16, up to 1e-13
in all)."""
import numpy as np
import pytest

import oracle as O
from cases import synthetic_fci

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,a,b,ex", [(6, 1, 0, [1, 0, 1]), (7, 4, 2, [3, 2, 5]), (9, 4, 3, [2, 2, 2]), (10, 3, 4, [2, 3, 3]),
                                      (12, 6, 2, [6, 2, 8]), (14, 6, 1, [6, 1, 7]), (16, 2, 5, [2, 5, 7]),
                                      (22, 3, 3, [2, 2, 2])])
def test_against_oracle(n, a, b, ex):
    from polyquant_gb300.detset import POLYQUANT_DETSET

    p = synthetic_fci(n, a, b, seed=80 + n, ex=ex)
    d = O.Detset(p)
    g = POLYQUANT_DETSET(p.n_orb, p.n_alpha, p.n_beta, p.h1, p.eri, p.ex_level)
    rng = np.random.default_rng(n)
    X = rng.standard_normal((d.n_dets, 11))
    X /= np.linalg.norm(X, axis=0)
    T = torch.from_numpy(X).cuda()
    ref = d.evaluate_s2(X)[:, 0]
    for k in (1, 3, 8, 11):
        assert np.abs(np.atleast_1d(g.s2(T[:, :k])) - ref[:k]).max() < 1e-12
    for spin in (0, 1):
        R = g.rdm1(T[:, 0], spin)
        assert np.abs(R - d.create_1rdm(X[:, 0].copy(), 0, spin)).max() < 1e-12
        assert np.array_equal(R, R.T)
    assert np.isnan(g.s2(T[:, :2] * float("nan"))).all()
