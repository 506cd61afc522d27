"""<S^2> and the alpha 1-RDM where one spin has few strings or none (columns and beta entries split over several blocks, no
flips): against the oracle, 1e-12 for sums of unit vectors as in the other tests of the lists."""
import numpy as np
import pytest

import oracle as O
from cases import synthetic_fci

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,a,b,ex", [(12, 1, 6, [1, 6, 7]), (13, 1, 5, [1, 5, 4]), (9, 0, 3, [0, 3, 3]), (11, 4, 0, [4, 0, 4]),
                                      (14, 1, 4, [1, 4, 5]), (6, 1, 1, [1, 1, 2])])
def test_against_oracle(n, a, b, ex):
    from polyquant_gb300.detset import POLYQUANT_DETSET

    p = synthetic_fci(n, a, b, seed=40 + n, ex=ex)
    d = O.Detset(p)
    g = POLYQUANT_DETSET(p.n_orb, p.n_alpha, p.n_beta, p.h1, p.eri, p.ex_level)
    X = np.random.default_rng(n).standard_normal((d.n_dets, 9))
    X /= np.linalg.norm(X, axis=0)
    T = torch.from_numpy(X).cuda()
    ref = d.evaluate_s2(X)[:, 0]
    for k in (1, 4, 9):
        assert np.abs(np.atleast_1d(g.s2(T[:, :k])) - ref[:k]).max() < 1e-12
    for spin in (0, 1):
        assert np.abs(g.rdm1(T[:, 0], spin) - d.create_1rdm(X[:, 0].copy(), 0, spin)).max() < 1e-12
