"""The beta 1-RDM with few entries a pair (a thread per entry): one beta electron, rows of unequal length, entry blocks and
row chunks that are partly filled, both sides of the rule, and NaN.  Sums of unit vectors against the oracle: 1e-12, as in
the other tests of the lists."""
import numpy as np
import pytest

import oracle as O
from cases import synthetic_fci

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,a,b,ex", [(5, 1, 1, [1, 1, 2]), (20, 3, 1, [3, 1, 4]), (24, 2, 1, [2, 1, 2]), (30, 2, 2, [2, 2, 2]),
                                      (9, 2, 4, [2, 4, 6]), (17, 2, 2, [2, 2, 3])])
def test_against_oracle(n, a, b, ex):
    from polyquant_gb300.detset import POLYQUANT_DETSET

    p = synthetic_fci(n, a, b, seed=60 + n, ex=ex)
    d = O.Detset(p)
    g = POLYQUANT_DETSET(p.n_orb, p.n_alpha, p.n_beta, p.h1, p.eri, p.ex_level)
    x = np.random.default_rng(n).standard_normal(d.n_dets)
    x /= np.linalg.norm(x)
    T = torch.from_numpy(x).cuda()
    for spin in (0, 1):
        R = g.rdm1(T, spin)
        assert np.abs(R - d.create_1rdm(x.copy(), 0, spin)).max() < 1e-12
    assert np.isnan(np.diag(g.rdm1(T * float("nan"), 1))).all()
