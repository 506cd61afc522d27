"""FP32 sigma of four roots over caller-chosen string lists that are long and filled enough for the same-spin tensor-core
GEMMs: the doubles matrix of the beta list is its own when the two lists differ (in length, in members or in order), and
shared when they are the same.  Against FP64, with the FP32 bound of the other shapes."""
from itertools import combinations

import numpy as np
import pytest

from cases import synthetic_fci

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SIGMA_RTOL_FP32 = 2e-5


@pytest.mark.parametrize("lists", ["shorter beta", "longer beta", "other members", "other order", "same"])
def test_lists_that_differ(lists):
    from polyquant_gb300._lib import PQ_FP32
    from polyquant_gb300.detset import POLYQUANT_DETSET

    p = synthetic_fci(12, 6, 6, seed=71)
    rng = np.random.default_rng(5)
    s = rng.permutation(np.array([sum(1 << o for o in c) for c in combinations(range(12), 6)], dtype=np.uint64))
    a = s[:600]
    b = {"shorter beta": s[:300], "longer beta": s[:800], "other members": s[300:900], "other order": a[::-1], "same": a}[lists]
    g = POLYQUANT_DETSET(p.n_orb, p.n_alpha, p.n_beta, p.h1, p.eri, restricted=p.restricted, charge=p.charge,
                         selected_strings=[[a, b]])
    X = torch.randn(g.N_dets, 4, device="cuda", dtype=torch.float64, generator=torch.Generator(device="cuda").manual_seed(2))
    S64, S = g.sigma(X), g.sigma(X, precision=PQ_FP32)
    g.close()
    assert (S - S64).abs().max().item() <= SIGMA_RTOL_FP32 * S64.abs().max().item()
