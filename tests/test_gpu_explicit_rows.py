"""The explicit Hamiltonian built a warp per determinant, on spaces with rows on both sides of the CTA-sharing
threshold, with more rows than one scan block, and rebuilt with a screening threshold in the arrays of the last
build.  The stored elements are those that sigma applies, so the two products differ by the order of at most 1e4
FP64 terms: 1e-12 of the largest."""
import numpy as np
import pytest

from cases import synthetic_fci

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,a,b,ex", [(21, 4, 4, [2, 2, 2]), (9, 4, 3, [3, 3, 4]), (10, 5, 4, [5, 4, 9]), (6, 1, 0, [1, 0, 1])])
def test_build_matches_sigma_and_prunes(n, a, b, ex):
    from polyquant_gb300.detset import POLYQUANT_DETSET

    p = synthetic_fci(n, a, b, seed=50 + n, ex=ex)
    g = POLYQUANT_DETSET(p.n_orb, p.n_alpha, p.n_beta, p.h1, p.eri, p.ex_level)
    C = torch.randn(3, g.N_dets, device="cuda", dtype=torch.float64).t()
    want = g.sigma(C)
    nnz = g.create_ham()
    for k in (1, 2, 3):
        assert (g.sigma(C[:, :k]) - want[:, :k]).abs().max().item() <= 1e-12 * want.abs().max().item()
    rp, col, val = g.ham_csr(upper=False)
    assert rp[-1] == nnz == len(val)
    row = np.repeat(np.arange(g.N_dets), np.diff(rp))
    assert np.all((np.diff(col) > 0) | (np.diff(row) > 0))  # every partner once
    assert np.all((val != 0.0) | (row == col))
    thr = float(np.median(np.abs(val)))
    kept = g.create_ham(screening_threshold=thr)
    rp2, col2, val2 = g.ham_csr(upper=False)
    big = np.abs(val) > thr
    assert kept == big.sum() and np.array_equal(col2, col[big]) and np.array_equal(val2, val[big])
    assert np.array_equal(np.diff(rp2), np.bincount(row[big], minlength=g.N_dets))
    g.release_ham()
    assert torch.equal(g.sigma(C), want)
