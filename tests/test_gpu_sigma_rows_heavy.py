"""Rows of every weight in the warp-per-determinant FP64 sigma: CTAs whose rows are all heavy (a warp each), or of which
one outweighs the others (shared by the CTA), against the explicit matrix.  Sums of at most 1e4 FP64 terms in another order: 1e-12 of
the largest value."""
import pytest

from cases import synthetic_fci
from test_gpu_sigma_path import _make

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-12


def _x(g, k):
    return torch.randn(k, g.N_dets, device="cuda", dtype=torch.float64, generator=torch.Generator(device="cuda").manual_seed(k)).t()


@pytest.mark.parametrize("n,a,b,ex", [(20, 3, 3, [3, 3, 4]), (30, 2, 2, [2, 2, 3]), (21, 4, 4, [2, 2, 2]), (44, 2, 1, [2, 1, 2])])
def test_heavy_rows_against_the_explicit_matrix(n, a, b, ex):
    g = _make(synthetic_fci(n, a, b, seed=5, ex=ex))
    X = _x(g, 4)
    S = [g.sigma(X[:, :k]) for k in (1, 2, 3, 4)]
    g.create_ham()
    for k in (1, 2, 3, 4):
        H = g.sigma(X[:, :k])
        assert (S[k - 1] - H).abs().max().item() <= TOL * H.abs().max().item()
    # rows of the matrix are what the elements are
    rp, col, val = g.ham_csr(upper=False)
    for i in (0, 1, g.N_dets // 2, g.N_dets - 1):
        j = col[rp[i]:rp[i + 1]]
        assert abs(g.elements([i] * len(j), j) - val[rp[i]:rp[i + 1]]).max() <= TOL * abs(val[rp[i]:rp[i + 1]]).max()
    g.close()
