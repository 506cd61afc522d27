"""What the FP64 digit products promise for entries far below the largest: an absolute error set by the column (or slice),
and full accuracy for a part that is given its own column.

sigma: H of two irreducible representations separates the determinants into blocks; C is of order one in one block and
1e-12 in the other.  The bound 1e-15 max row sum |H| max |C| holds in the small block too; the test asks for less than that,
1e-15 of the largest |sigma|, which is never larger.  In columns of their own both blocks have the 1e-13 of the other tests.

AO->MO with identity coefficients and integrals over 16 decades: 1e-16 n (largest of the slice) in either half."""
import numpy as np
import pytest

from cases import synthetic_fci
from test_gpu_sigma_path import _make, path

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _two_irreps(n, na, nb, seed):
    """Full CI whose even and odd orbitals belong to different representations of a group of two."""
    p = synthetic_fci(n, na, nb, seed=seed)
    odd = np.arange(n) % 2
    i, j = np.tril_indices(n)
    pair = odd[i] ^ odd[j]
    for s in range(2):
        p.h1[0][s] = np.where(odd[:, None] == odd[None, :], p.h1[0][s], 0.0)
    p.eri = {k: np.where(pair[:, None] == pair[None, :], v, 0.0) for k, v in p.eri.items()}
    return p, odd


def test_a_small_block_keeps_the_columns_bound(monkeypatch):
    from polyquant_gb300._lib import PQ_PATH_TENSOR

    n = 10
    p, odd = _two_irreps(n, 5, 5, 12)
    g = _make(p)
    monkeypatch.setenv("PQ_SIGMA64_GATHER", "1")
    r = _make(p)
    mask = sum(1 << int(o) for o in np.nonzero(odd)[0])
    par = [np.array([bin(int(w) & mask).count("1") & 1 for w in g.strings(0, s)[:, -1]]) for s in (0, 1)]
    small = torch.from_numpy((par[0][:, None] ^ par[1][None, :]).reshape(-1).astype(bool)).cuda()
    X = torch.randn(g.N_dets, 1, device="cuda", dtype=torch.float64)
    X[small] *= 1e-12
    R = r.sigma(X)  # exact zeros between the blocks: accurate in each
    assert (R[small].abs().max() < 1e-9 * R.abs().max()).item()
    S = g.sigma(X)
    assert path(g) == (PQ_PATH_TENSOR, 0)
    err = (S - R).abs()
    assert err[small].max().item() <= 1e-15 * R.abs().max().item()
    assert err.max().item() <= 1e-13 * R.abs().max().item()
    two = torch.cat([torch.where(small[:, None], 0.0, X), torch.where(small[:, None], X, 0.0)], 1)
    T = g.sigma(two)
    Q = r.sigma(two)
    assert path(g) == (PQ_PATH_TENSOR, 0)
    assert ((T - Q).abs().amax(0) <= 1e-13 * Q.abs().amax(0)).all()
    assert (T.sum(1) - R[:, 0])[small].abs().max().item() <= 1e-13 * R[small].abs().max().item()


def test_integrals_far_below_their_slice():
    from polyquant_gb300._lib import PQ_AO_PAIRS, PQ_XFORM_FP64
    from polyquant_gb300.integral import ao2mo

    n = 24
    q = n * (n + 1) // 2
    rng = np.random.default_rng(8)
    M = rng.standard_normal((q, q)) * 10.0 ** (-16.0 * rng.random((q, q)))
    M = 0.5 * (M + M.T)
    eye = torch.eye(n, device="cuda", dtype=torch.float64)
    out = ao2mo(torch.from_numpy(M).cuda(), eye, eye, layout=PQ_AO_PAIRS, mode=PQ_XFORM_FP64).cpu().numpy()
    bound = 1e-16 * n * (np.abs(M).max(0)[None, :] + np.abs(M).max(1)[:, None])
    assert (np.abs(out - M) <= bound).all()
