"""Which truncated spaces take the warp-per-determinant FP64 sigma: not the large ones that are nearly full, which the
element kernel does faster.  Both kernels on one space agree.  Sums of at most 1e4 FP64 terms in another order: 1e-12 of
the largest value."""
import pytest

from cases import synthetic_fci
from test_gpu_sigma_path import _make, path

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-12


def _x(g, k):
    return torch.randn(k, g.N_dets, device="cuda", dtype=torch.float64, generator=torch.Generator(device="cuda").manual_seed(k)).t()


@pytest.mark.parametrize("n,a,b,level,one,more", [
    (11, 5, 5, 4, "rows", "rows"),        # 45 311 determinants, short rows
    (11, 5, 5, 6, "element", "element"),  # 172 683, 32 packed singles, rows of the other kernel's CTAs mostly full
    (11, 4, 4, 7, "rows", "rows"),        # 330 beta strings fill 0.64 of two CTAs
    (12, 6, 6, 6, "rows", "rows"),        # 558 810, 64 packed singles, below the size
    (13, 6, 6, 8, "element", "rows"),     # 2 777 517
])
def test_rule(n, a, b, level, one, more):
    from polyquant_gb300 import _lib

    want = {"rows": _lib.PQ_PATH_ROWS, "element": _lib.PQ_PATH_ELEMENT}
    g = _make(synthetic_fci(n, a, b, seed=3, ex=[min(level, a), min(level, b), level]))
    X = _x(g, 3)
    S1 = g.sigma(X[:, :1])
    assert path(g)[0] == want[one]
    S = g.sigma(X)
    assert path(g)[0] == want[more]
    assert (S[:, :1] - S1).abs().max().item() <= TOL * S1.abs().max().item()
    g.close()
