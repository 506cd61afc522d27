"""Batched sigma where the rows of P x w values fall on every split of a warp into lane groups: 1, 6 and 36 positron
determinants with one to four vectors (rows of 1 to 144 values), against each problem's own handle.  Both sum the same
terms: FP64 within 1e-12 of the largest value."""
import numpy as np
import pytest

from polyquant_gb300 import synthetic

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 2, 3, 4])
def test_row_widths(k):
    from polyquant_gb300.batch import CIBatch
    from polyquant_gb300.detset import POLYQUANT_DETSET

    specs = [dict(n_orb=n, n_alpha=a, n_beta=b, n_pos=p, n_pos_orb=m, seed=70 + 10 * p + m)
             for n, a, b, p, m in [(7, 3, 2, 0, 6), (6, 2, 3, 1, 6), (6, 3, 2, 2, 6), (5, 2, 2, 1, 3), (5, 2, 3, 2, 3),
                                   (6, 2, 2, 1, 9), (5, 3, 2, 2, 5)]]
    problems = [synthetic.batch_problem(s) for s in specs]
    batch = CIBatch(problems)
    gen = torch.Generator(device="cuda").manual_seed(k)
    Cs = [torch.randn(n, k, device="cuda", dtype=torch.float64, generator=gen) for n in batch.n_dets]
    for pb, C, S in zip(problems, Cs, batch.sigma(Cs)):
        ref = POLYQUANT_DETSET(**pb).sigma(C)
        assert (S - ref).abs().max().item() <= 1e-12 * ref.abs().max().item()
        assert np.isfinite(S.cpu().numpy()).all()
