"""The FP32 full-CI sigma of four roots where a row of columns ends inside the two blocks of 256 that a CTA of the singles
kernel covers (462, 330 and 495 strings), against FP64 and the gathers of the same sigma: the FP32 bounds of the larger
shapes."""
import pytest

from cases import synthetic_fci

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SIGMA_RTOL_FP32 = 2e-5


@pytest.mark.parametrize("n,a,b", [(11, 5, 5), (11, 5, 4), (12, 4, 5)])
def test_ragged_columns(monkeypatch, n, a, b):
    from polyquant_gb300._lib import PQ_FP32
    from polyquant_gb300.detset import POLYQUANT_DETSET

    p = synthetic_fci(n, a, b, seed=60 + n + b)

    def make():
        return POLYQUANT_DETSET(p.n_orb, p.n_alpha, p.n_beta, p.h1, p.eri, p.ex_level, restricted=p.restricted,
                                charge=p.charge, max_collective_excitation_level=p.max_collective)

    g = make()
    monkeypatch.setenv("PQ_SIGMA32_NO_SS", "1")
    h = make()
    gen = torch.Generator(device="cuda").manual_seed(n + b)
    X = torch.randn(g.N_dets, 4, device="cuda", dtype=torch.float64, generator=gen)
    S64, S, G = g.sigma(X), g.sigma(X, precision=PQ_FP32), h.sigma(X, precision=PQ_FP32)
    scale = S64.abs().max().item()
    assert (S - S64).abs().max().item() <= SIGMA_RTOL_FP32 * scale
    assert (S - G).abs().max().item() <= SIGMA_RTOL_FP32 * scale
