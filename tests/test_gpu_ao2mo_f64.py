"""The FP64 AO->MO transform by digit products on the tensor cores, where its tiles, chunks and exponents can go
wrong.  Integrals of low rank, (mu nu|la si) = sum_L B_L B_L, give the result from small matrix products.  Both sides
round at FP64: 1e-14 of the largest value covers sums of 256 terms; where values spread over many decades the
comparison is row by row."""
import numpy as np
import pytest

import oracle as O
from polyquant_gb300 import synthetic

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-14


def _pairs(B, C):
    """(C^T B_L C) by pairs for each factor."""
    i, j = np.tril_indices(C.shape[1])
    return np.stack([(C.T @ b @ C)[i, j] for b in B])


def _factors(rng, n, L=4):
    B = rng.standard_normal((L, n, n))
    return 0.5 * (B + B.transpose(0, 2, 1))


def _packed(B):
    i, j = np.tril_indices(B.shape[1])
    F = torch.from_numpy(B[:, i, j]).cuda()
    M = F.t() @ F
    return M[torch.ones(M.shape, dtype=torch.bool, device="cuda").tril_()]


@pytest.mark.parametrize("n,m", [(1, 1), (2, 1), (5, 5), (16, 16), (17, 15), (31, 31), (32, 32), (33, 17), (48, 48),
                                (64, 64), (65, 65), (97, 81), (128, 128), (129, 113), (240, 9)])
def test_packed_sizes(n, m):
    from polyquant_gb300.integral import ao2mo

    rng = np.random.default_rng(1000 + n)
    B, C = _factors(rng, n), synthetic.mo_coefficients(n, m, seed=n)
    T = _pairs(B, C)
    ref = T.T @ T
    out = ao2mo(_packed(B), torch.from_numpy(C).cuda()).cpu().numpy()
    assert out.shape == ref.shape
    assert np.abs(out - ref).max() <= TOL * max(np.abs(ref).max(), np.abs(B).max() ** 2)


@pytest.mark.parametrize("na,ma,nb,mb", [(40, 37, 7, 6), (7, 7, 66, 64), (33, 1, 32, 32)])
def test_two_species_sizes(na, ma, nb, mb):
    from polyquant_gb300._lib import PQ_AO_PAIRS
    from polyquant_gb300.integral import ao2mo

    rng = np.random.default_rng(na + nb)
    Ba, Bb = _factors(rng, na), _factors(rng, nb)
    Ca, Cb = synthetic.mo_coefficients(na, ma, seed=1), synthetic.mo_coefficients(nb, mb, seed=2)
    ia, ib = np.tril_indices(na), np.tril_indices(nb)
    P = Ba[:, ia[0], ia[1]].T @ Bb[:, ib[0], ib[1]]
    ref = _pairs(Ba, Ca).T @ _pairs(Bb, Cb)
    out = ao2mo(torch.from_numpy(np.ascontiguousarray(P.T)).cuda(), torch.from_numpy(Ca).cuda(),
                torch.from_numpy(Cb).cuda(), layout=PQ_AO_PAIRS).cpu().numpy()
    assert np.abs(out - ref).max() <= TOL * np.abs(ref).max()


def test_scales_and_equal_values():
    """Magnitudes far from one, coefficients that spread over decades, and constant matrices (digits that all add)."""
    from polyquant_gb300.integral import ao2mo

    rng = np.random.default_rng(5)
    n = 40
    B, C = _factors(rng, n), synthetic.mo_coefficients(n, n, seed=3)
    for f in (2.0 ** -400, 1e-30, 1e25, 2.0 ** 300):
        T = _pairs(B, C)
        out = ao2mo(_packed(B) * f, torch.from_numpy(C).cuda()).cpu().numpy()
        assert np.abs(out / f - T.T @ T).max() <= TOL * np.abs(T.T @ T).max()
    W = C * 10.0 ** (-8.0 * np.arange(n) / n)  # MO columns of very different norms: their values keep their digits
    T = _pairs(B, W)
    ref = T.T @ T
    out = ao2mo(_packed(B), torch.from_numpy(W).cuda()).cpu().numpy()
    assert (np.abs(out - ref) <= 2e-13 * np.sqrt(np.outer(np.diag(ref), np.diag(ref)))).all()
    one = np.full((1, n, n), 1.0 / 3.0)
    Cc = np.full((n, n), -1.0 / 7.0)
    T = _pairs(one, Cc)
    out = ao2mo(_packed(one), torch.from_numpy(Cc).cuda()).cpu().numpy()
    assert np.abs(out - T.T @ T).max() <= TOL * np.abs(T.T @ T).max()
    assert not ao2mo(_packed(one) * 0.0, torch.from_numpy(Cc).cuda()).any().item()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_inputs_reach_the_result(bad):
    from polyquant_gb300.integral import ao2mo

    rng = np.random.default_rng(6)
    n = 20
    B, C = _factors(rng, n), synthetic.mo_coefficients(n, n, seed=4)
    P = _packed(B)
    Q = P.clone()
    Q[77] = bad
    assert not torch.isfinite(ao2mo(Q, torch.from_numpy(C).cuda())).any().item()
    C2 = C.copy()
    C2[3, 5] = bad
    out = ao2mo(P, torch.from_numpy(C2).cuda()).cpu().numpy()
    i, j = np.tril_indices(n)
    hit = (i == 5) | (j == 5)
    T = _pairs(B, C)
    ref = T.T @ T
    clean = ~hit[:, None] & ~hit[None, :]
    assert not np.isfinite(out[~clean]).any()
    assert np.abs(out - ref)[clean].max() <= TOL * np.abs(ref).max()


def test_against_the_oracle_and_twice_the_same():
    from polyquant_gb300.integral import ao2mo

    n = 26
    packed = synthetic.ao_eri_packed8(n, seed=9, L=64)
    C = synthetic.mo_coefficients(n, 23, seed=10)
    ref = O.ao2mo_full(O.unpack_packed8(packed, n), C, C)
    P, Cd = torch.from_numpy(packed).cuda(), torch.from_numpy(C).cuda()
    a, b = ao2mo(P, Cd), ao2mo(P, Cd)
    assert torch.equal(a, b)
    assert np.abs(a.cpu().numpy() - ref).max() <= 1e-13 * np.abs(ref).max()
