"""FP64 sigma with a warp per determinant (ci_sigma_rows.cu) against the oracle where its grouped tables and level
limits can go wrong: unequal spin lists and levels, a collective limit below the species limit, an empty spin,
unrestricted blocks, determinants on both sides of the CTA-sharing threshold, and every width.

FP64 sums of at most 1e4 terms differ from the oracle's order by about 1e4 * 2^-53 of the largest element, 1e-12.
"""
import ctypes

import numpy as np
import pytest

import oracle as O
from cases import synthetic_fci, synthetic_unrestricted

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-12


def _problem(name):
    if name == "one_empty_spin":
        return synthetic_fci(7, 2, 0, seed=3, ex=[2, 0, 2])
    if name == "unequal_levels":
        return synthetic_fci(9, 4, 3, seed=4, ex=[1, 3, 3])
    if name == "total_below_levels":
        return synthetic_fci(8, 4, 3, seed=5, ex=[3, 3, 4])
    if name == "unrestricted_cisd":
        return synthetic_unrestricted(8, 3, 4, seed=6, ex=[2, 2, 2])
    if name == "collective":
        p = synthetic_fci(9, 3, 3, seed=7, ex=[3, 3, 5])
        p.max_collective = 2
        return p
    if name == "heavy":  # the Fermi determinant has 1 + 2 * 68 + 2 * 816 + 68^2 connections
        return synthetic_fci(21, 4, 4, seed=8, ex=[2, 2, 2])
    return synthetic_fci(7, 3, 3, seed=9)  # full, 1225 determinants


@pytest.mark.parametrize("name", ["one_empty_spin", "unequal_levels", "total_below_levels", "unrestricted_cisd",
                                  "collective", "heavy", "full"])
def test_sigma_rows_against_oracle(name):
    from polyquant_gb300.detset import POLYQUANT_DETSET

    p = _problem(name)
    g = POLYQUANT_DETSET(p.n_orb, p.n_alpha, p.n_beta, p.h1, p.eri, p.ex_level, restricted=p.restricted,
                         charge=p.charge, max_collective_excitation_level=p.max_collective)
    ref = O.Detset(p)
    assert g.N_dets == ref.n_dets
    C = np.random.default_rng(2).standard_normal((ref.n_dets, 7))
    S_ref = ref.sigma(C)
    scale = np.abs(S_ref).max()
    for k in (1, 2, 3, 4, 7):
        S = g.sigma(torch.from_numpy(C[:, :k].copy()).cuda()).cpu().numpy()
        assert np.abs(S - S_ref[:, :k]).max() <= TOL * scale


def test_one_vector_in_place():
    """sigma written over its own input: a single FP64 vector is read in place only when the buffers are apart."""
    from polyquant_gb300 import _lib
    from polyquant_gb300.detset import POLYQUANT_DETSET

    for ex in ([4, 4, 8], [2, 2, 2]):
        p = synthetic_fci(8, 4, 4, seed=10, ex=ex)
        g = POLYQUANT_DETSET(p.n_orb, p.n_alpha, p.n_beta, p.h1, p.eri, p.ex_level)
        c = torch.randn(g.N_dets, device="cuda", dtype=torch.float64)
        want = g.sigma(c)
        x = c.clone()
        st = _lib.load().pq_ci_sigma(g._h, ctypes.c_void_p(x.data_ptr()), g.N_dets, 1, ctypes.c_void_p(x.data_ptr()),
                                     g.N_dets, _lib.PQ_FP64)
        torch.cuda.synchronize()
        assert st == _lib.PQ_OK and torch.equal(x, want)
