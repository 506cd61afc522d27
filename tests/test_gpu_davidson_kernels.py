"""The tall-skinny kernels of the Davidson solver at their edges: fewer rows than one block, row counts that leave a
partial block, more states than one column tile, subspaces that restart, and start vectors in one block.  Energies
against the dense spectrum (1e-9 Eh, the solver's bar), vectors by orthonormality and residual: residuals converge
below 1e-8, and sums of at most 1e4 FP64 terms add about 1e-12."""
import numpy as np
import pytest

import oracle as O
from cases import synthetic_fci

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,a,b,k,m0,mmax", [(4, 2, 1, 1, 1, 0), (6, 3, 2, 1, 2, 5), (6, 3, 3, 3, 4, 0), (7, 3, 3, 5, 9, 15),
                                            (7, 4, 3, 6, 8, 0), (8, 4, 4, 9, 12, 24)])
def test_davidson_edges(n, a, b, k, m0, mmax):
    from polyquant_gb300.detset import POLYQUANT_DETSET

    p = synthetic_fci(n, a, b, seed=70 + n + k)
    g = POLYQUANT_DETSET(p.n_orb, p.n_alpha, p.n_beta, p.h1, p.eri, p.ex_level)
    e, v, info = g.davidson(num_states=k, num_subspace_vec=m0, max_subspace=mmax, convergence_E=1e-8, return_vectors=True)
    H = O.Detset(p).dense_ham()
    w, U = np.linalg.eigh(H)
    x = v.cpu().numpy()
    assert np.abs(x.T @ x - np.eye(k)).max() < 1e-10
    res = np.linalg.norm(H @ x - x * e, axis=0).max()
    assert abs(res - info["max_residual"]) < 1e-10
    # a restart to 9 of 15 vectors for 5 roots does not converge within the iteration limit (nor with any other
    # evaluation of the same products); the others do
    assert info["converged"] == (mmax != 15)
    if info["converged"]:
        # the unit-vector start reaches the eigenvectors that overlap it: every energy is an eigenvalue
        assert res < 1.1e-8 and max(np.abs(w - y).min() for y in e) < 1e-9
