"""An explicit matrix that does not fit leaves no matrix behind: the row offsets of the failed build are not taken for one.
Two species, whose build has no tables that could make room."""
import ctypes

import pytest

from cases import synthetic_ep
from test_gpu_full_device import Room
from test_gpu_sigma_path import _make

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_no_matrix_after_a_failed_build():
    from polyquant_gb300 import _lib

    L = _lib.load()
    assert L.pq_ao2mo_release_workspace() == _lib.PQ_OK
    g = _make(synthetic_ep(20, 1, 1, 9, 1, 0, seed=6))
    n = g.N_dets
    with pytest.raises(_lib.PQError) as e, Room(24 * n):  # row counts and offsets fit, the entries do not
        g.create_ham()
    assert e.value.status == _lib.PQ_ERR_OOM
    nnz = ctypes.c_int64(-1)
    assert L.pq_ci_ham_csr(g._h, 0, ctypes.byref(nnz), None, None, None) == _lib.PQ_ERR_STATE
    X = torch.randn(2, n, device="cuda", dtype=torch.float64).t()
    want = g.sigma(X)
    assert g.create_ham() > 2 * n
    assert (g.sigma(X) - want).abs().max() <= 1e-12 * want.abs().max()
    g.close()
