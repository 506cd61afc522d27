"""The sizing of the FP64 tensor-core sigma (plan.fp64_tensor_bytes): its rules and its largest terms on the host, and on the
GPU against what handles hold after a sigma of four vectors (pq_debug_scratch_bytes) and whether they took that path."""
import ctypes

import pytest

from polyquant_gb300.plan import davidson_device_bytes, fp64_tensor_bytes


def test_terms_and_rules():
    n = 12870  # strings of FCI(16o, 8a8b)
    digits, dense = 14 * 4 * n * 12928, 14 * n * 12928
    got = fp64_tensor_bytes([16], [8], [8])
    assert digits + dense < got < 1.02 * (digits + dense)
    assert fp64_tensor_bytes([16], [8], [8], restricted=False) - got == dense
    assert fp64_tensor_bytes([16], [8], [8], num_vectors=1) == got - 3 * digits // 4
    # small, few alpha strings, more than 80 singles and orbitals, dense matrices that are too large
    assert fp64_tensor_bytes([9], [4], [4]) == fp64_tensor_bytes([16], [1], [6]) == 0
    assert fp64_tensor_bytes([18], [8], [8]) == fp64_tensor_bytes([17], [8], [8]) == 0
    base = davidson_device_bytes(n * n, 4, 20)
    assert davidson_device_bytes(n * n, 4, 20, fp64_space=([16], [8], [8], True)) == base + got
    assert davidson_device_bytes(n * n, 4, 20, fp64_space=([16], [8], [8], True), explicit_nnz=5) == \
        davidson_device_bytes(n * n, 4, 20, explicit_nnz=5)
    # positronium hydride in 60 + 40 orbitals: three pairs of 3600, 2400 and 2400 rows
    two = fp64_tensor_bytes([60, 40], [1, 1], [1, 0])
    matrices = 14 * (3600 * 3648 + 2 * 2400 * 2432)
    assert matrices < two < matrices + 3 * 4 * 144000 * (14 * 1.02 + 8 * 8)  # digits, and at most eight copies
    assert fp64_tensor_bytes([5, 4], [1, 1], [0, 0]) == fp64_tensor_bytes([6, 8], [3, 1], [2, 1]) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("space", [([10], [5], [5]), ([11], [5], [4]), ([13], [2], [8]), ([16], [1], [5]), ([12], [6], [6]),
                                   ([60, 40], [1, 1], [1, 0]), ([20, 7], [1, 1], [1, 1]), ([6, 8], [3, 1], [2, 1])])
def test_against_handles(space):
    torch = pytest.importorskip("torch")
    from cases import synthetic_ep, synthetic_fci
    from polyquant_gb300 import _lib
    from test_gpu_sigma_path import _make, path

    n, a, b = space
    g = _make(synthetic_fci(n[0], a[0], b[0], seed=1) if len(n) == 1 else synthetic_ep(n[0], a[0], b[0], n[1], a[1], b[1], seed=1))
    g.sigma(torch.randn(4, g.N_dets, device="cuda", dtype=torch.float64).t())
    want = fp64_tensor_bytes(n, a, b)
    assert (path(g)[0] == _lib.PQ_PATH_TENSOR) == (want > 0)
    if want:
        held = ctypes.c_int64()
        assert _lib.load().pq_debug_scratch_bytes(g._h, ctypes.byref(held)) == _lib.PQ_OK
        assert held.value <= 1.02 * want + 65536 and want <= 1.3 * held.value + 65536, (held.value, want)
