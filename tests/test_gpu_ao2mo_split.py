"""The split-precision AO->MO transform at the edges of its tiles: rows (MO, slice) of the second product in boxes of 32
slices and tiles of 128 rows, columns in boxes of 64, batches of slices.  Each product drops lo * lo and rounds lo, so
an operand is good to 2^-16 (BF16) or 2^-21 (TF32) of its value; four contractions, each with three such terms and FP32
sums, stay within 16 of those units of the largest value the absolute operands give."""
import numpy as np
import pytest

from polyquant_gb300 import synthetic

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

UNIT = {"bf16x3": 2.0**-16, "tf32x3": 2.0**-21}


def _pairs(B, C):
    i, j = np.tril_indices(C.shape[1])
    return np.stack([(C.T @ b @ C)[i, j] for b in B])


@pytest.mark.parametrize("mode", ["bf16x3", "tf32x3"])
@pytest.mark.parametrize("n,m", [(1, 1), (2, 2), (7, 5), (8, 8), (31, 16), (33, 31), (33, 32), (64, 63), (65, 65), (97, 3),
                                (129, 128), (129, 40), (150, 141)])
def test_sizes_and_layouts(mode, n, m):
    from polyquant_gb300._lib import PQ_AO_PAIRS, PQ_XFORM_BF16X3, PQ_XFORM_TF32X3
    from polyquant_gb300.integral import ao2mo

    x = {"bf16x3": PQ_XFORM_BF16X3, "tf32x3": PQ_XFORM_TF32X3}[mode]
    rng = np.random.default_rng(n * 1000 + m)
    B = rng.standard_normal((4, n, n))
    B = 0.5 * (B + B.transpose(0, 2, 1))
    C = rng.standard_normal((n, m)) / np.sqrt(n)
    i, j = np.tril_indices(n)
    F = torch.from_numpy(B[:, i, j]).cuda()
    M = F.t() @ F
    M = (M + M.t()) / 2
    T, Tabs = _pairs(B, C), _pairs(np.abs(B), np.abs(C))
    ref, scale = T.T @ T, (Tabs.T @ Tabs).max()
    Cd = torch.from_numpy(C).cuda()
    packed = M[torch.ones(M.shape, dtype=torch.bool, device="cuda").tril_()]
    out = ao2mo(packed, Cd, mode=x).cpu().numpy()
    assert out.shape == ref.shape
    assert np.abs(out - ref).max() <= 16 * UNIT[mode] * scale
    # the same values as a pair matrix: the same FP32 slices, so the same result
    full = ao2mo(M.contiguous(), Cd, layout=PQ_AO_PAIRS, mode=x).cpu().numpy()
    assert np.array_equal(full, out)
