"""Which kernels an FP64 sigma ran on (pq_debug_sigma_path): the shapes that the tests of the tensor-core paths compare
with the element kernel are in fact computed by the digit products, whose gate stays down; non-finite input raises it; and
the other spaces take the row kernel, the element kernel or the explicit matrix."""
import ctypes
from itertools import combinations

import numpy as np
import pytest

from cases import synthetic_en, synthetic_ep, synthetic_fci, synthetic_unrestricted

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _make(p, **kw):
    from polyquant_gb300.detset import POLYQUANT_DETSET

    return POLYQUANT_DETSET(p.n_orb, p.n_alpha, p.n_beta, p.h1, p.eri, p.ex_level, restricted=p.restricted,
                            charge=p.charge, max_collective_excitation_level=p.max_collective, **kw)


def path(g):
    from polyquant_gb300 import _lib

    w, f = ctypes.c_int32(-1), ctypes.c_int32(-1)
    assert _lib.load().pq_debug_sigma_path(g._h, ctypes.byref(w), ctypes.byref(f)) == _lib.PQ_OK
    return w.value, f.value


def _x(g, k):
    return torch.randn(k, g.N_dets, device="cuda", dtype=torch.float64).t()


@pytest.mark.parametrize("n,a,b,restricted", [(10, 5, 5, True), (11, 5, 4, True), (12, 6, 3, True), (13, 2, 8, True),
                                             (13, 8, 2, True), (15, 3, 3, True), (17, 2, 4, True), (10, 4, 6, False),
                                             (11, 5, 5, False)])
def test_full_ci_runs_on_the_tensor_cores(n, a, b, restricted):
    from polyquant_gb300._lib import PQ_PATH_NONE, PQ_PATH_TENSOR

    g = _make(synthetic_fci(n, a, b, seed=90 + n) if restricted else synthetic_unrestricted(n, a, b, seed=91))
    assert path(g) == (PQ_PATH_NONE, 0)
    for k in (1, 2, 3, 4, 5):
        g.sigma(_x(g, k))
        assert path(g) == (PQ_PATH_TENSOR, 0)
    g.sigma(_x(g, 2).cpu().numpy())
    assert path(g) == (PQ_PATH_TENSOR, 0)
    X = _x(g, 1)
    X[3, 0] = float("nan")
    g.sigma(X)
    assert path(g) == (PQ_PATH_TENSOR, 1)
    g.sigma(_x(g, 1))
    assert path(g) == (PQ_PATH_TENSOR, 0)
    g.close()


def test_selected_lists_run_on_the_tensor_cores():
    from polyquant_gb300._lib import PQ_PATH_TENSOR

    p = synthetic_fci(12, 4, 4, seed=98)
    s = np.random.default_rng(3).permutation(np.array([sum(1 << o for o in c) for c in combinations(range(12), 4)], dtype=np.uint64))
    g = _make(p, selected_strings=[[s[:300], s[100:250]]])
    g.sigma(_x(g, 3))
    assert path(g) == (PQ_PATH_TENSOR, 0)


@pytest.mark.parametrize("args", [(5, 1, 0, 4, 1, 0), (12, 1, 1, 7, 1, 0), (33, 1, 1, 9, 1, 0), (6, 2, 1, 5, 1, 1),
                                  (6, 2, 2, 4, 1, 1), (8, 2, 2, 6, 1, 0), (60, 1, 1, 40, 1, 0), (40, 1, 0, 40, 1, 1)])
def test_two_species_run_on_the_tensor_cores(monkeypatch, args):
    from polyquant_gb300._lib import PQ_PATH_TENSOR

    monkeypatch.setenv("PQ_TWO64_ALWAYS", "1")
    g = _make(synthetic_ep(*args, seed=sum(args)))
    for k in (1, 3, 6):
        g.sigma(_x(g, k))
        assert path(g) == (PQ_PATH_TENSOR, 0)
    g = _make(synthetic_en(6, 2, 1, 5, 1, 1, seed=5))
    g.sigma(_x(g, 2))
    assert path(g) == (PQ_PATH_TENSOR, 0)


def test_other_paths(monkeypatch):
    from polyquant_gb300._lib import PQ_PATH_ELEMENT, PQ_PATH_MATRIX, PQ_PATH_ROWS

    g = _make(synthetic_fci(10, 4, 4, seed=1, ex=[2, 2, 2]))
    g.sigma(_x(g, 2))
    assert path(g) == (PQ_PATH_ROWS, 0)
    g.create_ham()
    g.sigma(_x(g, 2))
    assert path(g) == (PQ_PATH_MATRIX, 0)
    monkeypatch.setenv("PQ_SIGMA64_GATHER", "1")
    g = _make(synthetic_fci(10, 5, 5, seed=2))
    g.sigma(_x(g, 2))
    assert path(g) == (PQ_PATH_ELEMENT, 0)


@pytest.mark.parametrize("n,a,b,tensor", [(16, 1, 5, False), (20, 1, 5, False), (12, 2, 6, True), (16, 8, 1, True)])
def test_few_alpha_strings_stay_with_the_element_kernel(n, a, b, tensor):
    """Fewer than a tile of 64 alpha strings leave the tensor-core kernels idle."""
    from polyquant_gb300._lib import PQ_PATH_ELEMENT, PQ_PATH_TENSOR

    g = _make(synthetic_fci(n, a, b, seed=7))
    g.sigma(_x(g, 2))
    assert path(g)[0] == (PQ_PATH_TENSOR if tensor else PQ_PATH_ELEMENT)


@pytest.mark.parametrize("args,tensor", [((6, 3, 2, 8, 1, 1), False), ((8, 1, 2, 10, 1, 1), False), ((20, 1, 1, 7, 1, 1), True),
                                         ((11, 2, 1, 18, 1, 0), True)])
def test_size_rule_of_two_species(args, tensor):
    """Four lists of which few strings are connected stay with the element kernel."""
    from polyquant_gb300._lib import PQ_PATH_ELEMENT, PQ_PATH_TENSOR

    g = _make(synthetic_ep(*args, seed=9))
    g.sigma(_x(g, 3))
    assert path(g)[0] == (PQ_PATH_TENSOR if tensor else PQ_PATH_ELEMENT)
