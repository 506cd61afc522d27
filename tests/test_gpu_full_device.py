"""A device that is too full for tables which only make a call faster (allocations beyond a limit fail as on a full
device, pq_debug_set_alloc_room): the call is answered without them."""
import ctypes

import pytest

from cases import synthetic_ep, synthetic_fci
from test_gpu_sigma_path import _make, path

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-12


class Room:
    """`with Room(bytes)`: the library may allocate that much more."""

    def __init__(self, room):
        self.room = room

    def __enter__(self):
        set_room(self.room)

    def __exit__(self, *a):
        set_room(-1)


def set_room(room):
    from polyquant_gb300 import _lib

    held = ctypes.c_int64()
    assert _lib.load().pq_debug_set_alloc_room(ctypes.c_longlong(room), ctypes.byref(held)) == _lib.PQ_OK
    return held.value


def _x(g, k):
    return torch.randn(k, g.N_dets, device="cuda", dtype=torch.float64).t()


def test_row_tables_do_not_fit():
    from polyquant_gb300 import _lib

    p = synthetic_fci(16, 4, 4, seed=2, ex=[2, 2, 2])
    before = set_room(-1)
    g = _make(p)
    size = set_room(-1) - before
    X = _x(g, 3)
    want = g.sigma(X)
    assert path(g)[0] == _lib.PQ_PATH_ROWS
    with Room(size - 1):
        r = _make(p)
    S = r.sigma(X)
    assert path(r)[0] == _lib.PQ_PATH_ELEMENT
    assert (S - want).abs().max().item() <= TOL * want.abs().max().item()
    nnz = r.create_ham()
    assert nnz == g.create_ham()
    with pytest.raises(_lib.PQError) as e, Room(0):
        _make(p)
    assert e.value.status == _lib.PQ_ERR_OOM


def test_batch_members_hold_no_row_tables():
    """Their sigma is the batched kernel's: a batch of one holds less than a handle, which has the row tables."""
    from polyquant_gb300.batch import CIBatch

    p = synthetic_fci(9, 4, 4, seed=3)
    start = set_room(-1)
    g = _make(p)
    handle = set_room(-1) - start
    b = CIBatch([dict(n_orb=p.n_orb, n_alpha=p.n_alpha, n_beta=p.n_beta, h1=p.h1, eri=p.eri, excitation_level=p.ex_level,
                      restricted=p.restricted, charge=p.charge)])
    batch = set_room(-1) - start - handle
    assert batch < handle, (batch, handle)
    b.close()
    g.close()


def test_transform_buffers_are_given_back():
    """What the transforms keep between calls goes when another allocation of the library does not fit."""
    from polyquant_gb300 import _lib
    from polyquant_gb300.integral import ao2mo

    n = 60
    npair = n * (n + 1) // 2
    P = torch.randn(npair * (npair + 1) // 2, device="cuda", dtype=torch.float64)
    C = torch.randn(n, n, device="cuda", dtype=torch.float64)
    assert _lib.load().pq_ao2mo_release_workspace() == _lib.PQ_OK
    before = set_room(-1)
    out = ao2mo(P, C, layout=_lib.PQ_AO_PACKED8, mode=_lib.PQ_XFORM_FP64)
    kept = set_room(-1) - before
    assert kept > 8 * npair * npair
    with Room(0):
        g = _make(synthetic_fci(10, 5, 5, seed=4))
    assert g.N_dets == 63504
    assert set_room(-1) - before < kept
    again = ao2mo(P, C, layout=_lib.PQ_AO_PACKED8, mode=_lib.PQ_XFORM_FP64)
    assert torch.equal(out, again)
    # a transform that does not fit beside its own buffers of an earlier call frees them and fails only then
    with Room(0), pytest.raises(_lib.PQError) as e:
        m = 90
        q = m * (m + 1) // 2
        ao2mo(torch.randn(q * (q + 1) // 2, device="cuda", dtype=torch.float64),
              torch.randn(m, m, device="cuda", dtype=torch.float64), layout=_lib.PQ_AO_PACKED8, mode=_lib.PQ_XFORM_FP64)
    assert e.value.status == _lib.PQ_ERR_OOM
    assert torch.equal(out, ao2mo(P, C, layout=_lib.PQ_AO_PACKED8, mode=_lib.PQ_XFORM_FP64))


def _need(make, run):
    """Device bytes that run(handle) takes from the library on a fresh handle, to within 2 %."""
    from polyquant_gb300 import _lib

    _lib.load().pq_ao2mo_release_workspace()  # else the first failure would free it
    lo, hi = 0, 1 << 20
    while True:
        g = make()
        try:
            with Room(hi):
                run(g)
            break
        except Exception:
            lo, hi = hi, 2 * hi
    while hi - lo > hi // 50:
        mid = (lo + hi) // 2
        g = make()
        try:
            with Room(mid):
                run(g)
            hi = mid
        except Exception:
            lo = mid
    return hi


@pytest.mark.parametrize("what", ["fp32", "davidson", "ham"])
@pytest.mark.parametrize("p", [lambda: synthetic_fci(11, 5, 5, seed=5), lambda: synthetic_ep(33, 1, 1, 9, 1, 0, seed=6)],
                         ids=["full", "two species"])
def test_tables_of_the_tensor_cores_make_room(monkeypatch, p, what):
    """A call that fits a handle without them fits one that has used them."""
    from polyquant_gb300 import _lib

    monkeypatch.setenv("PQ_TWO64_ALWAYS", "1")
    p = p()
    if what == "ham" and p.n_orb[0] == 11:
        p = synthetic_fci(10, 5, 4, seed=5)
    runs = {"fp32": lambda g: g.sigma(torch.ones(g.N_dets, 4, device="cuda", dtype=torch.float64), precision=_lib.PQ_FP32),
            "davidson": lambda g: g.davidson(num_states=1, num_subspace_vec=3, convergence_E=1e-6)[0],
            "ham": lambda g: g.create_ham()}
    run = runs[what]
    monkeypatch.setenv("PQ_SIGMA64_GATHER", "1")
    room = _need(lambda: _make(p), run)
    monkeypatch.delenv("PQ_SIGMA64_GATHER")
    g = _make(p)
    X = _x(g, 4)
    before = set_room(-1)
    S = g.sigma(X)
    tables = set_room(-1) - before
    assert path(g)[0] == _lib.PQ_PATH_TENSOR
    with Room(max(0, room - tables // 2)):
        out = run(g)
    if what == "davidson":
        assert abs(out - run(g)).max() < 1e-6
    g.release_ham()
    assert (g.sigma(X) - S).abs().max().item() <= TOL * S.abs().max().item()
    g.close()


def test_row_tables_make_room():
    """Likewise the row kernel's, when a solve does not fit beside them."""
    p = synthetic_fci(16, 4, 4, seed=7, ex=[2, 2, 2])
    g = _make(p)

    def run(h):
        return h.davidson(num_states=1, num_subspace_vec=3, convergence_E=1e-8)[0]

    e = run(g)
    room = _need(lambda: _make(p), run)  # with them
    with Room(room * 4 // 5):
        low = run(g)
    assert abs(low - e).max() < 1e-8
    g.close()
