"""Waits that run out in the AO->MO kernels: whatever the budget (one cycle stops a kernel at its first pending wait, longer
ones at some later point, or not at all where the pipeline is faster), a call either reports PQ_TIMEOUT or has the numbers
of an undisturbed one, so no warp goes on where some of its lanes have given up, and the next call is correct."""
import pytest

from polyquant_gb300 import synthetic

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["PQ_XFORM_BF16X3", "PQ_XFORM_TF32X3", "PQ_XFORM_FP64"])
@pytest.mark.parametrize("n,n_mo", [(24, 24), (72, 40), (130, 130)])
def test_timeout_or_the_same_numbers(mode, n, n_mo):
    from polyquant_gb300 import _lib
    from polyquant_gb300.integral import ao2mo

    L = _lib.load()
    P = torch.from_numpy(synthetic.ao_eri_packed8(n, seed=n, L=16)).cuda()
    C = torch.from_numpy(synthetic.mo_coefficients(n, n_mo, seed=n + 1)).cuda()
    want = ao2mo(P, C, mode=getattr(_lib, mode))
    try:
        for budget in (1, 100, 300, 700, 1000, 2000, 3000, 5000, 10000, 30000, 100000):
            L.pq_debug_set_wait_budget(budget)
            try:
                got = ao2mo(P, C, mode=getattr(_lib, mode))
            except _lib.PQError as e:
                assert e.status == _lib.PQ_TIMEOUT
            else:
                assert budget > 1 and torch.equal(got, want)
    finally:
        L.pq_debug_set_wait_budget(0)
    assert torch.equal(ao2mo(P, C, mode=getattr(_lib, mode)), want)
