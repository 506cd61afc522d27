"""FP64 sigma recorded into a CUDA graph: a first call under capture allocates nothing and records the element kernel,
and a graph that was recorded with few vectors replays correctly after calls with more vectors have grown the work
memory.  1e-13 of the column's largest value, as in the tests of the paths themselves."""
import ctypes

import pytest

from cases import synthetic_ep, synthetic_fci

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-13


class Case:
    """A handle on its own stream, and a reference handle on the element kernel."""

    def __init__(self, monkeypatch, p):
        from test_gpu_sigma_path import _make

        self.stream = torch.cuda.Stream()
        self.g = _make(p, stream=self.stream.cuda_stream)
        monkeypatch.setenv("PQ_SIGMA64_GATHER", "1")
        self.r = _make(p)
        monkeypatch.delenv("PQ_SIGMA64_GATHER")
        self.n = self.g.N_dets

    def call(self, X, Y, interleaved):
        from polyquant_gb300 import _lib

        L = _lib.load()
        x, y = ctypes.c_void_p(X.data_ptr()), ctypes.c_void_p(Y.data_ptr())
        if interleaved:
            return L.pq_ci_sigma_interleaved(self.g._h, x, y, X.shape[1], _lib.PQ_FP64, ctypes.c_double(0.0))
        return L.pq_ci_sigma(self.g._h, x, self.n, X.shape[0], y, self.n, _lib.PQ_FP64)

    def block(self, k, interleaved):
        return torch.randn((self.n, k) if interleaved else (k, self.n), device="cuda", dtype=torch.float64)

    def check(self, X, Y, interleaved):
        x, y = (X, Y) if interleaved else (X.t(), Y.t())
        R = self.r.sigma(x)
        torch.cuda.synchronize()
        assert ((y - R).abs().amax(0) <= TOL * R.abs().amax(0)).all()

    def record(self, X, Y, interleaved):
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=self.stream):
            st = self.call(X, Y, interleaved)
        assert st == 0
        return graph

    def replay(self, graph, X, Y, interleaved):
        X.copy_(torch.randn_like(X))
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        self.check(X, Y, interleaved)


FCI = lambda: synthetic_fci(10, 5, 5, seed=31)
EP = lambda: synthetic_ep(33, 1, 1, 9, 1, 0, seed=32)
CISD = lambda: synthetic_fci(11, 5, 5, seed=33, ex=[2, 2, 2])


@pytest.mark.parametrize("p", [FCI, EP, CISD], ids=["fci", "two species", "cisd"])
def test_first_call_under_capture(monkeypatch, p):
    from test_gpu_sigma_path import path
    from polyquant_gb300._lib import PQ_PATH_TENSOR

    monkeypatch.setenv("PQ_TWO64_ALWAYS", "1")
    c = Case(monkeypatch, p())
    X, Y = c.block(2, True), c.block(2, True)
    graph = c.record(X, Y, True)
    assert path(c.g)[0] != PQ_PATH_TENSOR
    c.replay(graph, X, Y, True)
    # a call outside the capture builds the tables; the graph stays what it was
    Z, W = c.block(4, True), c.block(4, True)
    torch.cuda.synchronize()
    assert c.call(Z, W, True) == 0
    c.check(Z, W, True)
    c.replay(graph, X, Y, True)


@pytest.mark.parametrize("interleaved", [True, False])
@pytest.mark.parametrize("p", [FCI, EP, CISD], ids=["fci", "two species", "cisd"])
def test_graph_survives_larger_calls(monkeypatch, p, interleaved):
    monkeypatch.setenv("PQ_TWO64_ALWAYS", "1")
    c = Case(monkeypatch, p())
    graphs = []
    for k in (1, 2) if interleaved else (1, 2, 3):
        X, Y = c.block(k, interleaved), c.block(k, interleaved)
        torch.cuda.synchronize()
        assert c.call(X, Y, interleaved) == 0
        graphs.append((c.record(X, Y, interleaved), X, Y))
    Z, W = c.block(4, interleaved), c.block(4, interleaved)
    torch.cuda.synchronize()
    assert c.call(Z, W, interleaved) == 0
    c.check(Z, W, interleaved)
    for graph, X, Y in graphs:
        c.replay(graph, X, Y, interleaved)
