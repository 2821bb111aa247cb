"""pfsoft_cuda_dsoft_noalloc builds a bandwidth's tables once: a recording holds the call's three launches and nothing
that builds tables, whatever bandwidths ran in between and also where it is the bandwidth's first call, and
gives pfsoft_cuda_dsoft's result in any order of calls and replays."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

REL_TOL = 1e-13


class _Case:
    def __init__(self, lib, B):
        g = torch.Generator(device="cuda")
        g.manual_seed(B)
        self.lib, self.B = lib, B
        self.grid = torch.randn((2 * B,) * 3, dtype=torch.complex128, device="cuda", generator=g)
        self.want = torch.empty(B * (4 * B * B - 1) // 3, dtype=torch.complex128, device="cuda")
        self.out = torch.empty_like(self.want)
        s = torch.cuda.current_stream().cuda_stream
        assert lib.pfsoft_cuda_dsoft(self.grid.data_ptr(), B, self.want.data_ptr(), None, 0, s) == 0

    def call(self, stream=None):
        s = (stream or torch.cuda.current_stream()).cuda_stream
        assert self.lib.pfsoft_cuda_dsoft_noalloc(self.grid.data_ptr(), self.B, self.out.data_ptr(), s) == 0

    def record(self, graph):
        torch.cuda.synchronize()
        side = torch.cuda.Stream()
        with torch.cuda.graph(graph, stream=side):
            self.call(side)
        return graph

    def check(self, run):
        self.out.fill_(complex("nan"))
        run()
        torch.cuda.synchronize()
        err = torch.linalg.vector_norm(self.out - self.want) / torch.linalg.vector_norm(self.want)
        assert err.item() <= REL_TOL, self.B


def _nodes(graph):
    n = ctypes.c_size_t()
    assert ctypes.CDLL("libcuda.so.1").cuGraphGetNodes(ctypes.c_void_p(graph.raw_cuda_graph()), None, ctypes.byref(n)) == 0
    return n.value


@pytest.mark.parametrize("B", [4, 16, 30, 32])
def test_recording_after_a_direct_call_builds_no_tables(lib, B):
    case, other = _Case(lib, B), _Case(lib, 9)
    case.check(case.call)
    other.check(other.call)
    graph = case.record(torch.cuda.CUDAGraph(keep_graph=True))
    assert _nodes(graph) <= 3
    other.check(other.call)
    case.check(graph.replay)
    case.check(case.call)


def test_recording_before_the_first_direct_call(lib):
    small = _Case(lib, 2)
    small.check(small.call)   # the device's first call
    a, b = _Case(lib, 23), _Case(lib, 27)   # no other test's bandwidths
    ga, gb = a.record(torch.cuda.CUDAGraph()), b.record(torch.cuda.CUDAGraph())
    for _ in range(2):
        a.check(ga.replay)
        b.check(gb.replay)
        a.check(a.call)
        small.check(small.call)
        a.check(ga.replay)
        b.check(b.call)


@pytest.mark.parametrize("B", [11, 29])   # no other test's bandwidths
def test_first_call_in_a_recording_builds_beside_it(lib, B):
    small, case = _Case(lib, 2), _Case(lib, B)
    small.check(small.call)   # the device's first call
    graph = case.record(torch.cuda.CUDAGraph(keep_graph=True))
    assert _nodes(graph) <= 3
    small.check(small.call)
    case.check(graph.replay)
    case.check(case.call)
