"""device_bytes counts what a graph holds on the GPU, its solvers' lists
among it."""
import ctypes as C

import pytest

import adds_b200 as A
from adds_b200 import _lib as L
from adds_b200 import graphs as G

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def held(dg):
    info = L.GraphInfo()
    L.check(L.lib().adds_graph_info(dg.handle, C.byref(info)), "adds_graph_info")
    return info.device_bytes


@pytest.mark.parametrize("kw", [{}, dict(engine=1), dict(engine=2), dict(wave=4)])
def test_lists_are_counted(kw):
    g = G.rmat(16, 16, seed=1)
    warm = A.Graph.from_csr(g)  # kernels' local memory is the device's, not a graph's
    warm.sssp(1, A.default_opts(**kw))
    warm.close()
    dg = A.Graph.from_csr(g)
    torch.cuda.synchronize()
    before, free0 = held(dg), torch.cuda.mem_get_info()[0]
    dg.sssp(1, A.default_opts(**kw))
    grew, took = held(dg) - before, free0 - torch.cuda.mem_get_info()[0]
    # some twenty allocations, each rounded up to at most 2 MB, or placed in
    # what the rounding of an earlier one left
    assert abs(grew - took) <= 48 << 20
    assert grew > 0
    dg.close()
