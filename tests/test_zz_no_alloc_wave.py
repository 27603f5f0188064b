"""The no-allocation entry point on both of its paths: the wave kernels, and
the phase engine where their lists overflow, at the limits of the scratch
array and with rows that are cut into pieces."""
import numpy as np
import pytest

from adds_b200 import _lib as L
from adds_b200 import graphs as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def solve(g, src):
    import torch
    row = torch.from_numpy(g.row.astype(np.uint32).view(np.int32)).cuda()
    edges = torch.from_numpy(np.stack([g.dst, g.w], 1).astype(np.uint32).view(np.int32).copy()).cuda()
    out = torch.empty(g.n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    L.check(L.lib().adds_sssp_noalloc(g.n, g.m, row.data_ptr(), edges.data_ptr() if g.m else None,
                                      g.wtype, src, out.data_ptr(), None), "adds_sssp_noalloc")
    return out.cpu().numpy().view(np.uint32)


def wide(n, wtype):
    # a star, and 20 hubs that each reach everything: the frontier is the graph
    src = np.concatenate([np.zeros(n - 1, np.int64)] + [np.full(n, 1 + h) for h in range(10)])
    dst = np.concatenate([np.arange(1, n)] + [np.arange(n)] * 10)
    w = np.random.default_rng(n).integers(1, 9, src.size)
    return G.from_edges(n, src, dst, w, wtype)


@pytest.mark.parametrize("wtype", [G.I32, G.F32])
def test_sizes_and_overflow(wtype):
    w = dict(wtype=wtype, w_lo=1, w_hi=1000)
    cases = [(G.from_edges(1, [], [], [], wtype), 0), (G.from_edges(2, [0], [1], [3], wtype), 0),
             (G.rmat(14, 16, seed=1, **w), 7), (G.grid(90, 70, 0.02, 8, seed=2, **w), 3000),
             (G.erdos_renyi(50001, 8, seed=3, **w), 50000), (wide(1 << 20, wtype), 0)]
    for g, s in cases + cases[:3]:  # the last ones after a large and an overflowing one
        assert np.array_equal(solve(g, s), O.dijkstra(g, s)[0]), (g.n, g.m)


def test_minus_zero_weights():
    g = G.grid(30, 20, 0.0, 8, wtype=G.F32, seed=5)
    w = g.w.view(np.float32).copy()
    w[::3] = -0.0
    neg = G.CSR(g.n, g.row, g.dst, w.view(np.uint32), G.F32)
    pos = G.CSR(g.n, g.row, g.dst, np.abs(w).view(np.uint32), G.F32)
    assert np.array_equal(solve(neg, 4), O.dijkstra(pos, 4)[0])
