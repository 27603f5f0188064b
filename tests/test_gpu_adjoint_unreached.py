"""Edges of the largest finite weight, as a mask sets them: the sum rounds to
the distance of a vertex that nothing reached, which is no child of anything."""
import numpy as np
import pytest

import adds_b200 as A
from adds_b200 import graphs as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
TOP = np.finfo(np.float32).max


def check(g, srcs):
    rng = np.random.default_rng(g.m)
    dg = A.Graph.from_csr(g)
    dist = np.stack([dg.sssp(s)[0] for s in srcs])
    assert np.array_equal(dist, np.stack([O.dijkstra(g, s)[0] for s in srcs]))
    seeds = rng.uniform(0.5, 1, size=(len(srcs), g.n)).astype(np.float32)
    want, _ = O.adjoint(g, srcs, dist.view(np.float32), seeds)
    dd, sd = torch.from_numpy(dist.view(np.float32)).cuda(), torch.from_numpy(seeds).cuda()
    gw = torch.full((g.m,), 7.0, device="cuda")
    dg.backward(srcs, dd.data_ptr(), sd.data_ptr(), gw.data_ptr())
    assert np.array_equal(gw.cpu().numpy(), want)
    dg.close()


@pytest.mark.parametrize("masked", [1, 2, 40])
@pytest.mark.parametrize("kids", [0, 1, 2, 40])
def test_masked_children(masked, kids):
    # 0 -> 1 -> 2, which has `kids` children and `masked` ones out of reach
    src, dst, w = [0, 1], [1, 2], [1.0, 2.0]
    for i in range(kids):
        src.append(2), dst.append(3 + i), w.append(0.5 + i)
    for i in range(masked):
        src.append(2), dst.append(3 + kids + i), w.append(TOP)
    # zero weights between vertices that nothing reaches
    src.append(3 + kids), dst.append(2 + kids + masked), w.append(0.0)
    check(G.from_edges(3 + kids + masked, src, dst, np.array(w, np.float32), G.F32), [0, 1])


def test_masked_grid():
    g = G.grid(70, 60, 0.02, 8, wtype=G.F32, w_lo=1.0, w_hi=100.0, seed=4)
    w = g.w.view(np.float32).copy()
    w[np.random.default_rng(2).random(g.m) < 0.4] = TOP
    check(G.CSR(g.n, g.row, g.dst, w.view(np.uint32), G.F32), [0, 2000, 4199])
