"""Adjoint walks at the sizes where their rules change: rows of 32 and 33
edges (tree edges as bits of a row or as a count), queries around a tile of
4,096 vertices, long chains, stars, and zero-gap ties on either side."""
import numpy as np
import pytest

import adds_b200 as A
from adds_b200 import graphs as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def check(g, srcs, seed=0):
    rng = np.random.default_rng(seed)
    dg = A.Graph.from_csr(g)
    dist = np.stack([O.dijkstra(g, s)[0] for s in srcs])
    seeds = rng.uniform(-1, 1, size=(len(srcs), g.n)).astype(np.float32)
    want, _ = O.adjoint(g, srcs, dist.view(np.float32), seeds)
    dd, sd = torch.from_numpy(dist.view(np.float32)).cuda(), torch.from_numpy(seeds).cuda()
    gw = torch.full((max(1, g.m),), 7.0, device="cuda")  # an empty tensor has no address
    dg.backward(srcs, dd.data_ptr(), sd.data_ptr(), gw.data_ptr())
    assert np.array_equal(gw[: g.m].cpu().numpy().view(np.uint32), want.view(np.uint32))
    dg.close()


@pytest.mark.parametrize("deg", [1, 31, 32, 33, 200])
def test_star_of_stars(deg):
    # vertex 0 has deg children, each with deg (at most 40) leaves
    k = min(deg, 40)
    src = [0] * deg + [1 + i for i in range(deg) for _ in range(k)]
    dst = list(range(1, 1 + deg)) + list(range(1 + deg, 1 + deg + deg * k))
    w = np.random.default_rng(deg).uniform(0.1, 2, len(src))
    check(G.from_edges(1 + deg + deg * k, src, dst, w, G.F32), [0, 1])


@pytest.mark.parametrize("n", [1, 2, 4095, 4096, 4097, 9000])
def test_chain_with_rungs(n):
    # a chain whose every third vertex has a second way that ties or loses
    src, dst = list(range(n - 1)), list(range(1, n))
    src += list(range(0, n - 2, 3))
    dst += list(range(2, n, 3))[: len(range(0, n - 2, 3))]
    w = np.concatenate([np.ones(n - 1), np.where(np.arange(len(src) - (n - 1)) % 2, 2.0, 2.5)])
    check(G.from_edges(n, src, dst, w, G.F32), [0, n // 2])


@pytest.mark.parametrize("extra", [0, 40])
def test_zero_gap_ties(extra):
    # zero-weight cycles; `extra` parallel edges lengthen a row past 32
    src, dst = [0, 1, 2, 2, 3, 3], [1, 2, 1, 3, 4, 2]
    w = [1.0, 0.0, 0.0, 0.0, 2.0, 0.0]
    src += [2] * extra
    dst += [4] * extra
    w += [9.0] * extra
    check(G.from_edges(5, src, dst, w, G.F32), [0, 3])


def test_grids_around_a_tile():
    for x, y in ((63, 65), (64, 64), (1, 5000), (150, 90)):
        g = G.grid(x, y, 0.05, 8, wtype=G.F32, seed=x)
        check(g, [0, g.n - 1, g.n // 3], seed=y)
