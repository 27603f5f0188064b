"""Batches whose wave lists overflow, through launch and sync: the batch moves
to an engine whose pool grows, as run does, with the sources that were
launched."""
import numpy as np
import pytest

import adds_b200 as A
from adds_b200 import graphs as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pair():
    leaves = 300000
    g = G.from_edges(leaves + 1, np.zeros(leaves, np.int64), np.arange(1, leaves + 1),
                     np.full(leaves, 3))
    r = G.grid(50, 50, 0.0, 8, wtype=G.I32, w_lo=1, w_hi=9, seed=1)
    dg, dr = A.Graph.from_csr(g), A.Graph.from_csr(r)
    yield g, r, dg, dr
    dg.close()
    dr.close()


def right(b, g, r, star, grid):
    assert np.array_equal(b.dist(0), O.dijkstra(g, star)[0])
    assert np.array_equal(b.dist(1), O.dijkstra(r, grid)[0])
    assert np.array_equal(b.dist(179), O.dijkstra(g, 1)[0])


def test_launch_and_sync_after_an_overflow(pair):
    g, r, dg, dr = pair
    b = A.Batch([dg, dr, dg] * 60, [0, 7, 1] * 60)
    b.launch()
    assert b.sync()["retries"] == 1
    right(b, g, r, 0, 7)
    for _ in range(2):  # from then on the engine
        b.launch()
        assert b.sync()["retries"] == 0
        right(b, g, r, 0, 7)
    b.close()


def test_run_counts_the_move(pair):
    g, r, dg, dr = pair
    b = A.Batch([dg, dr, dg] * 60, [0, 7, 1] * 60)
    assert b.run()["retries"] == 1
    assert b.run()["retries"] == 0
    right(b, g, r, 0, 7)
    b.close()


def test_sources_changed_before_the_sync(pair):
    """The launch had the old sources: its overflow is met with those, and the
    next launch has the new ones."""
    g, r, dg, dr = pair
    b = A.Batch([dg, dr, dg] * 60, [0, 7, 1] * 60)
    b.launch()
    b.set_sources([2, 9, 1] * 60)
    b.sync()
    right(b, g, r, 0, 7)
    b.launch()
    b.sync()
    right(b, g, r, 2, 9)
    b.close()
