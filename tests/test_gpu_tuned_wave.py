"""A tuned graph runs the configuration that was timed: where a wave kernel was
the fastest, its own width and its own number of CTAs, not the knobs that the
tuner found for an engine."""
import numpy as np
import pytest

import adds_b200 as A
from adds_b200 import graphs as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu
ASYNC, PHASE = 1, 2
GRAPHS = {"grid": lambda: G.grid(260, 200, 0.02, 8, wtype=G.F32, w_lo=1.0, w_hi=100.0, seed=22),
          "er": lambda: G.erdos_renyi(4001, 8, seed=3),
          "rmat": lambda: G.rmat(15, 16, seed=21, w_hi=10000)}


def ctas_of(wave):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return {1: 1, 2: 1, 3: sms, 4: sms}[wave]


@pytest.mark.parametrize("kind", list(GRAPHS))
def test_tuned_solves_run_what_was_timed(kind):
    g = GRAPHS[kind]()
    dg, fresh = A.Graph.from_csr(g), A.Graph.from_csr(g)
    untuned = fresh.sssp(77)[1]
    best, ms = dg.tune([5, 900])
    assert ms > 0 and best.delta_shift >= 0 and best.engine in (ASYNC, PHASE)
    want = O.dijkstra(g, 77)[0]
    a, sa = dg.sssp(77)                # tuned
    b, sb = dg.sssp(77, best)          # the same, named
    c, sc = fresh.sssp(77, best)       # the same on a graph that was never tuned
    for d, st in ((a, sa), (b, sb), (c, sc)):
        assert np.array_equal(d, want)
        assert st["engine"] == best.engine and st["delta_shift"] == best.delta_shift
    assert sa["ctas"] == sb["ctas"] == sc["ctas"]
    if kind == "grid":
        assert best.wave > 0  # some times faster than either engine here
    if best.wave > 0:
        # timed with every SM, rows laid out and widths chosen as an untuned solve does
        assert best.group_ctas == 0 and best.light_heavy == -1 and best.pull == 0
        assert sa["ctas"] == ctas_of(best.wave)
        if untuned["ctas"] == sa["ctas"]:
            assert untuned["delta_shift"] == best.delta_shift
        # the engine's knobs stay the graph's for a call that names an engine
        d, st = dg.sssp(77, A.default_opts(engine=PHASE))
        assert np.array_equal(d, want) and st["engine"] == PHASE
    # a time-out and a stream of the caller's leave the choice with the tuner
    d, st = dg.sssp(77, A.default_opts(timeout_ms=5000))
    assert np.array_equal(d, want) and st["ctas"] == sa["ctas"]
    fresh.close()
    dg.close()
