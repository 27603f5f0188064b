"""Several owners of one graph: batches and plain solves whose buckets have
different widths, so each marks the light edges of a row elsewhere.  Whatever
the others did in between, or do at the same time, a batch's distances are the
oracle's."""
import numpy as np
import pytest

import adds_b200 as A
from adds_b200 import graphs as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu
ASYNC, PHASE, POOL = 1, 2, 4


def graph(wtype, seed=21):
    g = G.rmat(14, 16, wtype=wtype, w_lo=1, w_hi=1000, seed=seed)
    return g, G.max_degree_vertex(g)


def weights(g, hi, seed):
    w = np.random.default_rng(seed).integers(1, hi + 1, g.m)
    w = w.astype(np.float32).view(np.uint32) if g.wtype == G.F32 else w.astype(np.uint32)
    return G.CSR(g.n, g.row, g.dst, w, g.wtype)


def right(b, g, srcs):
    for q, s in enumerate(srcs):
        assert np.array_equal(b.dist(q), O.dijkstra(g, s)[0]), (q, s)


def opts(**kw):
    return A.default_opts(timeout_ms=20000, **kw)


KINDS = {"pooled": dict(wave=POOL, light_heavy=1, pull=1), "phase": dict(engine=PHASE, pull=1),
         "async": dict(engine=ASYNC)}


@pytest.mark.parametrize("wtype", [G.I32, G.F32])
@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("nq", [1, 9])
def test_plain_solves_of_other_widths_between_runs(wtype, kind, nq):
    g, top = graph(wtype)
    srcs = ([top] + list(range(1, 16000, 1900)))[:nq]
    dg = A.Graph.from_csr(g)
    b = A.Batch([dg] * nq, srcs, opts(**KINDS[kind]))
    b.run()
    right(b, g, srcs)
    for shift in (2, 12, 5) if wtype == G.I32 else (9, 20, 12):
        for kw in (KINDS["pooled"], KINDS["phase"]):
            d, _ = dg.sssp(7, opts(delta_shift=shift, **kw))
            assert np.array_equal(d, O.dijkstra(g, 7)[0])
            b.run()
            right(b, g, srcs)
    b.close()
    dg.close()


@pytest.mark.parametrize("wtype", [G.I32, G.F32])
def test_weights_then_plain_solve_then_batch(wtype):
    """The batch keeps the width it was made with; a plain solve after an update
    to much smaller weights takes one of its own."""
    g, top = graph(wtype)
    srcs = [top, 3, 800, 9000]
    dg = A.Graph.from_csr(g)
    b = A.Batch([dg] * 4, srcs, opts(**KINDS["pooled"]))
    b.run()
    n = weights(g, 300, 1)
    dg.set_weights(n.w)
    b.run()
    right(b, n, srcs)
    for kw in (KINDS["pooled"], KINDS["phase"], {}):
        d, _ = dg.sssp(5, opts(**kw))
        assert np.array_equal(d, O.dijkstra(n, 5)[0])
        b.run()
        right(b, n, srcs)
    b.close()
    dg.close()


@pytest.mark.parametrize("wtype", [G.I32, G.F32])
def test_batches_of_two_widths(wtype):
    """In turn, and both in flight with plain solves beside them."""
    g, top = graph(wtype, 22)
    srcs = [top, 11, 5000]
    dg = A.Graph.from_csr(g)
    lo, hi = (3, 9) if wtype == G.I32 else (10, 17)
    bs = [A.Batch([dg] * 3, srcs, opts(delta_shift=s, group_ctas=20, **KINDS["pooled"])) for s in (lo, hi)]
    want = [O.dijkstra(g, s)[0] for s in srcs]
    for _ in range(2):
        for b in bs:
            b.run()
            for q in range(3):
                assert np.array_equal(b.dist(q), want[q])
    for turn in range(10):
        for b in bs:
            b.launch()
        d, _ = dg.sssp(srcs[1], opts(delta_shift=(lo, hi)[turn & 1] + 1, group_ctas=20, **KINDS["pooled"]))
        for b in bs:
            b.sync()
        assert np.array_equal(d, want[1])
        for b in bs:
            for q in range(3):
                assert np.array_equal(b.dist(q), want[q]), turn
    for b in bs:
        b.close()
    dg.close()


@pytest.mark.parametrize("wtype", [G.I32, G.F32])
def test_automatic_options(wtype):
    """Every option automatic: the plain solve's width follows the new weights
    and the batch's does not.  Against the phase engine on whole rows, which
    uses no split."""
    dg = A.Graph.generate(A.gen_spec("rmat", scale=19, wtype=wtype, w_lo=1, w_hi=10000, seed=3))
    rng = np.random.default_rng(1)
    srcs = [0] + [int(x) for x in rng.integers(0, dg.n, 63)]
    b = A.Batch([dg] * 64, srcs)
    b.run()
    w = rng.integers(1, 301, dg.m)
    dg.set_weights(w.astype(np.float32).view(np.uint32) if wtype == G.F32 else w.astype(np.uint32))
    some = range(0, 64, 4)
    want = {q: dg.sssp(srcs[q], opts(engine=PHASE, light_heavy=0))[0] for q in some}
    for beside in (False, False, True, True, True):
        if beside:
            b.launch()
            dg.sssp(5, opts(delta_shift=6, light_heavy=1))
            dg.sssp(5)
            b.sync()
        else:
            b.run()
            dg.sssp(5)
        for q in some:
            assert np.array_equal(b.dist(q), want[q]), (q, beside)
    b.close()
    dg.close()
