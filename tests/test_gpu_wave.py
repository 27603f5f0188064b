"""The wave kernels (one CTA or a group of CTAs per query, near-far lists)
against the oracle, at the sizes and shapes where they can go wrong: frontiers
that leave shared memory, rows around the length that is cut into pieces,
groups of one CTA and of uneven size, thresholds of one unit and past every
distance, equal paths, sums past INT32_MAX, and lists that overflow."""
import numpy as np
import pytest

import adds_b200 as A
from adds_b200 import graphs as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu
CTA, WIDE, GROUP, POOL = 1, 2, 3, 4
PIECE = 512  # edges of a long row per entry (wave_internal.h)


def check(g, srcs, **kw):
    dg = A.Graph.from_csr(g)
    try:
        st = None
        for s in srcs:
            d, st = dg.sssp(int(s), A.default_opts(timeout_ms=10000, **kw))
            assert np.array_equal(d, O.dijkstra(g, int(s))[0]), (s, kw)
        return st
    finally:
        dg.close()


def star(rows, wtype=G.I32, seed=0):
    """Vertex i has rows[i] edges to leaves of its own; the centres form a
    path."""
    src, dst, k = [], [], len(rows)
    for i, r in enumerate(rows):
        src += [i] * r + ([i] if i + 1 < len(rows) else [])
        dst += list(range(k, k + r)) + ([i + 1] if i + 1 < len(rows) else [])
        k += r
    w = np.random.default_rng(seed).integers(1, 50, size=len(src))
    return G.from_edges(k, src, dst, w.astype(np.float32) if wtype == G.F32 else w, wtype)


@pytest.mark.parametrize("wave", [CTA, WIDE, GROUP, POOL])
@pytest.mark.parametrize("wtype", [G.I32, G.F32])
def test_graph_families(wave, wtype):
    w = dict(wtype=wtype, w_lo=1, w_hi=100)
    check(G.grid(97, 61, 0.02, 8, seed=3, **w), [0, 97 * 30 + 48], wave=wave)
    check(G.erdos_renyi(3001, 8, seed=4, **w), [5, 2999], wave=wave)
    r = G.rmat(13, 16, seed=5, **w)
    assert r.degrees().max() > PIECE
    check(r, [G.max_degree_vertex(r), 77], wave=wave)


@pytest.mark.parametrize("wave", [CTA, WIDE, GROUP, POOL])
def test_rows_around_the_piece_length(wave):
    rows = [PIECE - 1, PIECE, PIECE + 1, 2 * PIECE, 2 * PIECE + 1, 7, 8, 9, 0, 5000]
    for wtype in (G.I32, G.F32):
        check(star(rows, wtype), [0, 4], wave=wave)


@pytest.mark.parametrize("wave", [GROUP, POOL])
@pytest.mark.parametrize("ctas", [1, 2, 7, 33, 148])
def test_group_sizes(wave, ctas):
    g = G.grid(80, 50, 0.02, 8, wtype=G.F32, w_lo=1.0, w_hi=100.0, seed=7)
    st = check(g, [0, 2040], wave=wave, group_ctas=ctas)
    assert st["ctas"] == ctas and st["retries"] == 0
    check(G.rmat(12, 16, seed=8), [1], wave=wave, group_ctas=ctas)


@pytest.mark.parametrize("wave", [CTA, WIDE, GROUP, POOL])
@pytest.mark.parametrize("shift", [0, 3, 20, 31])
def test_any_threshold_step(wave, shift):
    check(G.grid(40, 40, 0.02, 8, wtype=G.F32, w_lo=1.0, w_hi=100.0, seed=9), [820], wave=wave,
          delta_shift=shift)
    check(G.erdos_renyi(900, 5, seed=10), [3], wave=wave, delta_shift=shift)


@pytest.mark.parametrize("wave", [CTA, WIDE, GROUP, POOL])
def test_special_weights_and_shapes(wave):
    # equal paths everywhere: every weight 1, and zero-weight edges
    side = 64
    g = G.grid(side, side, 0.0, wtype=G.I32, w_lo=1, w_hi=1, seed=1)
    check(g, [0, side * 32 + 32], wave=wave)
    z = G.CSR(g.n, g.row, g.dst, np.zeros(g.m, np.uint32), G.I32)
    check(z, [5], wave=wave)
    # a chain, an isolated source, one vertex, self loops and double edges
    n = 3000
    check(G.from_edges(n, np.arange(n - 1), np.arange(1, n), np.full(n - 1, 7)), [0, n - 1], wave=wave)
    check(G.from_edges(1, [], [], []), [0], wave=wave)
    check(G.from_edges(3, [0, 0, 0, 1, 1], [0, 1, 1, 1, 2], [0, 9, 4, 1, 3]), [0], wave=wave)
    # sums that reach INT32_MAX are never accepted
    big = 0x7FFFFFFF
    check(G.from_edges(5, [0, 1, 0, 3], [1, 2, 3, 4], [big - 1, 1, big, 0]), [0], wave=wave)
    # infinite and very small float weights
    w = np.array([np.inf, 1e-45, 3e38, 3e38], dtype=np.float32)
    check(G.from_edges(5, [0, 0, 2, 3], [1, 2, 3, 4], w, G.F32), [0], wave=wave)


def test_automatic_choice_and_overflow():
    """Automatic knobs take a wave kernel; a frontier larger than its lists
    sends the solve to the engine that grows, with the same distances."""
    leaves = 300000
    g = G.from_edges(leaves + 1, np.zeros(leaves, np.int64), np.arange(1, leaves + 1),
                     np.full(leaves, 3))
    dg = A.Graph.from_csr(g)
    want = O.dijkstra(g, 0)[0]
    d, st = dg.sssp(0, A.default_opts(timeout_ms=10000, wave=CTA))
    assert st["retries"] == 1 and np.array_equal(d, want)
    d, st = dg.sssp(0, A.default_opts(timeout_ms=10000, wave=CTA))  # remembered
    assert st["retries"] == 0 and np.array_equal(d, want)
    dg.close()
    dg = A.Graph.from_csr(g)  # the same in the asynchronous form
    for _ in range(3):
        dg.sssp_async(0, A.default_opts(timeout_ms=10000, wave=CTA))
    dg.sync()
    assert np.array_equal(dg.last_dist(), want)
    outs = [np.empty(g.n, np.uint32) for _ in range(3)]
    dg.sssp_sources([0, 1, 0], outs)
    assert np.array_equal(outs[0], want) and np.array_equal(outs[2], want)
    dg.close()
    for g in (G.grid(70, 70, 0.02, 8, wtype=G.F32, seed=2), G.grid(30, 20, 0.0, 8, seed=2),
              G.rmat(12, 16, seed=2), G.erdos_renyi(2000, 8, seed=2)):
        dg = A.Graph.from_csr(g)
        d, st = dg.sssp(1)
        assert np.array_equal(d, O.dijkstra(g, 1)[0])
        auto = st["ctas"]
        d, st = dg.sssp(1, A.default_opts(engine=2))
        assert np.array_equal(d, O.dijkstra(g, 1)[0]) and st["ctas"] != auto
        dg.close()


@pytest.mark.parametrize("nq", [1, 5, 700])
def test_sparse_batches(nq):
    """Fewer and more queries than SMs, replayed, with new sources and new
    weights between the runs."""
    rng = np.random.default_rng(nq)
    gs = [G.grid(20 + 7 * i, 15 + 5 * i, 0.02, 8, wtype=G.F32, seed=i) for i in range(5)]
    dgs = [A.Graph.from_csr(g) for g in gs]
    pick = [int(x) for x in rng.integers(0, len(gs), size=nq)]
    b = A.Batch([dgs[p] for p in pick], [int(rng.integers(0, gs[p].n)) for p in pick])
    for turn in range(3):
        srcs = [int(rng.integers(0, gs[p].n)) for p in pick]
        b.set_sources(srcs)
        if turn == 2:
            for i, g in enumerate(gs):
                w = rng.uniform(0.5, 9, g.m).astype(np.float32)
                gs[i] = G.CSR(g.n, g.row, g.dst, w.view(np.uint32), G.F32)
                dgs[i].set_weights(w)
        b.run()
        b.run()
        for q in range(0, nq, max(1, nq // 60)):
            assert np.array_equal(b.dist(q), O.dijkstra(gs[pick[q]], srcs[q])[0]), (turn, q)
    b.close()
    for d in dgs:
        d.close()


def test_batch_overflow_moves_to_an_engine():
    leaves = 300000
    g = G.from_edges(leaves + 1, np.zeros(leaves, np.int64), np.arange(1, leaves + 1),
                     np.full(leaves, 3))
    r = G.grid(50, 50, 0.0, 8, wtype=G.I32, w_lo=1, w_hi=9, seed=1)
    dg, dr = A.Graph.from_csr(g), A.Graph.from_csr(r)
    b = A.Batch([dg, dr, dg] * 60, [0, 7, 1] * 60)
    for _ in range(2):
        b.run()
        assert np.array_equal(b.dist(0), O.dijkstra(g, 0)[0])
        assert np.array_equal(b.dist(1), O.dijkstra(r, 7)[0])
        assert np.array_equal(b.dist(179), O.dijkstra(g, 1)[0])
    b.close()
    dg.close()
    dr.close()


@pytest.mark.parametrize("wtype", [G.I32, G.F32])
@pytest.mark.parametrize("shift", [-1, 0, 9, 31])
def test_pooled_light_heavy(wtype, shift):
    """Rows cut at any width: light and heavy parts empty, short, and longer
    than a piece, on one CTA and on many."""
    w = dict(wtype=wtype, w_lo=1, w_hi=1000)
    r = G.rmat(13, 16, seed=6, **w)
    rows = [PIECE - 1, PIECE + 1, 2 * PIECE + 3, 3000, 5, 0, 7000]
    for ctas in (1, 5, 148):
        kw = dict(wave=POOL, light_heavy=1, delta_shift=shift, group_ctas=ctas)
        check(r, [G.max_degree_vertex(r), 11], **kw)
        check(star(rows, wtype, seed=ctas), [0], **kw)
    check(G.grid(60, 40, 0.02, 8, seed=8, **w), [7], wave=POOL, light_heavy=1, delta_shift=shift)


def test_pooled_weights_of_few_values():
    """Nearly every pending vertex falls below one raised threshold."""
    g = G.erdos_renyi(60000, 16, w_lo=1, w_hi=3, seed=9)
    for lh in (0, 1):
        st = check(g, [1, 59999], wave=POOL, light_heavy=lh)
        assert st["retries"] == 0


def test_pooled_after_weight_update():
    g = G.rmat(12, 16, seed=10)
    dg = A.Graph.from_csr(g)
    for seed in range(3):
        w = np.random.default_rng(seed).integers(1, 900 if seed else 5, g.m).astype(np.uint32)
        dg.set_weights(w)
        n = G.CSR(g.n, g.row, g.dst, w, G.I32)
        for lh in (0, 1):
            d, _ = dg.sssp(9, A.default_opts(timeout_ms=10000, wave=POOL, light_heavy=lh))
            assert np.array_equal(d, O.dijkstra(n, 9)[0])
    dg.close()


@pytest.mark.parametrize("nq,ctas", [(1, 0), (2, 0), (7, 20), (40, 0), (40, 1), (150, 3)])
@pytest.mark.parametrize("wtype", [G.I32, G.F32])
def test_batches_in_groups(nq, ctas, wtype):
    """Groups of CTAs that take several queries each, dense and sparse graphs,
    with new sources and new weights between runs."""
    rng = np.random.default_rng(nq + ctas)
    w = dict(wtype=wtype, w_lo=1, w_hi=100)
    gs = [G.rmat(11, 16, seed=1, **w), G.erdos_renyi(3000, 8, seed=2, **w),
          G.erdos_renyi(50, 6, seed=3, **w), G.rmat(13, 12, seed=4, **w),
          G.grid(50, 40, 0.02, 8, seed=5, **w)]
    dgs = [A.Graph.from_csr(g) for g in gs]
    pick = [int(x) for x in rng.integers(0, len(gs), size=nq)]
    for kw in ({}, dict(wave=POOL, light_heavy=1, group_ctas=ctas), dict(wave=GROUP, group_ctas=ctas)):
        b = A.Batch([dgs[p] for p in pick], [0] * nq, A.default_opts(timeout_ms=20000, **kw))
        for turn in range(2):
            srcs = [int(rng.integers(0, gs[p].n)) for p in pick]
            b.set_sources(srcs)
            if turn == 1:
                for i, g in enumerate(gs):
                    v = rng.integers(1, 50, g.m)
                    v = v.astype(np.float32).view(np.uint32) if wtype == G.F32 else v.astype(np.uint32)
                    gs[i] = G.CSR(g.n, g.row, g.dst, v, wtype)
                    dgs[i].set_weights(v)
            b.run()
            st = b.run()
            assert st["retries"] == 0
            for q in range(nq):
                assert np.array_equal(b.dist(q), O.dijkstra(gs[pick[q]], srcs[q])[0]), (kw, turn, q)
        b.close()
    for d in dgs:
        d.close()


@pytest.mark.parametrize("wtype", [G.I32, G.F32])
@pytest.mark.parametrize("ctas", [1, 4, 148])
def test_pulled_heavy_hops(wtype, ctas):
    """Heavy hops from the other side: fewer edges than pushing them, the same
    distances; sizes that are no multiple of a chunk, vertices without
    in-edges, unreachable ones, and new weights."""
    w = dict(wtype=wtype, w_lo=1, w_hi=1000)
    kw = dict(wave=POOL, light_heavy=1, group_ctas=ctas)
    r = G.rmat(14, 16, seed=11, **w)
    src = G.max_degree_vertex(r)
    push = check(r, [src], pull=-1, **kw)["edges_scanned"]
    pull = check(r, [src], pull=1, **kw)["edges_scanned"]
    assert pull < 0.8 * push
    for shift in (-1, 4, 9) if wtype == G.I32 else (-1, 10, 16):
        check(G.rmat(11, 24, seed=12, **w), [3, 500], pull=1, delta_shift=shift, **kw)
        check(G.erdos_renyi(4099, 12, seed=13, **w), [4098], pull=1, delta_shift=shift, **kw)
    rows = [3000, 700, 0, 5000]
    check(star(rows, wtype), [0], pull=1, **kw)
    dg = A.Graph.from_csr(r)
    for hi in (3, 700):
        v = np.random.default_rng(hi).integers(0, hi, r.m)
        v = v.astype(np.float32).view(np.uint32) if wtype == G.F32 else v.astype(np.uint32)
        dg.set_weights(v)
        d, _ = dg.sssp(src, A.default_opts(timeout_ms=10000, pull=1, **kw))
        assert np.array_equal(d, O.dijkstra(G.CSR(r.n, r.row, r.dst, v, wtype), src)[0])
    dg.close()
    small = G.rmat(12, 16, seed=14, **w)
    dg = A.Graph.from_csr(small)
    b = A.Batch([dg] * 9, list(range(0, 4050, 450)),
                A.default_opts(timeout_ms=20000, pull=1, **kw))
    for _ in range(2):
        b.run()
    for q in range(9):
        assert np.array_equal(b.dist(q), O.dijkstra(small, 450 * q)[0])
    b.close()
    dg.close()


@pytest.mark.parametrize("on_gpu", [True, False])
def test_weights_of_several_graphs_at_once(on_gpu):
    """Sizes around a tile of 4,096 edges; the mean is the one-graph call's; a
    graph named twice takes its last weights; invalid weights are refused."""
    import torch
    from adds_b200.autograd import _set_weights
    gs = [G.grid(s, 7, 0.0, 8, wtype=G.F32, seed=s) for s in (2, 40, 157, 158, 900, 6000)]
    assert any(g.m > 1 << 16 for g in gs)
    dgs = [A.Graph.from_csr(g) for g in gs]
    rng = np.random.default_rng(1)
    ws = [rng.uniform(0.5, 9, g.m).astype(np.float32) for g in gs]
    ws[1][::5] = -0.0
    put = (lambda w: torch.from_numpy(w).cuda()) if on_gpu else torch.from_numpy
    _set_weights(dgs, [put(w) for w in ws])
    for g, dg, w in zip(gs, dgs, ws):
        many = dg.avg_weight
        n = G.CSR(g.n, g.row, g.dst, np.abs(w).view(np.uint32), G.F32)
        assert np.array_equal(dg.sssp(1)[0], O.dijkstra(n, 1)[0])
        dg.set_weights(w)
        assert abs(dg.avg_weight - many) <= 1e-9 * many
    a, b = ws[4] * 2, ws[4] * 3
    _set_weights([dgs[4], dgs[0], dgs[4]], [put(a), put(ws[0]), put(b)])
    n = G.CSR(gs[4].n, gs[4].row, gs[4].dst, b.view(np.uint32), G.F32)
    assert np.array_equal(dgs[4].sssp(0)[0], O.dijkstra(n, 0)[0])
    bad = ws[3].copy()
    bad[-1] = np.nan
    with pytest.raises(A.AddsError):
        _set_weights(dgs[2:5], [put(ws[2]), put(bad), put(ws[4])])
    for d in dgs:
        d.close()


@pytest.mark.parametrize("wt,hi", [(0, 1), (0, 9), (0, 10000), (1, 1.0)])
@pytest.mark.parametrize("n", [98272, 98273, 300000])
def test_width_of_pooled_buckets(n, wt, hi):
    """Around the line from which long rows take a wider bucket, against the
    phase engine; weights all 1 and few-valued ones included."""
    rng = np.random.default_rng(n)
    m = 12 * n
    dst = rng.integers(0, n, m).astype(np.uint32)
    src = np.where(rng.random(m) < 0.05, 7, rng.integers(0, n, m)).astype(np.int64)
    w = rng.integers(1, hi + 1, m).astype(np.uint32) if wt == 0 else rng.random(m).astype(np.float32).view(np.uint32)
    order = np.argsort(src, kind="stable")
    row = np.zeros(n + 1, np.uint64)
    np.cumsum(np.bincount(src, minlength=n), out=row[1:])
    dg = A.Graph.from_csr(G.CSR(n, row, dst[order], w[order], wt))
    a, sa = dg.sssp(7)
    b, sb = dg.sssp(7, A.default_opts(engine=2))
    assert np.array_equal(a, b)
    assert sa["delta_shift"] >= sb["delta_shift"]
    assert n > 98272 or sa["delta_shift"] == sb["delta_shift"]
    dg.close()
