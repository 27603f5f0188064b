"""The work users of this framework have it do, as cases that can be timed.

Shortest paths are asked for one source at a time (a service, the drop-in
command), for a list of sources, for many small problems at once, and inside
a training step that needs the gradient of the distances.  Graphs are R-MAT
(social and web graphs), Erdos-Renyi, and grids with a few shortcuts (road
networks); weights are int32 or float32.  Every call leaves the options on
automatic, as a program that has not been tuned does.

Inputs are made on the GPU with torch from the seed alone.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import adds_b200 as A
from adds_b200 import graphs as G
from adds_b200.autograd import batched_sssp

INF_I = 0x7FFFFFFF
INF_F = 3.4028234663852886e38  # FLT_MAX
DEV = "cuda"


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # one small query of a service: the latency of a call
        {"name": "small_er", "kind": "plain", "graph": "er", "n": 4001, "ef": 8,
         "float": False, "hi": 1000, "sources": 1, "out": "host"},
        # one city's road network, float lengths, answer to the host
        {"name": "small_road", "kind": "plain", "graph": "road", "x": 517, "y": 301,
         "float": True, "lo": 1, "hi": 100, "sources": 1, "out": "host"},
        # the repository's R-MAT 16 configuration: a middling graph, one source
        {"name": "rmat16", "kind": "plain", "graph": "rmat", "scale": 16, "ef": 16,
         "float": False, "hi": 1000, "sources": 1, "out": "host"},
        # a list of sources on one graph, each answer to pinned host memory
        {"name": "rmat20_sources", "kind": "plain", "graph": "rmat", "scale": 20, "ef": 16,
         "float": False, "hi": 1000, "sources": 8, "out": "pinned"},
        # float weights U[0,1), the weights of the repository's R-MAT 26
        # configuration, answers kept on the GPU
        {"name": "rmat22_float", "kind": "plain", "graph": "rmat", "scale": 22, "ef": 16,
         "float": True, "lo": 0, "hi": 1, "sources": 2, "out": "device"},
        # the benchmark's default workload: one large graph
        {"name": "rmat24", "kind": "plain", "graph": "rmat", "scale": 24, "ef": 16,
         "float": False, "hi": 10000, "sources": 1, "out": "device"},
        # the repository's road-like configuration: many thin wave fronts
        {"name": "road4096", "kind": "plain", "graph": "road", "x": 4096, "y": 4096,
         "float": True, "lo": 1, "hi": 100, "sources": 1, "out": "device"},
        # the repository's batched configuration: 192 Erdos-Renyi graphs of
        # very different sizes and 64 sources on one R-MAT graph
        {"name": "batch_mixed", "kind": "batch", "er": 192, "n_lo": 1000, "n_hi": 1000000,
         "scale": 20, "rmat_sources": 64, "float": False, "hi": 1000},
        # routes from 60 depots on one road network, new depots each call
        {"name": "batch_routes", "kind": "routes", "x": 257, "y": 255, "sources": 60,
         "float": False, "lo": 1, "hi": 100},
        # the repository's differentiable configuration: forward and backward
        # over 128 grids with 16 sources each
        {"name": "train", "kind": "train", "grids": 128, "s_lo": 64, "s_hi": 512, "sources": 16,
         "targets": 64},
        # a small training step
        {"name": "train_small", "kind": "train", "grids": 5, "s_lo": 61, "s_hi": 130,
         "sources": 3, "targets": 20},
        # a solve for a program that owns all device memory itself
        {"name": "noalloc", "kind": "noalloc", "graph": "rmat", "scale": 16, "ef": 16,
         "float": False, "hi": 1000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plain", "plain", "plain", "batch", "routes", "train", "noalloc"])
    flt = rng.random() < 0.5
    w = {"float": flt, "lo": rng.choice([0, 1]), "hi": rng.choice([10, 100, 1000, 10000])}
    if kind in ("plain", "noalloc"):
        g = rng.choice(["er", "road", "rmat"])
        small = kind == "noalloc"  # that entry point's fixed working memory
        if g == "er":
            c = {"graph": g, "n": _log(rng, 1000, 300000 if small else 4000000),
                 "ef": rng.randint(4, 16)}
        elif g == "road":
            c = {"graph": g, "x": _log(rng, 40, 600 if small else 3000),
                 "y": _log(rng, 40, 600 if small else 3000)}
        else:
            c = {"graph": g, "scale": rng.randint(11, 18 if small else 23),
                 "ef": rng.choice([8, 12, 16, 16])}
        if not small:
            c.update(sources=rng.randint(1, 6), out=rng.choice(["host", "pinned", "device"]))
        return {"kind": kind, **c, **w}
    if kind == "batch":
        return {"kind": kind, "er": rng.randint(3, 96), "n_lo": 1000,
                "n_hi": _log(rng, 20000, 1000000), "scale": rng.randint(14, 20),
                "rmat_sources": rng.randint(1, 32), **w}
    if kind == "routes":
        return {"kind": kind, "x": _log(rng, 30, 700), "y": _log(rng, 30, 700),
                "sources": _log(rng, 2, 128), **w}
    lo = rng.randint(20, 120)
    return {"kind": "train", "grids": _log(rng, 1, 64), "s_lo": lo,
            "s_hi": rng.randint(lo, 400), "sources": rng.randint(1, 16),
            "targets": rng.randint(1, 100)}


# ---------------------------------------------------------------- inputs
def _gen(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed(seed * 1000003 + salt)


def _csr(keys, n):
    """Sorted unique edges src << 32 | dst without loops -> (row, src, dst)."""
    keys = torch.sort(keys).values
    keys = torch.unique_consecutive(keys)
    src = keys >> 32
    dst = keys & 0xFFFFFFFF
    keep = src != dst
    src, dst = src[keep], dst[keep]
    row = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(torch.bincount(src, minlength=n), 0, out=row[1:])
    return row, src, dst


def _rmat(scale, ef, gen):
    """a/b/c/d = 0.57/0.19/0.19/0.05, ef * 2^scale draws."""
    n = 1 << scale
    parts = []
    for lo in range(0, ef * n, 1 << 26):
        k = min(ef * n - lo, 1 << 26)
        key = torch.zeros(k, dtype=torch.int64, device=DEV)
        for _ in range(scale):
            u = torch.rand(k, generator=gen, device=DEV)
            s = (u >= 0.76).long()
            d = ((u >= 0.57) & (u < 0.76) | (u >= 0.95)).long()
            key = (key << 1) + (s << 32) + d
        parts.append(key)
    return n, *_csr(torch.cat(parts), n)


def _er(n, ef, gen):
    s = torch.randint(0, n, (ef * n,), generator=gen, device=DEV)
    d = torch.randint(0, n, (ef * n,), generator=gen, device=DEV)
    return n, *_csr((s << 32) | d, n)


def _grid_keys(x, y):
    v = torch.arange(x * y, device=DEV)
    vx = v % x
    parts = [(v[vx > 0] << 32) | (v[vx > 0] - 1), (v[vx < x - 1] << 32) | (v[vx < x - 1] + 1),
             (v[x:] << 32) | (v[x:] - x), (v[:x * y - x] << 32) | (v[:x * y - x] + x)]
    return parts


def _road(x, y, gen):
    """4 neighbours, and 2 % as many shortcuts within Manhattan radius 8."""
    parts = _grid_keys(x, y)
    k = int(0.02 * sum(p.numel() for p in parts))
    u = torch.randint(0, x * y, (k,), generator=gen, device=DEV)
    dx = torch.randint(-8, 9, (k,), generator=gen, device=DEV)
    dy = torch.randint(-8, 9, (k,), generator=gen, device=DEV)
    tx, ty = u % x + dx, u // x + dy
    ok = (dx.abs() + dy.abs() >= 2) & (dx.abs() + dy.abs() <= 8)
    ok &= (tx >= 0) & (tx < x) & (ty >= 0) & (ty < y)
    u, t = u[ok], (ty * x + tx)[ok]
    return x * y, *_csr(torch.cat(parts + [(u << 32) | t, (t << 32) | u]), x * y)


def _weights(c, m, gen):
    if c["float"]:
        lo, hi = float(c.get("lo", 1)), float(c["hi"])
        return lo + (hi - lo) * torch.rand(m, generator=gen, device=DEV)
    return torch.randint(c.get("lo", 1), c["hi"] + 1, (m,), generator=gen, device=DEV,
                         dtype=torch.int32)


def _inputs(c, seed, salt=0):
    """(n, row, src, dst, weights, sources) on the GPU for a case's graph."""
    gen = _gen(seed, salt)
    if c["graph"] == "rmat":
        n, row, src, dst = _rmat(c["scale"], c["ef"], gen)
    elif c["graph"] == "er":
        n, row, src, dst = _er(c["n"], c["ef"], gen)
    else:
        n, row, src, dst = _road(c["x"], c["y"], gen)
    w = _weights(c, src.numel(), gen)
    ns = c.get("sources", 1)
    has = torch.nonzero(row[1:] > row[:-1]).flatten()
    pick = torch.randperm(has.numel(), generator=gen, device=DEV)[:ns]
    return n, row, src, dst, w, [int(v) for v in has[pick].tolist()]


def _graph(c, inp):
    n, row, _, dst, w, _ = inp
    return A.Graph.from_csr(G.CSR(
        n, row.cpu().numpy().astype(np.uint64), dst.to(torch.int32).cpu().numpy().view(np.uint32),
        w.view(torch.int32).cpu().numpy().view(np.uint32), A.ADDS_F32 if c["float"] else A.ADDS_I32))


def _wt(c):
    return torch.float32 if c["float"] else torch.int32


def _spread(lo, hi, k):
    """k whole numbers spread over [lo, hi], evenly in their logarithm."""
    return [int(round(lo * (hi / lo) ** ((i + 0.5) / k))) for i in range(k)]


def _batch_graphs(c):
    """The graphs of a batch as one-graph cases, with the sources on each."""
    w = {k: c[k] for k in ("float", "lo", "hi") if k in c}
    for n in _spread(c["n_lo"], c["n_hi"], c["er"]):
        yield {"graph": "er", "n": n, "ef": 8, "sources": 1, **w}
    yield {"graph": "rmat", "scale": c["scale"], "ef": 16, "sources": c["rmat_sources"], **w}


def _batch_members(c, seed):
    """Its graphs, made by the framework's generator (hundreds of uploads
    from the host would take longer than all the timing), and sources that
    have an edge."""
    gen = _gen(seed)
    for i, gc in enumerate(_batch_graphs(c)):
        g = A.Graph.generate(A.gen_spec(
            gc["graph"], n=gc.get("n", 0), scale=gc.get("scale", 0), edge_factor=gc["ef"],
            wtype=A.ADDS_F32 if c["float"] else A.ADDS_I32, w_lo=c.get("lo", 1), w_hi=c["hi"],
            seed=1000 * seed + i))
        row = np.empty(g.n + 1, dtype=np.uint64)
        A.check(A.lib().adds_graph_download(g.handle, row.ctypes.data, None, None))
        row = torch.from_numpy(row.astype(np.int64)).to(DEV)
        has = torch.nonzero(row[1:] > row[:-1]).flatten()
        pick = torch.randperm(has.numel(), generator=gen, device=DEV)[:gc["sources"]]
        yield g, [int(v) for v in has[pick].tolist()]


def _square(s):
    """A plain s x s grid as its CSR: (row, src, dst)."""
    return _csr(torch.cat(_grid_keys(s, s)), s * s)


def _train_inputs(c, seed):
    """Per grid: side, weights, sources, targets and their coefficients."""
    gen = _gen(seed)
    for s in _spread(c["s_lo"], c["s_hi"], c["grids"]):
        m = 4 * s * (s - 1)
        w = torch.nn.functional.softplus(torch.randn(m, generator=gen, device=DEV))
        srcs = torch.randperm(s * s, generator=gen, device=DEV)[:c["sources"]].tolist()
        t = torch.randperm(s * s, generator=gen, device=DEV)[:c["targets"]]
        yield s, w, srcs, t, torch.rand(t.numel(), generator=gen, device=DEV)


def _padding(b):
    """Indices of the words between the queries of a batch's flat distances."""
    off = b.layout()[0].astype(np.int64)
    end = off + np.array([g.n for g in b.graphs])
    gaps = [np.arange(e, o) for e, o in zip(end[:-1], off[1:])]
    return torch.from_numpy(np.concatenate(gaps) if gaps else np.zeros(0, np.int64)).to(DEV)


def prepare(case, seed):
    c, st = case, {"case": case}
    if c["kind"] == "plain":
        inp = _inputs(c, seed)
        st["g"], st["srcs"] = _graph(c, inp), inp[5]
        n, ns = inp[0], len(inp[5])
        if c["out"] == "host":
            st["outs"] = [np.empty(n, dtype=np.float32 if c["float"] else np.int32)
                          for _ in range(ns)]
        elif c["out"] == "pinned":
            st["outs"] = [torch.empty(n, dtype=_wt(c), pin_memory=True) for _ in range(ns)]
        else:
            st["outs"] = [torch.empty(n, dtype=_wt(c), device=DEV) for _ in range(ns)]
    elif c["kind"] == "noalloc":
        n, row, _, dst, w, srcs = _inputs(c, seed)
        st["row"] = row.to(torch.int32)
        st["edges"] = torch.stack([dst.to(torch.int32), w.view(torch.int32)], 1).contiguous()
        st["n"], st["src"] = n, srcs[0]
        st["out"] = torch.empty(n, dtype=_wt(c), device=DEV)
    elif c["kind"] in ("batch", "routes"):
        gs, srcs = [], []
        if c["kind"] == "routes":
            inp = _inputs({"graph": "road", **c}, seed)
            gs, srcs = [_graph(c, inp)] * len(inp[5]), inp[5]
        else:
            for g, own in _batch_members(c, seed):
                gs += [g] * len(own)
                srcs += own
        st["b"], st["srcs"] = A.Batch(gs, srcs), srcs
        st["out"] = torch.empty(int(st["b"].layout()[1]), dtype=_wt(c), device=DEV)
        st["pad"] = _padding(st["b"])
    else:
        gs, qg, qs, ws, tq, tc = [], [], [], [], [], []
        for s, w, srcs, t, coef in _train_inputs(c, seed):
            g = A.Graph.generate(A.gen_spec("plain_grid", side=s, wtype=A.ADDS_F32, w_lo=1.0,
                                            w_hi=2.0, seed=1))
            torch.cuda.synchronize()
            g.set_weights(w)
            gs.append(g)
            qg += [g] * len(srcs)
            qs += srcs
            ws.append(w)
            tq += [t] * len(srcs)
            tc += [coef] * len(srcs)
        b = A.Batch(qg, qs)
        off = b.layout()[0].astype(np.int64)
        st["b"], st["graphs"] = b, gs
        st["w"] = torch.cat(ws).requires_grad_(True)
        st["sizes"] = [w.numel() for w in ws]
        st["target"] = torch.cat([t + int(o) for t, o in zip(tq, off)])
        st["coef"] = torch.cat(tc)
        st["pad"] = _padding(b)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return st


# ---------------------------------------------------------------- one pass
def run(state):
    c = state["case"]
    if c["kind"] == "plain":
        if len(state["srcs"]) == 1:
            state["g"].sssp(state["srcs"][0], out=state["outs"][0])
        else:
            state["g"].sssp_sources(state["srcs"], state["outs"])
        return state["outs"]
    if c["kind"] == "noalloc":
        stream = torch.cuda.current_stream().cuda_stream
        A.check(A.lib().adds_sssp_noalloc(
            state["n"], state["edges"].shape[0], state["row"].data_ptr(),
            state["edges"].data_ptr(), A.ADDS_F32 if c["float"] else A.ADDS_I32, state["src"],
            state["out"].data_ptr(), stream), "adds_sssp_noalloc")
        return state["out"]
    b = state["b"]
    if c["kind"] in ("batch", "routes"):
        if c["kind"] == "routes":
            b.set_sources(state["srcs"])
        b.run()
        b.dist_all(state["out"])
        return state["out"].index_fill_(0, state["pad"], 0)
    flat = batched_sssp(b, state["graphs"], list(state["w"].split(state["sizes"])))
    loss = (flat[state["target"]] * state["coef"]).sum()
    grad, = torch.autograd.grad(loss, state["w"])
    return {"dist": flat.detach().index_fill_(0, state["pad"], 0), "grad": grad}


# ---------------------------------------------------------------- its work
def _edges(c):
    if c["graph"] == "road":
        return int(4.15 * c["x"] * c["y"])
    return c["ef"] * (c["n"] if c["graph"] == "er" else 1 << c["scale"])


def _vertices(c):
    return {"er": lambda: c["n"], "rmat": lambda: 1 << c["scale"],
            "road": lambda: c["x"] * c["y"]}[c["graph"]]()


def work(case):
    """The graph read once, every distance written once; one addition for
    each edge of each solve.  A training step also reads a gradient for each
    distance and writes one for each weight."""
    c = case
    if c["kind"] == "train":
        n = m = 0
        for s in _spread(c["s_lo"], c["s_hi"], c["grids"]):
            n, m = n + s * s, m + 4 * s * (s - 1)
        return {"bytes": 4 * n + 12 * m + 8 * n * c["sources"], "flops": 2 * m * c["sources"]}
    one = {"batch": lambda: list(_batch_graphs(c)), "routes": lambda: [{"graph": "road", **c}]}
    b = f = 0
    for gc in one.get(c["kind"], lambda: [c])():
        n, m, ns = _vertices(gc), _edges(gc), gc.get("sources", 1)
        b, f = b + 4 * n + 8 * m + 4 * n * ns, f + m * ns
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------- in 64 bits
def _relax(n, src, dst, w, source, inf):
    """Bellman-Ford with 64-bit distances."""
    big = math.inf if w.dtype == torch.float64 else 1 << 62
    d = torch.full((n,), big, dtype=w.dtype, device=DEV)
    d[source] = 0
    while True:
        before = d.clone()
        for _ in range(4 if n < (1 << 20) else 1):
            t = d[src]
            cand = torch.where(t == big, big, t + w)
            d = d.scatter_reduce(0, dst, cand, "amin")
        if torch.equal(before, d):
            return torch.where(d == big, inf, d)


def _exact_graph(c, inp):
    n, _, src, dst, w, srcs = inp
    w = w.double() if c["float"] else w.long()
    return [_relax(n, src, dst, w, s, INF_F if c["float"] else INF_I) for s in srcs]


def _flat(dists):
    """Distances of the queries laid out as a batch does: 32-word multiples."""
    out = []
    for i, d in enumerate(dists):
        out.append(d)
        if i + 1 < len(dists):
            out.append(torch.zeros(-d.numel() % 32, dtype=d.dtype, device=DEV))
    return torch.cat(out)


def exact(case, seed):
    c = case
    if c["kind"] == "plain" or c["kind"] == "noalloc":
        if c["graph"] == "road" and c["x"] * c["y"] > 1 << 20:
            return None  # thousands of rounds
        d = _exact_graph(c, _inputs(c, seed))
        return d if c["kind"] == "plain" else d[0]
    if c["kind"] in ("batch", "routes"):
        if c["kind"] == "routes":
            if c["x"] * c["y"] * c["sources"] > 1 << 23:
                return None  # too many rounds
            return _flat(_exact_graph(c, _inputs({"graph": "road", **c}, seed)))
        dists = []
        for g, srcs in _batch_members(c, seed):
            csr = g.download()
            row = torch.from_numpy(csr.row.astype(np.int64)).to(DEV)
            src = torch.repeat_interleave(torch.arange(g.n, device=DEV), row[1:] - row[:-1])
            dst = torch.from_numpy(csr.dst.astype(np.int64)).to(DEV)
            w = torch.from_numpy(csr.weights().copy()).to(DEV)
            dists += _exact_graph(c, (g.n, row, src, dst, w, srcs))
            g.close()
        return _flat(dists)
    if c["grids"] * c["sources"] * c["s_hi"] > 1 << 14:
        return None
    dists = []
    for s, w, srcs, _, _ in _train_inputs(c, seed):
        _, src, dst = _square(s)
        dists += [_relax(s * s, src, dst, w.double(), x, INF_F) for x in srcs]
    # the gradient follows one shortest path tree among equal ones: no value
    return {"dist": _flat(dists), "grad": None}
