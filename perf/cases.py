"""Performance cases of the decomposition library.

Each case is one piece of work a program hands to the library through its
Python front end (the thin ctypes layer over librtr.so): a decomposition of a
fresh edge list, repeated stages on a graph that stays resident, counting in
either layout, a batch of independent graphs, text input, the nucleus path and
a pool of served graphs.  The graph shapes are those of the repository's
workloads (rtrex_cuda_b200.graphgen): G(n,p) with planted cliques, Chung-Lu
with planted communities, R-MAT and stochastic block models.

listed() names the cases, draw(rng) gives another of the same ranges,
prepare(case, seed) makes what a program holds before the call, run(state) is
one pass and work(case) its irreducible bytes and operations.
"""
from __future__ import annotations

import math

import numpy as np

from rtrex_cuda_b200 import Graph, RtrError, Server, graphgen, lib


def listed():
    return [
        # one small request: a new 1K-edge graph, from host arrays to clusters (the smallest served size)
        {"name": "new_small", "op": "new", "graph": "gnp", "edges": 1003, "eps": 0.3},
        # the 10,000-vertex planted-clique graph, resident, decomposed again (another eps, a parameter study)
        {"name": "resident_cliques", "op": "resident", "graph": "gnp", "edges": 83777, "eps": 0.3},
        # the stages called one by one on a block-model graph at the paper's eps, with the weights and
        # statuses a caller inspects between them, then the expansion of the clusters (mode e)
        {"name": "stages_sbm", "op": "stages", "graph": "sbm", "edges": 20011, "eps": 0.1, "threshold": 1},
        # the co-purchase-shaped graph, a new edge list from host arrays to clusters
        {"name": "new_copurchase", "op": "new", "graph": "chung_lu", "edges": 926000, "eps": 0.3},
        # the same shape resident in device memory (the benchmark's step)
        {"name": "resident_copurchase", "op": "resident", "graph": "chung_lu", "edges": 926000, "eps": 0.3},
        # a skewed graph with hubs and long triangle lists, resident: the cascading clean at its deepest
        {"name": "resident_hubs", "op": "resident", "graph": "rmat", "edges": 203311, "eps": 0.3},
        # weighted triangle counting alone, triangle lists kept, every weight read back
        {"name": "count_lists", "op": "count", "graph": "rmat", "edges": 500009, "mode": 0},
        # counting at the size where the lists no longer fit beside other work: rows layout, perVertex read back
        {"name": "count_rows", "op": "count", "graph": "rmat_device", "scale": 19, "mode": 2},
        # independent block-model graphs of 1K to 200K edges, one new batch from host arrays to clusters
        {"name": "batch_new", "op": "batch", "graphs": 64, "eps": 0.3},
        # Escape edge-list text to a device CSR, read back
        {"name": "load_text", "op": "load", "graph": "chung_lu", "edges": 400009},
        # the truss hierarchy of a mid-sized community graph
        {"name": "nucleus_sbm", "op": "nucleus", "graph": "sbm", "edges": 30011},
        # requests over a pool of registered graphs of mixed shapes, submitted together
        {"name": "served_pool", "op": "serve", "graphs": 12, "requests": 24, "max_edges": 60000, "eps": 0.3},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["new", "new", "resident", "resident", "stages", "count", "rows", "batch", "load", "nucleus",
                     "serve"])
    eps = rng.choice([0.3, 0.3, 0.1, 0.2])
    if op in ("new", "resident"):
        shape = rng.choice(["gnp", "chung_lu", "rmat", "sbm"])
        top = {"gnp": 300000, "chung_lu": 900000, "rmat": 150000, "sbm": 200000}[shape]
        return {"op": op, "graph": shape, "edges": _log(rng, 1000, top), "eps": eps}
    if op == "stages":
        shape = rng.choice(["gnp", "sbm"])
        return {"op": op, "graph": shape, "edges": _log(rng, 1000, 100000), "eps": eps, "threshold": rng.choice([1, 2])}
    if op == "count":
        shape = rng.choice(["gnp", "chung_lu", "rmat", "sbm"])
        return {"op": op, "graph": shape, "edges": _log(rng, 1000, 450000), "mode": 0}
    if op == "rows":
        if rng.random() < 0.5:
            return {"op": "count", "graph": "rmat_device", "scale": rng.randint(14, 18), "mode": 2}
        shape = rng.choice(["gnp", "rmat"])
        return {"op": "count", "graph": shape, "edges": _log(rng, 1000, 450000), "mode": 2}
    if op == "batch":
        return {"op": op, "graphs": _log(rng, 4, 60), "eps": eps}
    if op == "load":
        return {"op": op, "graph": rng.choice(["gnp", "chung_lu", "sbm"]), "edges": _log(rng, 1000, 390000)}
    if op == "nucleus":
        return {"op": op, "graph": rng.choice(["gnp", "sbm"]), "edges": _log(rng, 1000, 30000)}
    k = rng.randint(4, 12)
    return {"op": "serve", "graphs": k, "requests": 2 * k, "max_edges": _log(rng, 8000, 60000), "eps": eps}


# Edges asked of a generator for each one kept: duplicates and sampling noise
# leave every shape at least this close to its target.
_SURPLUS = {"gnp": 1.15, "chung_lu": 1.1, "rmat": 1.3, "sbm": 1.25}


def _graph(shape, m, seed):
    """(n, u, v): a simple undirected graph of exactly m edges; n depends on the shape and m alone."""
    want = m * _SURPLUS[shape]
    for attempt in range(100):
        s = seed + 7919 * attempt
        if shape == "gnp":
            n = max(64, int(round(m / 8.35)))
            g = graphgen.gnp_cliques(n=n, p=16.7 * _SURPLUS[shape] / (n - 1), n_cliques=max(1, n // 500),
                                     clique_size=min(20, n // 4), seed=s)
        elif shape == "chung_lu":
            g = graphgen.chung_lu(n=max(64, int(round(m * 335 / 926))), target_edges=want,
                                  n_comm=max(1, int(round(m * 2000 / 926000))), seed=s)
        elif shape == "rmat":
            scale = max(8, int(round(math.log2(m / 10.0))))
            pairs = want * (1.3 + 0.3 * attempt)  # R-MAT repeats more pairs the smaller it is
            g = graphgen.rmat(scale=scale, edge_factor=max(1, int(math.ceil(pairs / (1 << scale)))), seed=s)
        else:
            g = graphgen.sbm(int(want), s)
        if g[1].size >= m:
            keep = np.sort(np.random.default_rng(seed).permutation(g[1].size)[:m])
            return g[0], np.ascontiguousarray(g[1][keep]), np.ascontiguousarray(g[2][keep])
    raise RuntimeError("no %s graph of %d edges" % (shape, m))


def _edges(case, seed):
    return _graph(case["graph"], int(case["edges"]), seed)


def _sizes(count, lo, hi):
    """`count` edge counts spread evenly over the logarithm of [lo, hi]."""
    return [int(round(lo * (hi / lo) ** ((i + 0.5) / count))) for i in range(count)]


def _text(n, u, v):
    body = np.char.add(np.char.add(u.astype("S"), b" "), v.astype("S"))
    return b"%d %d\n" % (n, u.size) + b"\n".join(body.tolist()) + b"\n"


def _check(rc):
    if rc:
        raise RtrError(rc, lib().rtr_last_error().decode())


class _Buffers:
    """Result buffers a program keeps for one graph, sized for the largest
    answer (every vertex its own cluster); the count says how much is filled."""

    def __init__(self, n):
        i64 = lambda k: np.zeros(k, np.int64)  # noqa: E731
        self.seed, self.nv, self.ne, self.cut, self.vert, self.cof = (i64(n) for _ in range(6))
        self.off = i64(n + 1)

    def clusters(self, g):
        """The clusters of the extracted graph g, in creation order."""
        k = g.num_clusters()
        _check(lib().rtr_get_clusters(g.handle, self.seed.ctypes.data, self.nv.ctypes.data, self.ne.ctypes.data,
                                      self.cut.ctypes.data, self.off.ctypes.data, self.vert.ctypes.data))
        _check(lib().rtr_get_cluster_of(g.handle, self.cof.ctypes.data))
        return {"clusters": k, "seed": self.seed, "nv": self.nv, "ne": self.ne, "cut": self.cut, "off": self.off,
                "vert": self.vert, "cluster_of": self.cof}


class _Handle(Graph):
    """Graph with its C handle, for the C ABI calls that fill kept buffers."""

    @property
    def handle(self):
        return self._h


def _pad(buf, x):
    buf[:x.size] = x
    return buf


def prepare(case, seed):
    op = case["op"]
    if op == "batch":
        sizes = np.array(_sizes(int(case["graphs"]), 1e3, 2e5))
        graphs = [_graph("sbm", int(m), 1000 * seed + i) for i, m in enumerate(sizes)]
        n = sum(g[0] for g in graphs)
        return {"case": case, "graphs": graphs, "buffers": _Buffers(n)}
    if op == "serve":
        sizes = _sizes(int(case["graphs"]), 1e3, float(case["max_edges"]))
        srv = Server(device=0, hbm_budget=16 << 30)
        ids = [srv.add_graph(*_graph("rmat" if i % 2 else "gnp", m, 1000 * seed + i)) for i, m in enumerate(sizes)]
        order = np.random.default_rng(int(case["requests"])).integers(0, len(ids), int(case["requests"]))
        return {"case": case, "server": srv, "requests": [ids[i] for i in order]}
    if case["graph"] == "rmat_device":
        g = _Handle.from_rmat(int(case["scale"]), seed=seed)
        g.set_count_mode(int(case["mode"]))
        return {"case": case, "handle": g}
    n, u, v = _edges(case, seed)
    if op == "load":
        return {"case": case, "text": _text(n, u, v)}
    if op == "new":
        return {"case": case, "edges": (n, u, v), "buffers": _Buffers(n)}
    g = _Handle.from_edges(n, u, v)
    if op == "count":
        g.set_count_mode(int(case["mode"]))
    state = {"case": case, "handle": g, "buffers": _Buffers(n)}
    if op == "stages":
        state["moved"] = [np.zeros(n, np.int64), np.zeros(n, np.int64), np.zeros(n, np.int64), np.zeros(n + 1, np.int64),
                          np.zeros(n, np.int64), np.zeros(n, np.int64), np.zeros(n, np.float64)]
    if op == "nucleus":
        state["tree"] = [np.zeros(u.size, np.int64) for _ in range(5)] + [np.zeros(4 * u.size, np.int64)]
    return state


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "new":
        with _Handle.from_edges(*state["edges"]) as g:
            g.decompose(case["eps"])
            return state["buffers"].clusters(g)
    if op == "resident":
        g = state["handle"]
        g.decompose(case["eps"])
        return state["buffers"].clusters(g)
    if op == "stages":
        g = state["handle"]
        out = {"triangles": g.count()}
        out["perEdge"], out["perVertex"], out["support"], _ = g.weights()
        out["left"] = g.clean(case["eps"])
        out["status"] = g.status()
        out["perEdge_left"], out["perVertex_left"], out["support_left"], _ = g.weights()
        g.extract()
        out.update(state["buffers"].clusters(g))
        out["moved"] = g.expand(int(case["threshold"]))
        c, cof = g.expanded()
        names = ("x_nv", "x_ne", "x_cut", "x_off", "x_vert", "moved_vertex", "moved_score")
        out.update(zip(names, map(_pad, state["moved"], (c.nv, c.ne, c.cut, c.off, c.vert) + g.scores())))
        out["x_cluster_of"] = cof
        return out
    if op == "count":
        g = state["handle"]
        g.count()
        whole = case["graph"] != "rmat_device"
        pe, pv, sup, total = g.weights(per_edge=whole, support=whole)
        out = {"triangles": total, "perVertex": pv}
        if whole:
            out.update(perEdge=pe, support=sup)
        return out
    if op == "batch":
        with _Handle.batch(state["graphs"]) as g:
            g.decompose(case["eps"])
            out = state["buffers"].clusters(g)
            out["counts"] = g.batch_cluster_counts()
            return out
    if op == "load":
        with Graph.from_escape_text(state["text"]) as g:
            off, nb = g.csr()
            return {"offsets": off, "nbors": nb}
    if op == "nucleus":
        g = state["handle"]
        out = {"nuclei": g.nucleus()}
        out.update(zip(("c", "nv", "ne", "parent", "off", "vert"), map(_pad, state["tree"], g.nuclei())))
        return out
    if op == "serve":
        srv = state["server"]
        reqs = [srv.submit(i, case["eps"]) for i in state["requests"]]
        done = [srv.wait(r) for r in reqs]
        out = {k: np.array([d[k] for d in done], np.int64) for k in ("status", "n_clusters", "triangles",
                                                                     "triangles_left")}
        out["cluster_of"] = np.concatenate([d["cluster_of"] for d in done])
        return out
    raise ValueError(op)


def work(case):
    """Bytes: the edge list (or the resident CSR) read once and the results
    written once; operations: a comparison per row entry of each edge's
    intersection, from the shapes' mean row lengths."""
    op = case["op"]
    if op == "batch":
        m = float(sum(_sizes(int(case["graphs"]), 1e3, 2e5)))
        n, rows = m / 7.0, 14.0
    elif op == "serve":
        m = int(case["requests"]) / int(case["graphs"]) * sum(_sizes(int(case["graphs"]), 1e3, float(case["max_edges"])))
        n, rows = m / 9.0, 20.0
    elif case["graph"] == "rmat_device":
        n = float(1 << int(case["scale"]))
        m, rows = 14.0 * n, 200.0
    else:
        m = float(case["edges"])
        n = m / {"gnp": 8.35, "chung_lu": 2.76, "rmat": 10.0, "sbm": 7.0}[case["graph"]]
        rows = {"gnp": 17.0, "chung_lu": 15.0, "rmat": 60.0, "sbm": 14.0}[case["graph"]]
    csr = 8.0 * n + 8.0 * m
    clusters = 8.0 * n * 3 + 8.0 * n
    flops = 2.0 * rows * m
    if op == "new" or op == "batch":
        nbytes = 16.0 * m + clusters
    elif op == "resident" or op == "nucleus":
        nbytes = csr + clusters
    elif op == "stages":
        nbytes = csr + 2 * (24.0 * m + 8.0 * n) + 2.0 * m + 2 * clusters
    elif op == "count":
        nbytes = csr + 8.0 * n + (0.0 if case["graph"] == "rmat_device" else 24.0 * m)
    elif op == "load":
        nbytes = 13.5 * m + 8.0 * n + 16.0 * m
        flops = 0.0
    else:
        nbytes = csr + 8.0 * n
    return {"bytes": nbytes, "flops": flops}


def _csr(n, u, v):
    src = np.concatenate([u, v])
    dst = np.concatenate([v, u])
    order = np.lexsort((dst, src))
    src, dst = src[order], dst[order]
    off = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(src, minlength=n), out=off[1:])
    return off, dst, src


def _weights(n, u, v):
    """Weighted triangle counting in numpy: every wedge of the degree-ordered
    orientation is looked up among the edges."""
    off, nb, src = _csr(n, u, v)
    deg = np.diff(off)
    key = src * n + nb  # ascending
    rank = np.empty(n, np.int64)
    rank[np.lexsort((np.arange(n), deg))] = np.arange(n)
    keep = rank[src] < rank[nb]
    osrc, odst, oslot = src[keep], nb[keep], np.nonzero(keep)[0]
    ooff = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(osrc, minlength=n), out=ooff[1:])
    pe = np.zeros(key.size)
    pv = np.zeros(n)
    sup = np.zeros(key.size, np.int64)
    total = 0
    later = ooff[osrc + 1] - np.arange(osrc.size) - 1  # wedges led by each oriented slot
    ends = np.cumsum(later)
    lo = 0
    while lo < osrc.size:
        base = ends[lo - 1] if lo else 0
        hi = max(lo + 1, int(np.searchsorted(ends, base + (1 << 22), side="right")))
        first = np.repeat(np.arange(lo, hi), later[lo:hi])
        second = first + 1 + np.arange(first.size) - np.repeat(ends[lo:hi] - later[lo:hi] - base, later[lo:hi])
        b, c = odst[first], odst[second]
        pos = np.searchsorted(key, b * n + c)
        hit = (pos < key.size) & (key[np.minimum(pos, key.size - 1)] == b * n + c)
        first, second, pos = first[hit], second[hit], pos[hit]
        a, b, c = osrc[first], b[hit], c[hit]
        w = 1.0 / (deg[a] * deg[b] * deg[c]).astype(np.float64)
        total += int(a.size)
        for x in (a, b, c):
            pv += np.bincount(x, weights=w, minlength=n)
        for s, (x, y) in ((oslot[first], (a, b)), (oslot[second], (a, c)), (pos, (b, c))):
            for t in (s, np.searchsorted(key, y * n + x)):
                pe += np.bincount(t, weights=w, minlength=key.size)
                sup += np.bincount(t, minlength=key.size)
        lo = hi
    return total, pe, pv, sup


def exact(case, seed):
    """What run returns, in 64-bit numpy: the CSR of a text load and the
    weights of a count.  The clean's survivors and the clusters depend on the
    order of the replayed operations and have no such value."""
    op = case["op"]
    if op == "load":
        n, u, v = _edges(case, seed)
        off, nb, _ = _csr(n, u, v)
        return {"offsets": off, "nbors": nb}
    if op == "count" and case["graph"] != "rmat_device" and int(case["edges"]) <= 520000:
        total, pe, pv, sup = _weights(*_edges(case, seed))
        return {"triangles": total, "perVertex": pv, "perEdge": pe, "support": sup.astype(np.uint32)}
    return None
