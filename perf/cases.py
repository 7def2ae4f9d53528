"""The calls whose speed matters to a user of the engine, through the Python binding.

Each case is one call (or one pass of a prepared object) on a seeded synthetic graph of the kinds
the engine is used on: road-like grids (4-neighbour, 5% of the pairs missing, a few highways,
independent integer weights per direction) and random geometric 3-nearest-neighbour graphs.

kinds:
  source     single_source: one source's dependency vector (the reference's ISSBrandesBC)
  exact      exact_bc of one graph
  batch      multi_exact_bc of several random geometric graphs
  sweep      cluster_eval_batch: every community of a partition, borders included
  plan       ClusterPlan.run: the same sweep prepared once
  pivots     dependency_batch: weighted pivots over a whole graph
  clustered  clustered_bc: sweep, pivots and correction, the whole approximate BC
  select     cluster_classes and kmeans: the pivot selection of every community
  load       Graph.from_text and Graph.csr: edge-list text to CSR arrays
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "fast-bc_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import fastbc_gpu as fg  # noqa: E402
import graphs  # noqa: E402

PREC = {"fp64": fg.FP64, "fp32c": fg.FP32C}
SCHED = {"plain": fg.PLAIN, "batched": fg.BATCHED}


def listed():
    return [
        # one source of a small network: latency and launches
        {"name": "source_small", "kind": "source", "rows": 33, "cols": 31, "prec": "fp64"},
        # one source of a city-to-region sized network, as a caller of the single-source interface asks for it
        {"name": "source_large", "kind": "source", "rows": 1000, "cols": 1049, "prec": "fp64"},
        # the smallest exact configuration (32 x 32), batched FP64
        {"name": "exact_32x32", "kind": "exact", "rows": 32, "cols": 32, "prec": "fp64", "sched": "batched"},
        # exact BC with the binding's default arguments
        {"name": "exact_default", "kind": "exact", "rows": 90, "cols": 71, "prec": "fp64", "sched": "plain"},
        # exact BC of a whole mid-sized network, compensated FP32
        {"name": "exact_128x128", "kind": "exact", "rows": 128, "cols": 128, "prec": "fp32c", "sched": "batched"},
        # a batch of random geometric graphs of mixed sizes in one call
        {"name": "batch_rgg", "kind": "batch", "count": 10, "lo": 1024, "hi": 8192, "prec": "fp32c"},
        # the community sweep of the 256 x 256 network (76 communities of some 860 vertices)
        {"name": "sweep_256x256", "kind": "sweep", "rows": 256, "cols": 256, "regions": 76, "prec": "fp32c"},
        # a prepared sweep of larger communities (some 8,000 vertices each), FP64
        {"name": "plan_large", "kind": "plan", "rows": 230, "cols": 219, "regions": 6, "prec": "fp64"},
        # the whole clustered approximation on the 256 x 256 network
        {"name": "clustered_256x256", "kind": "clustered", "rows": 256, "cols": 256, "regions": 76, "share": 0.02, "prec": "fp32c"},
        # the pivot phase of the 2048 x 2048 network (4.2 million vertices)
        {"name": "pivots_2048x2048", "kind": "pivots", "rows": 2048, "cols": 2048, "count": 280, "prec": "fp32c"},
        # the pivot selection of a partitioned network: exact classes, then k-means
        {"name": "select_108x108", "kind": "select", "rows": 108, "cols": 108, "regions": 20},
        # reading an edge list of half a million vertices into CSR arrays
        {"name": "load_text", "kind": "load", "rows": 700, "cols": 733},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def grid(lo, hi):  # a ragged grid of lo .. hi vertices
        n = log(lo, hi)
        rows = max(2, int(math.sqrt(n) * rng.uniform(0.7, 1.4)))
        return {"rows": rows, "cols": max(2, n // rows)}

    def regions(c, lo, hi):  # communities of lo .. hi vertices on average
        return max(2, c["rows"] * c["cols"] // log(lo, hi))

    kind = rng.choice(["source", "source", "exact", "exact", "batch", "sweep", "plan", "pivots", "clustered", "select", "load"])
    prec = rng.choice(["fp64", "fp32c"])
    if kind == "source":
        return {"kind": kind, **grid(1000, 600000), "prec": prec}
    if kind == "exact":
        sched = rng.choice(["plain", "batched", "batched"])
        return {"kind": kind, **grid(900, 6400 if sched == "plain" else 16384), "prec": prec, "sched": sched}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(3, 10), "lo": 1024, "hi": log(1500, 8192), "prec": prec}
    if kind == "sweep":
        c = grid(12000, 65536)
        return {"kind": kind, **c, "regions": regions(c, 300, 1800), "prec": prec}
    if kind == "plan":
        c = grid(16000, 50000)
        return {"kind": kind, **c, "regions": regions(c, 700, 8000), "prec": prec}
    if kind == "pivots":
        return {"kind": kind, **grid(20000, 2000000), "count": log(30, 280), "prec": prec}
    if kind == "clustered":
        c = grid(16000, 65536)
        return {"kind": kind, **c, "regions": regions(c, 400, 1500), "share": round(rng.uniform(0.005, 0.02), 4), "prec": prec}
    if kind == "select":
        c = grid(4000, 11664)
        return {"kind": kind, **c, "regions": regions(c, 250, 580)}
    return {"kind": kind, **grid(30000, 513100)}


# ------------------------------------------------------------------------------ inputs
def _road(case, seed):
    """A road-like grid's edge list: every kept neighbour pair in both directions with weights of
    1..100 each, and highways (0.2% of the vertices, within 32 rows and columns, weights 1..20).
    Where the size of the results follows the edges (their number, the communities' borders), the
    layout belongs to the case and the seed gives the weights."""
    rows, cols = case["rows"], case["cols"]
    rng = np.random.default_rng([rows, cols, 0 if case["kind"] in ("sweep", "plan", "select", "load") else 1 + seed])
    n = rows * cols
    ids = np.arange(n, dtype=np.int32).reshape(rows, cols)
    a = np.concatenate([ids[:, :-1].ravel(), ids[:-1].ravel()])
    b = np.concatenate([ids[:, 1:].ravel(), ids[1:].ravel()])
    keep = rng.random(a.size, dtype=np.float32) >= 0.05
    keep[rows * (cols - 1) - 1] = True  # the last vertex has an edge, so that there are rows * cols vertices
    a, b = a[keep], b[keep]
    h = rng.integers(0, n, int(0.002 * n))
    r = np.clip(h // cols + rng.integers(-32, 33, h.size), 0, rows - 1)
    c = np.clip(h % cols + rng.integers(-32, 33, h.size), 0, cols - 1)
    t = r * cols + c
    h, t = h[h != t].astype(np.int32), t[h != t].astype(np.int32)
    src = np.concatenate([a, b, h, t])
    dst = np.concatenate([b, a, t, h])
    rng = np.random.default_rng([seed, 0])
    w = np.concatenate([rng.integers(1, 101, 2 * a.size, dtype=np.int32), rng.integers(1, 21, 2 * h.size, dtype=np.int32)])
    return n, src, dst, w


def _rgg(case, seed):
    rng = np.random.default_rng([case["count"], case["hi"]])
    sizes = np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), case["count"])).round().astype(int)
    sizes[0] = case["hi"]
    return [graphs.rgg_knn(int(n), seed=seed % (1 << 20), gid=i) for i, n in enumerate(sizes)]


def _regions(case):
    """A partition into irregular communities: every vertex goes to the nearest of random centres."""
    rows, cols, k = case["rows"], case["cols"], case["regions"]
    rng = np.random.default_rng([rows, cols, k])
    centre = rng.choice(rows * cols, k, replace=False)
    r, c = np.divmod(np.arange(rows * cols), cols)
    best, reg = np.full(rows * cols, np.inf), np.zeros(rows * cols, np.int64)
    for i, v in enumerate(centre):
        d = (r - v // cols) ** 2 + (c - v % cols) ** 2
        near = d < best
        best[near] = d[near]
        reg[near] = i
    order = np.argsort(reg, kind="stable").astype(np.int32)
    return np.split(order, np.cumsum(np.bincount(reg, minlength=k))[:-1])


def _pivots(case, seed, groups):
    """Pivots of each community (a share of its vertices) with class sizes that add up to its size."""
    rng = np.random.default_rng([seed, 2])
    piv, cards = [], []
    for vs in groups:
        k = max(1, int(round(case["share"] * vs.size)))
        piv.append(rng.choice(vs, k, replace=False).astype(np.int32))
        cards.append((1 + rng.multinomial(vs.size - k, np.full(k, 1.0 / k))).astype(np.float64))
    return piv, cards


def _sources(case, seed, n, count):
    rng = np.random.default_rng([seed, 3])
    return rng.choice(n, count, replace=False).astype(np.int32), rng.integers(1, 200, count).astype(np.float64)


def _point_sets(cs, classes, ev):
    """The k-means inputs of every community: its class pivots' border vectors, shifted by their least length."""
    sets = []
    for c, (piv, size) in enumerate(classes):
        vs = cs.vertices[cs.off[c]:cs.off[c + 1]]
        nb, e = int(cs.boff[c + 1] - cs.boff[c]), int(ev.entry_off[c])
        at = np.searchsorted(vs, piv)
        d = ev.border_dist[e:e + vs.size * nb].reshape(vs.size, nb)[at]
        s = ev.border_sigma[e:e + vs.size * nb].reshape(vs.size, nb)[at]
        sets.append((d - d.min(axis=1, keepdims=True), s.astype(np.int32), size))
    return sets


def prepare(case, seed):
    fg.init(0)
    kind = case["kind"]
    state = {"kind": kind, "prec": PREC[case.get("prec", "fp64")], "sched": SCHED[case.get("sched", "batched")]}
    if kind == "batch":
        state["graphs"] = [fg.Graph.from_edgelist(el) for el in _rgg(case, seed)]
        return state
    n, src, dst, w = _road(case, seed)
    if kind == "load":
        state["text"] = graphs.EdgeList(n, src, dst, w).text()
        return state
    g = state["g"] = fg.Graph.from_edges(src, dst, w)
    if kind == "source":
        state["source"] = int(_sources(case, seed, n, 1)[0][0])
    elif kind == "pivots":
        state["pivots"], state["cards"] = _sources(case, seed, n, case["count"])
    elif kind != "exact":
        groups = _regions(case)
        cs = state["cs"] = fg.ClusterSet.from_lists(groups).with_borders(g)
        if kind == "plan":
            state["plan"] = fg.ClusterPlan(g, cs, state["prec"])
        elif kind == "clustered":
            state["pivots"], state["cards"] = _pivots(case, seed, groups)
        elif kind == "select":
            state["ev"] = fg.cluster_eval_batch(g, cs, fg.FP64, fg.BATCHED)
            state["sets"] = _point_sets(cs, fg.cluster_classes(g, cs, state["ev"].intra_bc, state["ev"]), state["ev"])
    return state


# ------------------------------------------------------------------------------ the calls
def _flat(pairs, n):
    """The lists of every community back to back, in arrays of n entries (their number follows the weights)."""
    out = np.full((2, n), -1, np.int32)
    for i in (0, 1):
        x = np.concatenate([p[i] for p in pairs])
        out[i, :x.size] = x
    return list(out)


def run(state):
    kind, prec, sched, g = state["kind"], state["prec"], state["sched"], state.get("g")
    if kind == "source":
        return fg.single_source(g, state["source"], prec)
    if kind == "exact":
        return fg.exact_bc(g, prec, sched)
    if kind == "batch":
        return fg.multi_exact_bc(state["graphs"], prec)
    if kind == "pivots":
        return fg.dependency_batch(g, state["pivots"], state["cards"], prec, sched)
    if kind == "clustered":
        return fg.clustered_bc(g, state["cs"], state["pivots"], state["cards"], prec, sched)
    if kind == "select":
        classes = fg.cluster_classes(g, state["cs"], state["ev"].intra_bc, state["ev"])
        return _flat(classes, g.n) + _flat(fg.kmeans(state["sets"]), g.n)
    if kind == "load":
        return list(fg.Graph.from_text(state["text"]).csr())
    ev = state["plan"].run() if kind == "plan" else fg.cluster_eval_batch(g, state["cs"], prec, sched)
    return [ev.intra_bc, ev.border_dist, ev.border_sigma.view(np.int64)]


# ------------------------------------------------------------------------------ what it cannot do without
def work(case):
    """Bytes: the graph read once, the results written once.  Operations: per source and edge an
    add and a compare, per source and vertex the count, the ratio and the two dependency steps."""
    kind = case["kind"]
    if kind == "batch":
        sizes = [case["hi"]] + [math.sqrt(case["lo"] * case["hi"])] * (case["count"] - 1)
        return {"bytes": sum(8 * 4.4 * n + 12 * n for n in sizes), "flops": sum(n * (2 * 4.4 * n + 4 * n) for n in sizes)}
    n = case["rows"] * case["cols"]
    m = 3.8 * n
    graph = 8 * m + 4 * n
    if kind == "load":
        return {"bytes": 19 * m + 12 * m + 8 * n, "flops": 19 * m}
    if kind == "source":
        return {"bytes": graph + 8 * n, "flops": 2 * m + 4 * n}
    if kind == "exact":
        return {"bytes": graph + 8 * n, "flops": n * (2 * m + 4 * n)}
    if kind == "pivots":
        return {"bytes": graph + 8 * n, "flops": case["count"] * (2 * m + 4 * n)}
    size = n / case["regions"]
    borders = 4 * 0.9 * math.sqrt(size)
    sweep = n * (2 * 3.7 * size + 4 * size)
    if kind == "select":  # one k-means start and one step over half the points as centroids
        return {"bytes": 16 * n * borders + 16 * n, "flops": 2 * 6 * n * (size / 2) * borders}
    if kind == "clustered":
        return {"bytes": graph + 8 * n, "flops": sweep + case["share"] * n * (2 * m + 4 * n)}
    return {"bytes": graph + 8 * n + 16 * n * borders, "flops": sweep}


# ------------------------------------------------------------------------------ values in 64 bits
def _merged(n, src, dst, w):
    """Edges sorted by (source, destination), the weights of a repeated pair added up."""
    key, at = np.unique(src.astype(np.int64) * n + dst, return_inverse=True)
    return key // n, key % n, np.bincount(at, weights=w).astype(np.int64)


def _columns(n, at, other, w, dev):
    """The edges sorted by `at` as columns: (vertices of more than d edges, their d-th edge's other end, its weight)."""
    order = np.argsort(at, kind="stable")
    at, other, w = at[order], other[order], w[order]
    start = np.searchsorted(at, np.arange(n))
    rank = np.arange(at.size) - start[at]
    cols = []
    for d in range(int(rank.max()) + 1 if at.size else 0):
        on = rank == d
        cols.append(tuple(torch.from_numpy(np.ascontiguousarray(x[on])).to(dev) for x in (at, other, w)))
    return cols


def _settle(step, x):
    """step() applied until nothing changes."""
    while True:
        for _ in range(16):
            y = step(x)
            x, last = y, x
        if torch.equal(x, last):
            return x


def _dependencies(n, src, dst, w, sources):
    """Distances, path counts and dependencies of each source (columns), by plain fixed-point sweeps in 64 bits."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    into, out = _columns(n, dst, src, w, dev), _columns(n, src, dst, w, dev)
    far = 1 << 40
    per = max(1, min(len(sources), 100_000_000 // max(n, 1)))
    for lo in range(0, len(sources), per):
        s = torch.as_tensor(np.asarray(sources[lo:lo + per], np.int64), device=dev)
        k = torch.arange(s.numel(), device=dev)
        start = torch.full((n, s.numel()), far, dtype=torch.int64, device=dev)
        start[s, k] = 0

        def nearer(d):
            new = d.clone()
            for v, u, x in into:
                new[v] = torch.minimum(new[v], d[u] + x[:, None])
            return new

        dist = _settle(nearer, start)
        reached = dist < far
        in_tight = [(v, u, (dist[u] + x[:, None] == dist[v]) & reached[v]) for v, u, x in into]
        one = torch.zeros((n, s.numel()), dtype=torch.float64, device=dev)
        one[s, k] = 1.0

        def count(c):
            new = one.clone()
            for v, u, t in in_tight:
                new[v] += c[u] * t
            return new

        sigma = _settle(count, one)
        del in_tight
        share = [(v, x, torch.where((dist[v] + y[:, None] == dist[x]) & reached[v], sigma[v] / sigma[x], 0.0)) for v, x, y in out]

        def back(d):
            new = torch.zeros_like(d)
            for v, x, r in share:
                new[v] += r * (1.0 + d[x])
            return new

        delta = _settle(back, torch.zeros_like(one))
        delta[s, k] = 0.0
        yield lo, dist, reached, delta


def _bc(n, src, dst, w, sources, cards=None):
    bc = np.zeros(n)
    for lo, _, _, delta in _dependencies(n, src, dst, w, sources):
        c = torch.ones(delta.shape[1], dtype=torch.float64, device=delta.device) if cards is None else \
            torch.as_tensor(cards[lo:lo + delta.shape[1]], device=delta.device)
        bc += (delta * c).sum(dim=1).cpu().numpy()
    return bc


def _sweep(n, src, dst, w, groups):
    """Intra-community BC and every vertex's distances to its community's borders (0 when unreached)."""
    reg = np.zeros(n, np.int64)
    for i, vs in enumerate(groups):
        reg[vs] = i
    inside = reg[src] == reg[dst]
    border = np.zeros(n, bool)
    border[src[~inside]] = border[dst[~inside]] = True
    bc, dists = np.zeros(n), []
    for i, vs in enumerate(groups):
        on = inside & (reg[src] == i)
        local = np.zeros(n, np.int64)
        local[vs] = np.arange(vs.size)
        at = torch.from_numpy(np.flatnonzero(border[vs]))
        for _, dist, reached, delta in _dependencies(vs.size, local[src[on]], local[dst[on]], w[on], np.arange(vs.size)):
            bc[vs] += delta.sum(dim=1).cpu().numpy()
            rows = torch.where(reached, dist, 0)[at.to(dist.device)]
            dists.append(rows.T.double().cpu().numpy().ravel())
    return bc, np.concatenate(dists)


def exact(case, seed):
    kind = case["kind"]
    if kind == "select":
        return None  # whole numbers only
    if kind == "batch":
        return [_bc(el.n, el.src.astype(np.int64), el.dst.astype(np.int64), el.w.astype(np.int64), np.arange(el.n)) for el in _rgg(case, seed)]
    edges = _road(case, seed)
    n = edges[0]
    if kind == "pivots" and n * case["count"] > 30_000_000:
        return None
    src, dst, w = _merged(*edges)
    if kind == "load":
        return [None, None, w.astype(np.float64)]
    if kind == "source":
        return _bc(n, src, dst, w, _sources(case, seed, n, 1)[0])
    if kind == "exact":
        return _bc(n, src, dst, w, np.arange(n))
    if kind == "pivots":
        return _bc(n, src, dst, w, *_sources(case, seed, n, case["count"]))
    groups = _regions(case)
    intra, dist = _sweep(n, src, dst, w, groups)
    if kind != "clustered":
        return [intra, dist, None]
    piv, cards = _pivots(case, seed, groups)
    bc = intra + _bc(n, src, dst, w, np.concatenate(piv), np.concatenate(cards))
    for vs, c in zip(groups, cards):
        bc[vs] -= intra[vs] * c.sum()
    return bc
