"""The locality order built on the device is the host's recursion, whatever the timing: a batched source on
the graph gives bit for bit what it gives on a copy whose ids the test has relabelled itself by that
recursion (a vertex's dependency is summed in the order of its row, so another order shows in the last bits),
and so do several handles of one graph."""
import numpy as np
import pytest

import graphs
from test_gpu_team import _comb

pytestmark = pytest.mark.gpu


def _bisection(rp, col, leaf=16):
    """Recursive BFS bisection: a part in BFS order from its first vertex not yet reached, halved; leaves by id."""
    n = rp.size - 1
    rows = [col[rp[v]:rp[v + 1]].tolist() for v in range(n)]
    order, owner, seen, tag = list(range(n)), [0] * n, [0] * n, 0
    todo = [(0, n)]
    while todo:
        lo, hi = todo.pop()
        if hi - lo <= leaf:
            order[lo:hi] = sorted(order[lo:hi])
            continue
        tag += 1
        part = order[lo:hi]
        for v in part:
            owner[v] = tag
        q = []
        for s in part:
            if seen[s] == tag:
                continue
            h = len(q)
            q.append(s)
            seen[s] = tag
            while h < len(q):
                for x in rows[q[h]]:
                    if owner[x] == tag and seen[x] != tag:
                        seen[x] = tag
                        q.append(x)
                h += 1
        order[lo:hi] = q
        mid = lo + (hi - lo) // 2
        todo += [(mid, hi), (lo, mid)]
    new = np.empty(n, np.int64)
    new[order] = np.arange(n)
    return new


def _run(fg, g, source, order_min_n):
    old = fg.get_option("order_min_n")
    fg.set_option("order_min_n", order_min_n)
    try:
        return [fg.dependency_batch(g, np.array([source], np.int32), None, p, fg.BATCHED) for p in (fg.FP64, fg.FP32C)]
    finally:
        fg.set_option("order_min_n", old)


def _shuffled(el, extra, seed):
    """The graph with its ids shuffled (the last one kept) and `extra` single vertices that only lead into it."""
    n = el.n + extra
    new = np.append(np.random.default_rng(seed).permutation(n - 1), n - 1)
    single = np.arange(el.n, n)
    s, d = new[np.concatenate([el.src, single, [n - 1]])], new[np.concatenate([el.dst, np.zeros(extra + 1, int)])]
    return s, d, np.concatenate([el.w, np.full(extra + 1, 7)])


@pytest.mark.parametrize("edges", [lambda: (lambda e: (e.src, e.dst, e.w))(graphs.road_grid(3, 11, seed=1)),
                                   lambda: (lambda e: (e.src, e.dst, e.w))(graphs.road_grid(101, 103, seed=2)),
                                   lambda: (lambda e: (e.src, e.dst, e.w))(graphs.rgg_knn(9000, k=5, seed=3)),
                                   lambda: _shuffled(graphs.road_grid(90, 77, seed=4), 60, 5),
                                   lambda: _shuffled(graphs.road_grid(371, 379, seed=6), 9, 7)])
def test_order_is_the_recursion(fg, edges):
    """Parts on one warp up to parts on a cluster of blocks (above 131,072 vertices), with single vertices too."""
    s, d, w = edges()
    g = fg.Graph.from_edges(np.asarray(s, np.int32), np.asarray(d, np.int32), np.asarray(w, np.float64))
    rp, col, wt = g.csr()
    new = _bisection(rp, col)
    src = np.repeat(np.arange(g.n), np.diff(rp))
    h = fg.Graph.from_edges(new[src].astype(np.int32), new[col].astype(np.int32), wt)
    source = g.n // 3
    for a, b in zip(_run(fg, g, source, 0), _run(fg, h, int(new[source]), 1 << 30)):
        assert np.array_equal(a, b[new])


@pytest.mark.parametrize("edges", [lambda: (lambda e: (e.src, e.dst, e.w))(graphs.road_grid(512, 512, seed=8)),
                                   lambda: _comb(1200, 3000, 60, 3), lambda: _comb(4000, 60000, 60, 4)])
def test_order_is_the_same_again(fg, edges):
    """Large parts, and parts of more rounds than they are given, on four handles of one graph."""
    s, d, w = edges()
    out = []
    for _ in range(4):
        g = fg.Graph.from_edges(np.asarray(s, np.int32), np.asarray(d, np.int32), np.asarray(w, np.float64))
        out.append(_run(fg, g, g.n // 3, 0))
        g.free()
    for o in out[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(out[0], o))
