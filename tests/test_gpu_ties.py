"""Graphs rich in equally long ways: units whose path counts will outgrow 24 bits start with the kernels of wider
counts, without a run in the team or log kernel that would be given back.  The share of ties (on a graph of up to
1,024 vertices taken over all of them) and the line are restated here."""
import numpy as np
import pytest

import graphs
import oracle
from test_gpu_parity import rel_err
from test_gpu_team import FORMS

pytestmark = pytest.mark.gpu


def _grid(rows, cols, w):
    ids = np.arange(rows * cols).reshape(rows, cols)
    a = np.concatenate([ids[:, :-1].ravel(), ids[:-1].ravel()])
    b = np.concatenate([ids[:, 1:].ravel(), ids[1:].ravel()])
    return np.concatenate([a, b]), np.concatenate([b, a]), w(np.random.default_rng(rows), 2 * a.size)


def _rgg(n, k, w=None):
    el = graphs.rgg_knn(n, k=k, seed=n)
    return el.src, el.dst, el.w if w is None else w(None, el.m)


def _one(rng, m):
    return np.full(m, 40)


def _two(rng, m):
    return rng.choice([40, 80], m)


def _ring(rng, n):
    """A ring with each vertex's next two and 10% of these edges elsewhere: ties as in a grid, but few hops."""
    a = np.repeat(np.arange(n), 2)
    b = (a + np.tile([1, 2], n)) % n
    b = np.where(rng.random(a.size) < 0.1, rng.integers(0, n, a.size), b)
    a, b = np.append(a[a != b], n - 1), np.append(b[a != b], 0)
    key = np.unique(np.concatenate([a * n + b, b * n + a]))
    return key // n, key % n, np.full(key.size, 40)


def _ties(g):
    """(tied, all) of the vertices within two edges of each sampled vertex."""
    rp, col, w = g.csr()
    tied = seen = 0
    for k in range(min(g.n, 1024)):
        u = k * g.n // min(g.n, 1024)
        ways = {}
        for e in range(rp[u], min(rp[u + 1], rp[u] + 16)):
            x = col[e]
            for y, length in [(x, w[e])] + [(col[f], w[e] + w[f]) for f in range(rp[x], min(rp[x + 1], rp[x] + 16))]:
                if y != u:
                    ways.setdefault(int(y), []).append(length)
        seen += len(ways)
        tied += sum(v.count(min(v)) > 1 for v in ways.values())
    return tied, seen


@pytest.mark.parametrize("build_m", [0, 1 << 30])  # the CSR built on the device and by the host
@pytest.mark.parametrize("edges,rich", [
    (lambda: _grid(14, 14, _one), False), (lambda: _grid(18, 18, _one), True), (lambda: _grid(16, 16, _one), False),
    (lambda: _grid(60, 60, _one), True),
    (lambda: _grid(4, 250, _one), True), (lambda: _grid(31, 33, _two), False),
    (lambda: _ring(np.random.default_rng(4), 4000), False), (lambda: _grid(90, 71, _two), True), (lambda: _grid(2, 1, _one), False), (lambda: _rgg(1000, 3), False),
    (lambda: _rgg(1000, 12), False), (lambda: _rgg(1000, 3, _one), False), (lambda: _rgg(3000, 3, _one), True)])
def test_rich_graphs_are_not_begun_twice(fg, edges, rich, build_m):
    s, d, w = edges()
    old = fg.get_option("csr_device_min_m")
    try:
        fg.set_option("csr_device_min_m", build_m)
        g = fg.Graph.from_edges(s.astype(np.int32), d.astype(np.int32), w.astype(np.float64))
    finally:
        fg.set_option("csr_device_min_m", old)
    tied, seen = _ties(g)
    m = g.csr()[1].size
    over = (tied / seen * g.n) ** 2 / m if tied >= 0.02 * seen else 0.0
    assert (over >= 8) == rich or (not rich and over > 15)  # (the ring: not as deep)
    src = np.linspace(0, g.n - 1, min(g.n, 700)).astype(np.int32)
    ref = oracle.pivot_batch(oracle.CSR(*g.csr()), src, np.ones(src.size), threads=8)
    for prec, tol in FORMS:
        st = fg.Stats()
        assert rel_err(fg.dependency_batch(g, src, None, prec, fg.BATCHED, stats=st), ref) <= tol
        assert (st.retries >= src.size) == rich
        if st.retries == src.size:  # (else counts beyond 48 bits too)
            assert st.launches == 1
        one = fg.single_source(g, int(src[-1]), prec, stats=st)
        assert rel_err(one, oracle.exact_bc_sources(oracle.CSR(*g.csr()), src[-1:])) <= tol
        if over >= 64:
            assert st.launches - st.retries == 1  # (the plain kernel, again where 64 bits overflow)
