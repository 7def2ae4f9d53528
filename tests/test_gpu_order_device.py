"""The locality order built on the device: sizes around its leaves and its halvings, several components,
edges without a reverse, rows at the longest it takes, parts ordered by a cluster of blocks, and the graphs
it leaves to the host (a longer row, a part of too many rounds, many components).  A lost or repeated vertex,
row or weight shows in the dependencies against the oracle."""
import numpy as np
import pytest

import graphs
import oracle
from test_gpu_parity import rel_err
from test_gpu_team import FORMS, _both, _comb, _graph

pytestmark = pytest.mark.gpu


@pytest.fixture
def relabel_all(fg):
    old = fg.get_option("order_min_n")
    fg.set_option("order_min_n", 0)
    yield
    fg.set_option("order_min_n", old)


def _check(fg, g, og, npiv, kernels=(4096, 0)):
    rng = np.random.default_rng(npiv)
    piv = rng.choice(og.n, min(npiv, og.n), replace=False).astype(np.int32)
    cards = rng.integers(1, 9, piv.size).astype(np.float64)
    ref = oracle.pivot_batch(og, piv, cards)
    old = fg.get_option("warp_max_n")
    try:
        for k in kernels:  # 0: the frontier kernel, which reads the packed rows and reverse weights as well
            fg.set_option("warp_max_n", k)
            for prec, tol in FORMS:
                assert rel_err(fg.dependency_batch(g, piv, cards, prec, fg.BATCHED), ref) <= tol
    finally:
        fg.set_option("warp_max_n", old)


@pytest.mark.parametrize("rows,cols", [(1, 1), (1, 16), (1, 17), (3, 11), (8, 32), (19, 27), (101, 103)])
def test_sizes(fg, relabel_all, rows, cols):
    el = graphs.road_grid(rows, cols, seed=cols)
    _check(fg, fg.Graph.from_edgelist(el), oracle.CSR.from_edgelist(el), 12)


def test_shuffled_components(fg, relabel_all):
    """Five grids and some single vertices, ids shuffled."""
    els = [graphs.road_grid(r, r + 3, seed=r) for r in (40, 31, 12, 5, 2)]
    off = np.cumsum([0] + [e.n for e in els])
    n = int(off[-1]) + 20
    new = np.random.default_rng(2).permutation(n)
    new[[0, n - 1]] = new[[n - 1, 0]]
    s = new[np.concatenate([e.src + o for e, o in zip(els, off)] + [np.arange(off[-1], n)])]
    d = new[np.concatenate([e.dst + o for e, o in zip(els, off)] + [np.zeros(20, int)])]  # no edge back
    w = np.concatenate([e.w for e in els] + [np.full(20, 7)])
    g, og = _graph(fg, s, d, w)
    _check(fg, g, og, 40)


@pytest.mark.parametrize("deg", [63, 64, 65])
def test_long_rows(fg, relabel_all, deg):
    rng = np.random.default_rng(deg)
    ring = np.arange(700)
    hub = rng.choice(np.arange(2, 699), deg - 2, replace=False)
    a, b = np.concatenate([ring, np.zeros(hub.size, int)]), np.concatenate([(ring + 1) % 700, hub])
    w1, w2 = rng.integers(1, 200, a.size), rng.integers(1, 200, a.size)
    g, og = _graph(fg, *_both(a, b, w1, w2))
    _check(fg, g, og, 12)


def test_wide_weights(fg, relabel_all):
    el = graphs.road_grid(30, 31, seed=8)
    g, og = _graph(fg, el.src, el.dst, np.asarray(el.w) * 90)
    _check(fg, g, og, 12)


@pytest.mark.parametrize("spine,n", [(1200, 3000), (5000, 150000)])
def test_too_many_rounds(fg, relabel_all, spine, n):
    s, d, w = _comb(spine, n, 60, 3)
    g, og = _graph(fg, s, d, w)
    _check(fg, g, og, 3, (4096,))


@pytest.mark.parametrize("single", [0, 20, 30000])
def test_cluster_of_blocks(fg, relabel_all, single):
    """135,000 vertices and more in one part; `single` vertices that only a search of its own finds."""
    el = graphs.road_grid(300, 450, seed=6)
    extra = np.arange(el.n, el.n + single)
    g, og = _graph(fg, np.concatenate([el.src, extra]), np.concatenate([el.dst, np.zeros(single, int)]),
                   np.concatenate([el.w, np.full(single, 9)]))
    _check(fg, g, og, 3, (4096,))
