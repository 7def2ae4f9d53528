"""The log kernel (larger segments, global-memory state) at the edges of what it takes: each of its forms
by the number of sources, rows of more than four and more than eight edges, renewed stamps, an
overflowing log, graphs with and without the locality order, and the ways a source leaves it (path
counts, rounds, distances).  Weighted pivots against the oracle."""
import numpy as np
import pytest

import graphs
import oracle
from test_gpu_parity import rel_err
from test_gpu_team import FORMS, _both, _comb, _graph

pytestmark = pytest.mark.gpu


def _check(fg, g, og, count, retries=None, seed=1):
    rng = np.random.default_rng(seed)
    src = rng.choice(g.n, min(count, g.n), replace=False).astype(np.int32)
    cards = rng.integers(1, 50, src.size).astype(np.float64)
    ref = oracle.pivot_batch(og, src, cards, threads=8)
    for prec, tol in FORMS:
        st = fg.Stats()
        got = fg.dependency_batch(g, src, cards, prec, fg.BATCHED, stats=st)
        assert rel_err(got, ref) <= tol
        if retries is not None:
            assert (st.retries > 0) == retries
    return st


@pytest.mark.parametrize("count,group", [(1, 1), (3, 1), (150, 1), (300, 1), (1500, 4)])
def test_forms_by_count(fg, count, group):
    el = graphs.road_grid(131, 127, seed=6)  # (few sources of up to 16,384 vertices run in shared memory)
    st = _check(fg, fg.Graph.from_edgelist(el), oracle.CSR.from_edgelist(el), count, retries=False)
    assert st.group == group


@pytest.mark.parametrize("n,k,count", [(16500, 3, 60), (17001, 5, 40), (16600, 7, 20)])
def test_long_rows(fg, n, k, count):
    el = graphs.rgg_knn(n, k=k, seed=n)
    assert 4 < np.bincount(el.src, minlength=n).max() <= 16
    _check(fg, fg.Graph.from_edgelist(el), oracle.CSR.from_edgelist(el), count)


@pytest.mark.parametrize("rows,cols", [(255, 256), (257, 256)])  # below and above the locality order's size
def test_locality_order(fg, rows, cols):
    el = graphs.road_grid(rows, cols, seed=rows)
    _check(fg, fg.Graph.from_edgelist(el), oracle.CSR.from_edgelist(el), 12, retries=False)


def test_unreached_and_wide_buckets(fg):
    """A grid with a second component, buckets of one distance and so wide that the log overflows."""
    el = graphs.road_grid(130, 130, seed=8)
    s = np.concatenate([el.src, [16900, 16901]])
    d = np.concatenate([el.dst, [16901, 16900]])
    g, og = _graph(fg, s, d, np.concatenate([el.w, [9, 9]]))
    old = fg.get_option("delta")
    try:
        for delta in (0, 1, 1 << 20):
            fg.set_option("delta", delta)
            _check(fg, g, og, 20)
        src = np.array([16900], np.int32)
        assert np.all(fg.dependency_batch(g, src, None, fg.FP64, fg.BATCHED) == 0)
    finally:
        fg.set_option("delta", old)


def test_renewed_stamps(fg):
    s, d, w = _comb(3000, 17000, 200, 2)  # 3,000 rounds of ten-bit stamps
    g, og = _graph(fg, s, d, w)
    _check(fg, g, og, 4, retries=False)


def test_sources_that_leave(fg):
    """More rounds than are kept; distances beyond a word's 22 bits; path counts beyond 2^24."""
    s, d, w = _comb(9000, 17000, 100, 3)
    g, og = _graph(fg, s, d, w)
    _check(fg, g, og, 3, retries=True)
    s, d, w = _comb(17000, 70000, 255, 4)
    w[:16999] = w[69999:69999 + 16999] = 255
    g, og = _graph(fg, s, d, w)
    src = np.array([0, 16999], np.int32)
    ref = oracle.pivot_batch(og, src, np.ones(2), threads=8)
    st = fg.Stats()
    assert rel_err(fg.dependency_batch(g, src, None, fg.FP64, fg.BATCHED, stats=st), ref) <= 1e-9 and st.retries > 0
    ids = np.arange(16900).reshape(130, 130)
    a = np.concatenate([ids[:, :-1].ravel(), ids[:-1].ravel()])
    b = np.concatenate([ids[:, 1:].ravel(), ids[1:].ravel()])
    g, og = _graph(fg, *_both(a, b, np.full(a.size, 9), np.full(a.size, 9)))
    _check(fg, g, og, 5, retries=True)


@pytest.mark.parametrize("count", [1, 3, 60])
def test_cluster_of_blocks(fg, count):
    """Fewer sources than SMs of a graph of more than 524,288 vertices: several blocks to a source; the
    single source in the input order, the batch in the locality order."""
    el = graphs.road_grid(730, 740, seed=5)
    g, og = fg.Graph.from_edgelist(el), oracle.CSR.from_edgelist(el)
    _check(fg, g, og, count, retries=False)
    if count == 1:
        ref = oracle.exact_bc_sources(og, np.array([777], np.int32))
        for prec, tol in FORMS:
            assert rel_err(fg.single_source(g, 777, prec), ref) <= tol
        old = fg.get_option("iter_mult")
        fg.set_option("iter_mult", 0)
        try:
            with pytest.raises(fg.FbcError) as e:
                fg.single_source(g, 777)
            assert e.value.code == fg.FBC_ERR_ITER_LIMIT
        finally:
            fg.set_option("iter_mult", old)
        assert rel_err(fg.single_source(g, 777), ref) <= FORMS[0][1]


@pytest.mark.parametrize("sources", [500, 511, 512, 1500])
def test_units_given_back_unstarted(fg, sources):
    """A grid of equal weights: nearly every source has 2^24 and more shortest paths somewhere, so from 512
    sources on most are handed back without being begun."""
    ids = np.arange(95 * 95).reshape(95, 95)
    a = np.concatenate([ids[:, :-1].ravel(), ids[:-1].ravel()])
    b = np.concatenate([ids[:, 1:].ravel(), ids[1:].ravel()])
    g = fg.Graph.from_edges(np.concatenate([a, b]).astype(np.int32), np.concatenate([b, a]).astype(np.int32),
                            np.full(2 * a.size, 40.0))
    og = oracle.CSR(*g.csr())
    src = np.linspace(0, ids.size - 1, sources).astype(np.int32)
    ref = oracle.pivot_batch(og, src, np.ones(sources))
    for prec, tol in FORMS:
        st = fg.Stats()
        assert rel_err(fg.dependency_batch(g, src, None, prec, fg.BATCHED, stats=st), ref) <= tol
        assert st.retries >= sources


def test_small_weights_on_many_vertices(fg):
    """Weights below 32 on more than 74 * maxw^2 vertices start with the kernels of wider counts."""
    el = graphs.rgg_knn(24000, seed=7, gid=3)
    assert el.w.max() < 18
    g, og = fg.Graph.from_edgelist(el), oracle.CSR.from_edgelist(el)
    src = np.linspace(0, el.n - 1, 12).astype(np.int32)
    ref = oracle.pivot_batch(og, src, np.ones(12))
    for prec, tol in FORMS:
        st = fg.Stats()
        assert rel_err(fg.dependency_batch(g, src, None, prec, fg.BATCHED, stats=st), ref) <= tol
        assert st.retries == 0
