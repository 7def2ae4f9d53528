"""The team kernel (shared-memory state, log of pops) at the edges of what it takes: sizes around its
16-vertex padding and its one-warp / several-warp teams, rows of more than four and more than eight
edges, distances that leave few stamp bits, buckets so wide that the log overflows, and the two ways a
source leaves it (path counts from 2^24 on, more rounds than it keeps).  All against the oracle's exact
BC; border vectors bit-exact against the plain schedule."""
import numpy as np
import pytest

import graphs
import oracle
from test_gpu_parity import TOL_FP32C, TOL_FP64, rel_err

pytestmark = pytest.mark.gpu
FORMS = [(0, TOL_FP64), (1, TOL_FP32C)]


def _graph(fg, src, dst, w):
    g = fg.Graph.from_edges(np.asarray(src, np.int32), np.asarray(dst, np.int32), np.asarray(w, np.float64))
    return g, oracle.CSR(*g.csr())


def _both(a, b, w1, w2):
    return np.concatenate([a, b]), np.concatenate([b, a]), np.concatenate([w1, w2])


def _comb(spine, n, wmax, seed):
    """A path with leaves on it: as many rounds as the path is long."""
    rng = np.random.default_rng(seed)
    a = np.arange(spine - 1)
    leaf = np.arange(spine, n)
    a, b = np.concatenate([a, rng.integers(0, spine, leaf.size)]), np.concatenate([a + 1, leaf])
    return _both(a, b, rng.integers(wmax // 2, wmax + 1, a.size), rng.integers(wmax // 2, wmax + 1, a.size))


def _check(fg, g, og, retries=None):
    ref = oracle.exact_bc(og)
    for prec, tol in FORMS:
        st = fg.Stats()
        assert rel_err(fg.exact_bc(g, prec, fg.BATCHED, stats=st), ref) <= tol
        if retries is not None:
            assert (st.retries > 0) == retries


@pytest.mark.parametrize("rows,cols", [(1, 2), (3, 5), (4, 4), (1, 17), (31, 33), (32, 32), (37, 43), (60, 69)])
def test_sizes(fg, rows, cols):
    el = graphs.road_grid(rows, cols, seed=rows)
    _check(fg, fg.Graph.from_edgelist(el), oracle.CSR.from_edgelist(el))


@pytest.mark.parametrize("n,k", [(300, 3), (900, 5), (700, 7), (2600, 4)])
def test_long_rows(fg, n, k):
    el = graphs.rgg_knn(n, k=k, seed=n)
    deg = np.bincount(el.src, minlength=n)
    assert 4 < deg.max() <= 16  # linked quads; 16-bit masks from nine edges on
    _check(fg, fg.Graph.from_edgelist(el), oracle.CSR.from_edgelist(el))


def test_few_stamps(fg):
    """Eight stamp bits and about 300 rounds: the stamps are renewed on the way."""
    s, d, w = _comb(300, 1200, 13900, 5)
    g, og = _graph(fg, s, d, w)
    assert (1200 * 13900 + 1).bit_length() == 24
    _check(fg, g, og, retries=False)


def test_wide_buckets_overflow_the_log(fg):
    el = graphs.road_grid(40, 40, seed=3)
    g, og = fg.Graph.from_edgelist(el), oracle.CSR.from_edgelist(el)
    old = fg.get_option("delta")
    try:
        for delta in (1, 1 << 20):
            fg.set_option("delta", delta)
            _check(fg, g, og, retries=delta == 1)  # buckets of one distance: more rounds than are kept
    finally:
        fg.set_option("delta", old)


def test_many_rounds_leave_the_kernel(fg):
    s, d, w = _comb(700, 720, 60, 9)
    g, og = _graph(fg, s, d, w)
    _check(fg, g, og, retries=True)


def test_large_counts_leave_the_kernel(fg):
    """A grid of equal weights: most sources have more than 2^24 shortest paths somewhere."""
    ids = np.arange(900).reshape(30, 30)
    a = np.concatenate([ids[:, :-1].ravel(), ids[:-1].ravel()])
    b = np.concatenate([ids[:, 1:].ravel(), ids[1:].ravel()])
    s, d, w = _both(a, b, np.full(a.size, 9), np.full(a.size, 9))
    g, og = _graph(fg, s, d, w)
    _check(fg, g, og, retries=True)
    cs = fg.ClusterSet.from_lists([ids[:15].ravel(), ids[15:].ravel()]).with_borders(g)
    ref = fg.cluster_eval_batch(g, cs, fg.FP64, fg.PLAIN)
    plan = fg.ClusterPlan(g, cs, fg.FP64)
    for ev in (plan.run(), plan.run(), fg.cluster_eval_batch(g, cs, fg.FP64, fg.BATCHED)):
        assert rel_err(ev.intra_bc, ref.intra_bc) <= TOL_FP64
        assert np.array_equal(ev.border_dist, ref.border_dist) and np.array_equal(ev.border_sigma, ref.border_sigma)


@pytest.mark.parametrize("prec,tol", FORMS)
def test_community_sizes_in_one_sweep(fg, prec, tol):
    """Communities from one vertex to several thousand in one call and in one plan (teams of every
    width, rows in shared and in global memory, communities for the frontier kernel)."""
    el = graphs.road_grid(170, 200, seed=12)
    g = fg.Graph.from_edgelist(el)
    cuts = np.cumsum([1, 15, 16, 17, 500, 1100, 2100, 4200, 8300])
    cs = fg.ClusterSet.from_lists(np.split(np.arange(el.n, dtype=np.int32), cuts)).with_borders(g)
    ref = fg.cluster_eval_batch(g, cs, fg.FP64, fg.PLAIN)
    for ev in (fg.cluster_eval_batch(g, cs, prec, fg.BATCHED), fg.ClusterPlan(g, cs, prec).run()):
        assert rel_err(ev.intra_bc, ref.intra_bc) <= tol
        assert np.array_equal(ev.border_dist, ref.border_dist) and np.array_equal(ev.border_sigma, ref.border_sigma)


@pytest.mark.parametrize("rows,cols,counts", [(92, 95, (1, 40)), (128, 128, (1, 300, 620)), (129, 128, (1,))])
def test_few_sources_of_larger_graphs(fg, rows, cols, counts):
    """Up to four sources per SM run in shared memory with room for one source (8,700 to 16,384 vertices);
    more, or a larger graph, in the log kernel.  Single sources, too."""
    el = graphs.road_grid(rows, cols, seed=rows)
    g, og = fg.Graph.from_edgelist(el), oracle.CSR.from_edgelist(el)
    for count in counts:
        src = np.arange(0, g.n, g.n // count, dtype=np.int32)[:count]
        ref = oracle.exact_bc_sources(og, src, threads=8)
        for prec, tol in FORMS:
            st = fg.Stats()
            assert rel_err(fg.dependency_batch(g, src, None, prec, fg.BATCHED, stats=st), ref) <= tol
            assert (st.group == 0) == (g.n <= 16384 and count <= 608)
            if count == 1:
                assert rel_err(fg.single_source(g, 0, prec), ref) <= tol


@pytest.mark.parametrize("prec,tol", FORMS)
def test_single_source_forms(fg, prec, tol):
    """A single source by the team kernel, the log kernel (input order) and, for rows too long for both, the
    plain kernel; the source's own entry is 0; a bad source is refused."""
    for el in (graphs.road_grid(20, 31, seed=2), graphs.road_grid(260, 270, seed=2), graphs.rgg_knn(3000, k=12, seed=21)):
        g, og = fg.Graph.from_edgelist(el), oracle.CSR.from_edgelist(el)
        for s in (0, el.n - 1):
            got = fg.single_source(g, s, prec)
            assert got[s] == 0 and rel_err(got, oracle.exact_bc_sources(og, np.array([s], np.int32))) <= tol
        for s in (-1, el.n):
            with pytest.raises(fg.FbcError) as e:
                fg.single_source(g, s, prec)
            assert e.value.code == fg.FBC_ERR_INVALID_ARG
