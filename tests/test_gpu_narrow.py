"""Long narrow graphs, of more and smaller rounds than road networks: round starts that run into the log's free end
(team kernel), sources that leave both kernels early because more rounds would come than are kept, and segments whose
sources leave because other kernels are faster on them.  Against the oracle."""
import numpy as np
import pytest

import oracle
from test_gpu_parity import rel_err
from test_gpu_team import FORMS
from test_gpu_ties import _grid

pytestmark = pytest.mark.gpu


def _strip(fg, rows, cols):
    s, d, w = _grid(rows, cols, lambda rng, m: rng.integers(1, 101, m))
    g = fg.Graph.from_edges(s.astype(np.int32), d.astype(np.int32), w.astype(np.float64))
    return g, oracle.CSR(*g.csr())


@pytest.mark.parametrize("delta", [0, 1 << 20])  # buckets so wide that the log overflows and is begun again
@pytest.mark.parametrize("rows,cols", [(1, 15), (1, 64), (1, 130), (1, 400), (2, 190), (3, 333), (4, 300), (5, 401)])
def test_rounds_in_the_log(fg, rows, cols, delta):
    g, og = _strip(fg, rows, cols)
    ref = oracle.exact_bc(og)
    old = fg.get_option("delta")
    try:
        fg.set_option("delta", delta)
        for prec, tol in FORMS:
            st = fg.Stats()
            assert rel_err(fg.exact_bc(g, prec, fg.BATCHED, stats=st), ref) <= tol
            assert st.retries == 0
            src = g.n - 1
            assert rel_err(fg.single_source(g, src, prec), oracle.exact_bc_sources(og, np.array([src], np.int32))) <= tol
    finally:
        fg.set_option("delta", old)


@pytest.mark.parametrize("rows,cols,count", [(1, 1300, 1300), (1, 1300, 40), (1, 4500, 2000), (10, 700, 7000), (5, 1000, 5000),
                                             (1, 9000, 700), (12, 800, 5200)])
def test_narrow_sources_leave(fg, rows, cols, count):
    """Few and many sources; the last two cases are the log kernel's."""
    g, og = _strip(fg, rows, cols)
    src = np.linspace(0, g.n - 1, count).astype(np.int32)
    ref = oracle.pivot_batch(og, src, np.ones(count), threads=8)
    for prec, tol in FORMS:
        st = fg.Stats()
        assert rel_err(fg.dependency_batch(g, src, None, prec, fg.BATCHED, stats=st), ref) <= tol
        assert st.retries >= 0.6 * count


@pytest.mark.parametrize("rows,cols,count", [(60, 80, 4800), (40, 100, 4000), (8, 500, 4000), (105, 100, 5000)])
def test_ordinary_and_small_ones_stay(fg, rows, cols, count):
    g, og = _strip(fg, rows, cols)
    src = np.linspace(0, g.n - 1, count).astype(np.int32)
    ref = oracle.pivot_batch(og, src, np.ones(count), threads=8)
    for prec, tol in FORMS:
        st = fg.Stats()
        assert rel_err(fg.dependency_batch(g, src, None, prec, fg.BATCHED, stats=st), ref) <= tol
        assert st.retries == 0
