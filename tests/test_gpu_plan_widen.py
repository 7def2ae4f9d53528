"""A prepared sweep in which some communities' path counts outgrow 24 bits: the first run is redone, and
from then on the plan replays with wider counts for those communities, with the same results."""
import numpy as np
import pytest

from test_gpu_parity import rel_err
from test_gpu_team import FORMS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols,strips", [(120, (6, 1, 8, 4)), (1200, (4, 1)), (3000, (4, 1))])
@pytest.mark.parametrize("prec,tol", FORMS)
def test_plan_is_captured_again(fg, cols, strips, prec, tol):
    """Strips of equal weights: 4 of 1,200 have 2.9e8 shortest paths corner to corner, 8 of 120 9e10."""
    ids = np.arange(sum(strips) * cols).reshape(-1, cols)
    a = np.concatenate([ids[:, :-1].ravel(), ids[:-1].ravel()])
    b = np.concatenate([ids[:, 1:].ravel(), ids[1:].ravel()])
    g = fg.Graph.from_edges(np.concatenate([a, b]).astype(np.int32), np.concatenate([b, a]).astype(np.int32),
                            np.full(2 * a.size, 40.0))
    cs = fg.ClusterSet.from_lists(np.split(np.arange(ids.size, dtype=np.int32), np.cumsum(strips)[:-1] * cols)).with_borders(g)
    ref = fg.cluster_eval_batch(g, cs, fg.FP64, fg.PLAIN)
    plan = fg.ClusterPlan(g, cs, prec)
    assert plan.captured
    for run in range(3):
        st = fg.Stats()
        ev = plan.run(st)
        assert (st.retries > 0) == (run == 0)
        assert rel_err(ev.intra_bc, ref.intra_bc) <= tol
        assert np.array_equal(ev.border_dist, ref.border_dist) and np.array_equal(ev.border_sigma, ref.border_sigma)
