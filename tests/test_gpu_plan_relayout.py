"""A prepared sweep that is captured again after its first run (a community's path counts outgrew their
kernel) while another community runs on the frontier kernel, whose slots the first run has used: the
new capture starts from cleared slots and keeps the options of the plan's creation, so options changed
between creation and the first run leave the results of every run as they are."""
import numpy as np
import pytest

import graphs
from test_gpu_parity import rel_err
from test_gpu_team import FORMS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("before,after", [({"group": 4}, {"group": 1}), ({"group": 4}, {"group": 2, "frontier_threads": 64}),
                                          ({"group": 0}, {"group": 1}), ({"group": 1}, {"warp_max_n": 0})])
@pytest.mark.parametrize("prec,tol", FORMS)
def test_slots_and_options_of_the_new_capture(fg, before, after, prec, tol):
    """900 vertices of equal weights (3e16 shortest paths corner to corner) beside a road grid of 10,500
    vertices with weights above 255, which only the frontier kernel takes."""
    ids = np.arange(900).reshape(30, 30)
    a = np.concatenate([ids[:, :-1].ravel(), ids[:-1].ravel()])
    b = np.concatenate([ids[:, 1:].ravel(), ids[1:].ravel()])
    el = graphs.road_grid(100, 105, seed=4)
    src = np.concatenate([a, b, el.src + 900, [899, 900]])
    dst = np.concatenate([b, a, el.dst + 900, [900, 899]])
    w = np.concatenate([np.full(2 * a.size, 40.0), 3.0 * el.w, [300.0, 300.0]])
    g = fg.Graph.from_edges(src.astype(np.int32), dst.astype(np.int32), w)
    cs = fg.ClusterSet.from_lists([np.arange(900, dtype=np.int32), np.arange(900, g.n, dtype=np.int32)]).with_borders(g)
    ref = fg.cluster_eval_batch(g, cs, fg.FP64, fg.PLAIN)
    old = {k: fg.get_option(k) for k in {**before, **after}}
    try:
        for k, v in before.items():
            fg.set_option(k, v)
        plan = fg.ClusterPlan(g, cs, prec)
        assert plan.captured
        for k, v in after.items():
            fg.set_option(k, v)
        for run in range(3):
            st = fg.Stats()
            ev = plan.run(st)
            assert run == 0 or st.retries == 0  # replayed
            assert rel_err(ev.intra_bc, ref.intra_bc) <= tol
            assert np.array_equal(ev.border_dist, ref.border_dist) and np.array_equal(ev.border_sigma, ref.border_sigma)
    finally:
        for k, v in old.items():
            fg.set_option(k, v)
