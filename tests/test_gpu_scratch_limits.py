"""Calls with little device memory left."""
import pytest

import graphs
from test_gpu_parity import TOL_FP64, rel_err

pytestmark = pytest.mark.gpu
MB = 1 << 20


@pytest.fixture
def left(fg):
    """left(m): the device with m MB free, kept workspaces and scratch given back first."""
    torch = pytest.importorskip("torch")
    old = {k: fg.get_option(k) for k in ("ws_budget_mb", "warp_max_n", "order_min_n", "scratch_keep_mb")}
    tiny = fg.Graph.from_edgelist(graphs.road_grid(5, 5, seed=1))
    held = []

    def leave(m):
        held.clear()
        torch.cuda.empty_cache()
        if m:
            fg.set_option("ws_budget_mb", 1)  # a workspace above the cap goes, and those beside it
            fg.exact_bc(tiny, fg.FP64, fg.PLAIN)
            fg.set_option("ws_budget_mb", 0)
            torch.cuda.synchronize()
            held.append(torch.empty(torch.cuda.mem_get_info()[0] - m * MB, dtype=torch.uint8, device="cuda"))

    fg.set_option("order_min_n", 1 << 30)
    fg.set_option("scratch_keep_mb", 0)
    try:
        yield leave
    finally:
        leave(0)
        for k, v in old.items():
            fg.set_option(k, v)


def test_the_call_after_one_without_memory(fg, left):
    g = fg.Graph.from_edgelist(graphs.road_grid(1000, 1000, seed=3))
    h = fg.Graph.from_edgelist(graphs.road_grid(9, 9, seed=3))
    ref = fg.exact_bc(h, fg.FP64, fg.PLAIN)
    left(4)
    with pytest.raises(fg.FbcError) as e:
        fg.single_source(g, 5)
    assert e.value.code == fg.FBC_ERR_OOM
    assert rel_err(fg.exact_bc(h, fg.FP64, fg.PLAIN), ref) <= TOL_FP64  # (summed in any order)
