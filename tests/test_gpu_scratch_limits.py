"""Calls with little device memory left: what the team and log kernels take besides the older kernels' memory (rows
as quads) is no reason to fail, the older kernels run instead."""
import subprocess
import sys

import numpy as np
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


def test_whole_graph_with_room_for_the_frontier_kernel_only(fg, left):
    """1M vertices: a source of the frontier kernel needs some 60 bytes a vertex, one of the log kernel 45 and its quads 36."""
    el = graphs.road_grid(1000, 1000, seed=3)
    src = np.array([1234, 777777], np.int32)
    csr = fg.Graph.from_edgelist(el)
    ref = fg.dependency_batch(csr, src, None, fg.FP64, fg.BATCHED)
    fg.set_option("warp_max_n", 0)
    fg.dependency_batch(csr, src, None, fg.FP64, fg.BATCHED)  # (what both keep is allocated)
    fg.set_option("warp_max_n", 4096)
    csr.free()
    small = fg.Graph.from_edgelist(graphs.road_grid(5, 5, seed=1))
    fg.exact_bc(small, fg.FP64, fg.PLAIN)  # (a kernel's first launch takes memory too)
    ran = 0
    for m in range(24, 105, 8):
        left(0)
        g = fg.Graph.from_edgelist(el)  # (a graph keeps its quads)
        left(m)
        try:
            out = fg.dependency_batch(g, src, None, fg.FP64, fg.BATCHED)
        except fg.FbcError as e:
            assert e.code == fg.FBC_ERR_OOM
            left(m)
            fg.set_option("warp_max_n", 0)
            with pytest.raises(fg.FbcError):
                fg.dependency_batch(g, src, None, fg.FP64, fg.BATCHED)
            fg.set_option("warp_max_n", 4096)
        else:
            assert np.allclose(out, ref, rtol=1e-9, atol=1e-9)
            ran += 1
        g.free()
    assert 4 <= ran <= 9


_CHILD = """
import sys
sys.path[:0] = {paths!r}
import numpy as np, torch
import fastbc_gpu as fg, graphs
fg.init(0)
one = graphs.road_grid(25, 40, seed=4)  # 200 communities of 1,000 vertices, without borders
at = np.arange(200)[:, None] * 1000
g = fg.Graph.from_edges((one.src + at).ravel().astype(np.int32), (one.dst + at).ravel().astype(np.int32), np.tile(one.w, 200).astype(float))
cs = fg.ClusterSet.from_lists(np.split(np.arange(200000, dtype=np.int32), 200)).with_borders(g)
few = fg.ClusterSet.from_lists([np.arange(1000, dtype=np.int32)]).with_borders(g)
def run(which, cs):
    return (fg.cluster_eval_batch(g, cs, fg.FP32C, fg.BATCHED) if which == "sweep" else fg.ClusterPlan(g, cs, fg.FP32C).run()).intra_bc
ref = fg.cluster_eval_batch(g, cs, fg.FP64, fg.PLAIN).intra_bc
h = fg.Graph.from_edgelist(graphs.rgg_knn(400, k=20))  # every kernel's first launch, which takes memory too
fg.exact_bc(h, fg.FP32C, fg.BATCHED)
fg.exact_bc(h, fg.FP64, fg.PLAIN)
run({which!r}, few)
fg.set_option("ws_budget_mb", 1)  # kept workspaces and scratch go
fg.exact_bc(h, fg.FP64, fg.PLAIN)
fg.set_option("ws_budget_mb", 0)
fg.set_option("scratch_keep_mb", 0)
for m in {sizes!r}:
    torch.cuda.synchronize()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (m << 20), dtype=torch.uint8, device="cuda")
    try:
        print(m, "ok" if np.allclose(run({which!r}, cs), ref, rtol=1e-6, atol=1e-6) else "wrong")
    except fg.FbcError as e:
        print(m, str(e).replace(" ", "_"))
    del fill
    torch.cuda.empty_cache()
"""


@pytest.mark.parametrize("which,sizes", [("sweep", [14, 200]), ("plan", [32, 200])])
def test_communities_without_room_for_their_quads(fg, which, sizes):
    """Quads and units of the communities take 14 MB of the library's (and of a plan) beside the older kernels' 8."""
    pytest.importorskip("torch")
    code = _CHILD.format(paths=sys.path[:4], sizes=sizes, which=which)
    out = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stderr
    assert out.stdout.split() == [w for m in sizes for w in (str(m), "ok")]
