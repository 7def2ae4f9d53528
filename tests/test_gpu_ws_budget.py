"""`ws_budget_mb` caps what the plain, frontier and log kernels keep for their slots together: with a small
cap set, workspaces of earlier calls go, results stay as they are, and a call alternating between the kernels
never holds more than the cap beside what the rest of the library holds."""
import numpy as np
import pytest

import graphs
import oracle
from test_gpu_parity import rel_err
from test_gpu_team import FORMS

pytestmark = pytest.mark.gpu


def test_kept_workspaces_share_the_cap(fg):
    torch = pytest.importorskip("torch")
    el = graphs.road_grid(255, 255, seed=5)
    g, og = fg.Graph.from_edgelist(el), oracle.CSR.from_edgelist(el)
    src = np.linspace(0, el.n - 1, 1300).astype(np.int32)
    ref = oracle.pivot_batch(og, src[::65], np.ones(20))

    def all_kernels(which):
        out = []
        for sched, wmax in ((fg.PLAIN, 4096), (fg.BATCHED, 0), (fg.BATCHED, 4096)):  # plain, frontier, log
            fg.set_option("warp_max_n", wmax)
            out += [fg.dependency_batch(g, which, None, p, sched) for p, _ in FORMS]
        fg.set_option("warp_max_n", old["warp_max_n"])
        return out

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    old = {k: fg.get_option(k) for k in ("ws_budget_mb", "warp_max_n", "scratch_keep_mb")}
    try:
        all_kernels(src)  # some 2 GB of slots and more each
        held = free()
        fg.set_option("ws_budget_mb", 256)
        got = all_kernels(src[::65])
        for k, out in enumerate(got):
            assert rel_err(out, ref) <= FORMS[k % 2][1]
        assert free() - held >= 4 << 30
        small = free()
        all_kernels(src)
        assert small - free() <= 300 << 20
    finally:
        for k, v in old.items():
            fg.set_option(k, v)
