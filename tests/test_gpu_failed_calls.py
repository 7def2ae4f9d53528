"""What a failed call leaves behind: a single source's output is zeros, whichever kernel was to run it."""
import ctypes as C

import numpy as np
import pytest

import graphs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,warp_max_n", [(20, 31, 4096), (150, 140, 4096), (20, 31, 0)])  # team, log, plain
def test_failed_single_source_leaves_zeros(fg, rows, cols, warp_max_n):
    g = fg.Graph.from_edgelist(graphs.road_grid(rows, cols, seed=2))
    old = {k: fg.get_option(k) for k in ("iter_mult", "warp_max_n")}
    out = np.full(g.n, 7.0)
    try:
        fg.set_option("warp_max_n", warp_max_n)
        fg.set_option("iter_mult", 0)
        rc = fg.lib.fbc_single_source(g._h, 3, fg.FP64, out.ctypes.data_as(C.c_void_p), None)
        assert rc == fg.FBC_ERR_ITER_LIMIT and not out.any()
        fg.set_option("iter_mult", old["iter_mult"])
        out[:] = 7.0
        assert fg.lib.fbc_single_source(g._h, 3, 9, out.ctypes.data_as(C.c_void_p), None) == fg.FBC_ERR_INVALID_ARG
        assert not out.any()
    finally:
        for k, v in old.items():
            fg.set_option(k, v)
