"""Downloading a graph that was built on the device: with next to no device memory left, and with only
some of the arrays asked for."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ring(fg, n):
    v = np.arange(n, dtype=np.int32)
    return fg.Graph.from_edges(np.tile(v, 3), np.concatenate([(v + k) % n for k in (1, 2, 3)]).astype(np.int32),
                               np.repeat([5.0, 11.0, 17.0], n))


def _ring_csr(n):
    col = (np.arange(n, dtype=np.int64)[:, None] + [1, 2, 3]) % n
    at = np.argsort(col, axis=1)
    return np.arange(n + 1) * 3, np.take_along_axis(col, at, 1).ravel(), np.tile([5.0, 11.0, 17.0], (n, 1))[np.arange(n)[:, None], at].ravel()


def test_download_needs_no_device_memory(fg):
    """4M vertices, 12M edges: 176 MB in the caller's types, with 64 MB left on the device."""
    torch = pytest.importorskip("torch")
    n = 4_000_000
    old = fg.get_option("scratch_keep_mb")
    fg.set_option("scratch_keep_mb", 0)  # the pool keeps nothing that the call could use
    fill = None
    try:
        g = _ring(fg, n)
        _ring(fg, 70_000).csr()
        torch.cuda.synchronize()
        fill = torch.empty(torch.cuda.mem_get_info()[0] - (64 << 20), dtype=torch.uint8, device="cuda")
        got = g.csr()
    finally:
        del fill
        torch.cuda.empty_cache()
        fg.set_option("scratch_keep_mb", old)
    assert all(np.array_equal(a, b) for a, b in zip(got, _ring_csr(n)))


@pytest.mark.parametrize("want", [(1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (0, 0, 0)])
def test_only_the_arrays_asked_for(fg, want):
    n = 70_000
    g = _ring(fg, n)
    out = [np.full(n + 1, -1, np.int64), np.full(3 * n, -1, np.int32), np.full(3 * n, -1.0)]
    ptr = [a.ctypes.data_as(C.c_void_p) if k else None for a, k in zip(out, want)]
    assert fg.lib.fbc_graph_download(g._h, *ptr) == fg.FBC_OK
    for a, k, ref in zip(out, want, _ring_csr(n)):
        assert np.array_equal(a, ref) if k else np.all(a == -1)
