"""The plain kernel's two ways over a warp's rows (each lane its own row when all 32 have at most 16
edges, else the warp together) and its block sizes: row lengths around a multiple of four and around
16, rows of both kinds in one frontier, path counts that leave 64 bits, and the numbers of sources above
which smaller blocks run.  Against the oracle's exact BC."""
import numpy as np
import pytest

import graphs
import oracle
from test_gpu_parity import rel_err
from test_gpu_team import FORMS, _both, _graph

pytestmark = pytest.mark.gpu


def _check(fg, g, og):
    ref = oracle.exact_bc(og)
    for prec, tol in FORMS:
        assert rel_err(fg.exact_bc(g, prec, fg.PLAIN), ref) <= tol


@pytest.mark.parametrize("deg", [1, 3, 4, 5, 8, 15, 16, 17, 18, 33])
def test_row_lengths(fg, deg):
    """A ring of 40 hubs, each with deg - 2 further edges (leaves, some shared with the next hub)."""
    rng = np.random.default_rng(deg)
    a, b, nxt = list(range(40)), [(i + 1) % 40 for i in range(40)], 40
    for i in range(40):
        for _ in range(max(0, deg - 2)):
            a.append(i)
            b.append(nxt)
            if rng.integers(2):
                a.append((i + 1) % 40)
                b.append(nxt)
            nxt += 1
    w = rng.integers(1, 6, len(a))
    g, og = _graph(fg, *_both(np.array(a), np.array(b), w, w))
    _check(fg, g, og)


def test_one_long_row_among_short_ones(fg):
    el = graphs.road_grid(20, 23, seed=4)
    extra = np.arange(1, 460, 9)
    s = np.concatenate([el.src, np.zeros(extra.size, int), extra])
    d = np.concatenate([el.dst, extra, np.zeros(extra.size, int)])
    w = np.concatenate([el.w, np.full(2 * extra.size, 40)])
    g, og = _graph(fg, s, d, w)
    _check(fg, g, og)


@pytest.mark.parametrize("rows,cols", [(1, 2), (5, 13), (19, 32), (21, 29), (32, 38), (33, 37), (39, 40)])
def test_block_sizes(fg, rows, cols):
    """Above 608 and 1,216 sources (four and eight a multiprocessor) the blocks become smaller."""
    el = graphs.road_grid(rows, cols, seed=rows)
    _check(fg, fg.Graph.from_edgelist(el), oracle.CSR.from_edgelist(el))


def test_counts_beyond_64_bits(fg):
    """A chain of 70 diamonds: 2^70 shortest paths end to end, so the end sources run with FP64 counts."""
    k = 70
    j, m = np.arange(k) * 3, np.arange(k) * 3 + 1
    a = np.concatenate([j, j, m, m + 1])
    b = np.concatenate([m, m + 1, j + 3, j + 3])
    w = np.full(a.size, 2)
    g, og = _graph(fg, *_both(a, b, w, w))
    _check(fg, g, og)
