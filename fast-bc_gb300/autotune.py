"""Autotuner for the batched schedule's knobs.

Picks, per workload, the bucket width of the near-far distance pass (``delta``), the block
size of the frontier kernel (``frontier_threads``, ``wide_threads``) where that is what runs and the number of sources
per work item of the shared-memory kernels (``chunk_max``) by timing candidates on a sample of the
workload's units with the library's own CUDA events (``Stats.kernel_ms``).  Results only
change speed, never values: every candidate computes the same distances, path counts and
dependencies (a vertex's dependency is summed in adjacency order whatever the schedule).

    choice = autotune.tune_pivots(graph, sources, cards, fg.FP32C)      # applies and returns it
    choice = autotune.tune_clusters(graph, cluster_set, fg.FP32C)
"""
from __future__ import annotations

import itertools

import numpy as np

import fastbc_gpu as fg


def _time(f, reps: int = 3) -> float:
    # the least of a few runs: candidates a percent or two apart are otherwise picked by noise
    best = float("inf")
    for _ in range(reps):
        st = fg.Stats()
        f(st)
        best = min(best, st.kernel_ms)
    return best


def _mean_weight(g: fg.Graph) -> float:
    _, _, w = g.csr()
    return float(np.mean(w)) if w.size else 1.0


def _apply(choice: dict) -> dict:
    for k, v in choice.items():
        fg.set_option(k, int(v))
    return choice


def _search(time_of, deltas, knob: str, values) -> dict:
    """The fastest of the deltas (with the knob as it is) and, where the knob matters, of all their combinations
    with its values.  It does not on graphs that the team and log kernels take, which is most of them: then all its
    values time alike (within 2%), and it stays as it was."""
    was = fg.get_option(knob)
    tried = {}

    def timed(delta, value):
        if (delta, value) not in tried:
            _apply({"delta": delta, knob: value})
            tried[delta, value] = time_of()
        return tried[delta, value]

    mid = deltas[len(deltas) // 2]
    own = timed(mid, was)
    matters = any(abs(timed(mid, v) - own) > 0.02 * own for v in values)
    for delta, value in itertools.product(deltas, values if matters else (was,)):
        timed(delta, value)
    if not matters:
        tried = {k: t for k, t in tried.items() if k[1] == was}
    delta, value = min(tried, key=tried.get)
    return _apply({"delta": delta, knob: value})


def tune_pivots(g: fg.Graph, sources, cards=None, precision: int = fg.FP32C, sample: int = 4096,
                deltas=(2, 4, 8), threads=(64, 96, 128, 512)) -> dict:
    """Whole-graph sources (pivots, exact mode): delta (as multiples of the mean weight) and, for graphs that
    only the frontier kernel takes, its block size (of wide_n or more vertices, which run one source per SM, the
    wide block size, 512 or 1024 threads, and wider buckets).  Up to `sample`
    sources the whole list is timed, so the number of waves over the concurrent slots (which the
    block size sets) is the real one."""
    knob, reps = "frontier_threads", 3
    if g.n >= fg.get_option("wide_n"):
        knob, threads, deltas, reps = "wide_threads", (512, 1024), (4, 8, 16), 2
    src = np.asarray(sources, np.int32)
    idx = np.linspace(0, src.size - 1, min(sample, src.size)).astype(np.int64)
    s = src[idx]
    c = None if cards is None else np.asarray(cards, np.float64)[idx]
    mw = _mean_weight(g)
    return _search(lambda: _time(lambda st: fg.dependency_batch(g, s, c, precision, fg.BATCHED, stats=st), reps),
                   [max(1, int(round(dm * mw))) for dm in deltas], knob, threads)


def tune_clusters(g: fg.Graph, cs: fg.ClusterSet, precision: int = fg.FP32C, sample: int = 16,
                  deltas=(2, 4, 8), chunks=(128, 512), threads=(128,)) -> dict:
    """Cluster sources: delta, the shared-memory kernels' chunk size and (for clusters that only the
    frontier kernel takes) its block size, on a sample of the clusters (every k-th,
    keeping the size mix)."""
    cs = cs.with_borders(g)
    k = max(1, cs.count // sample)
    pick = list(range(0, cs.count, k))
    sub = fg.ClusterSet.from_lists([cs.vertices[cs.off[c]:cs.off[c + 1]] for c in pick],
                                   [cs.borders[cs.boff[c]:cs.boff[c + 1]] for c in pick])
    mw = _mean_weight(g)
    best, arg = float("inf"), None
    for dm, ch, bt in itertools.product(deltas, chunks, threads):
        choice = {"delta": max(1, int(round(dm * mw))), "chunk_max": ch, "frontier_threads": bt}
        _apply(choice)
        t = _time(lambda st: fg.cluster_eval_batch(g, sub, precision, fg.BATCHED, stats=st))
        if t < best:
            best, arg = t, choice
    return _apply(arg)
