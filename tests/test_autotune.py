"""The autotuner's choice from given timings: a knob that the running kernel does not read stays as it was, whatever the
noise, and is not swept with every delta; one that matters is (CPU: the timings are the test's)."""
import pytest

import autotune


class _Engine:
    def __init__(self, reads, noise):
        self.opt = {"delta": 0, "frontier_threads": 128, "wide_threads": 1024, "wide_n": 1000}
        self.reads, self.noise, self.calls = reads, noise, 0

    def time(self, g, s, c, precision, sched, stats):
        self.calls += 1
        t = {20: 1.2, 40: 1.0, 80: 1.1, 160: 1.3}[self.opt["delta"]]
        if self.reads:
            t *= {64: 1.3, 96: 0.9, 128: 1.0, 512: 1.5, 1024: 1.0}[self.opt[self.reads]]
        stats.kernel_ms = t * (1 + self.noise * ((self.calls * 7919) % 11 - 5) / 5)


@pytest.mark.parametrize("noise", [0.0, 0.005])
@pytest.mark.parametrize("n,reads,want", [(500, None, {"delta": 40, "frontier_threads": 128}),
                                          (500, "frontier_threads", {"delta": 40, "frontier_threads": 96}),
                                          (5000, None, {"delta": 40, "wide_threads": 1024}),
                                          (5000, "wide_threads", {"delta": 40, "wide_threads": 1024})])
def test_choice(monkeypatch, n, reads, want, noise):
    e = _Engine(reads, noise)
    fg = autotune.fg
    monkeypatch.setattr(fg, "get_option", e.opt.__getitem__)
    monkeypatch.setattr(fg, "set_option", e.opt.__setitem__)
    monkeypatch.setattr(fg, "dependency_batch", e.time)
    monkeypatch.setattr(autotune, "_mean_weight", lambda g: 10.0)
    g = type("G", (), {"n": n})()
    assert autotune.tune_pivots(g, range(100)) == want
    assert all(e.opt[k] == v for k, v in want.items())
    if reads is None:  # the deltas and, once, the knob's values
        assert e.opt["frontier_threads"] == 128 and e.opt["wide_threads"] == 1024
        assert e.calls <= (2 * (3 + 1) if n >= 1000 else 3 * (3 + 3))
