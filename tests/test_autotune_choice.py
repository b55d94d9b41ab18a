"""The tuner's choice among its timed candidates, with a solver whose steps take
given times (no GPU): the default sweep stays unless another is clearly faster,
since the state it is timed on, usually the lattice at rest, is not the one a run
spends its time in."""
from types import SimpleNamespace

import pytest

from aquagpusph_gb300 import autotune as at


class Clock:
    def __init__(self, times):
        self.now, self.times, self.tuning = 0.0, times, None
        self.N = 5878404
        self.params = SimpleNamespace(dims=3, h=0.01, boundary=0, scheme=0)

    def set_tuning(self, v, b):
        self.tuning = (v, b)

    def step(self, n, graph=True, stream=None):
        self.now += n * self.times.get(self.tuning, self.times.get(self.tuning[0], 30.0)) * 1e-3

    def scalars(self, stream=None):
        pass

    check = scalars


def choose(monkeypatch, times, fast=False):
    sv = Clock(times)
    monkeypatch.setattr(at, "gpu_name", lambda: "none")
    monkeypatch.setattr(at, "time", SimpleNamespace(perf_counter=lambda: sv.now))
    c = at.autotune(sv, fast, use_cache=False)
    assert sv.tuning == (c["variant"], c["blocks_per_sm"])
    assert len(c["candidates"]) == len(list(at.candidates(at.clustered_applies(sv, fast))))
    return c


def test_default_stays_beside_a_slightly_faster_variant(monkeypatch):
    """The queued sweep by 3% on the lattice (it is 2 to 20% slower off it)."""
    c = choose(monkeypatch, {16: 19.2, (1, 12): 18.7, (11, 16): 19.9})
    assert (c["variant"], c["blocks_per_sm"]) == (16, 3)
    assert c["ms_per_step"] == pytest.approx(19.2)


def test_a_clearly_faster_variant_is_taken(monkeypatch):
    c = choose(monkeypatch, {16: 19.2, (1, 12): 17.0, (11, 16): 16.5})
    assert (c["variant"], c["blocks_per_sm"]) == (11, 16)
    assert c["ms_per_step"] == pytest.approx(16.5)


def test_blocks_of_the_default_are_chosen_freely(monkeypatch):
    c = choose(monkeypatch, {(16, 1): 9.0, (16, 2): 6.1, (16, 3): 6.2, (9, 14): 6.0}, fast=True)
    assert (c["variant"], c["blocks_per_sm"]) == (16, 2)


def test_choices_of_the_old_rule_do_not_apply():
    sv = Clock({})
    assert at.signature(sv, False).endswith("|default")
