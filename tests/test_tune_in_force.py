"""A tuning run that finds no clear winner leaves the setting in force: the library's own choice
of group cells is not switched off by a sample that gains little from it."""
import pytest
import torch

from hyperflow_gb300 import tune


class Ctx:
    """The tuning entry points of a library that starts at its default, and nothing else."""

    def __init__(self):
        self.now = [4, 17]
        self.lib = self

    def hf_get_chem_tuning(self, m, c):
        m._obj.value, c._obj.value = self.now

    def hf_set_chem_tuning(self, m, c):
        self.now = [m or self.now[0], c or self.now[1]]
        return 0

    def check(self, st, what):
        assert st == 0

    def counters(self):
        return {"chem_coop_cells": 0, "chem_steps": 0}


@pytest.fixture
def ctx(monkeypatch):
    """times[setting] is what a call or a step takes under it."""
    ctx = Ctx()
    ctx.times = {}

    class Event:
        def record(self):
            pass

        def elapsed_time(self, other):
            return ctx.times.get(tuple(ctx.now), 100.0)

    class Work:
        def __init__(self, *a, **k):
            pass

        def advance(self, *a):
            pass

        step = run = close = lambda self, *a, **k: None

    monkeypatch.setattr(tune, "_events", lambda: (Event(), Event()))
    monkeypatch.setattr(tune.S, "ChemistryBatch", Work)
    monkeypatch.setattr(tune.S, "Stepper", Work)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda: None)
    return ctx


def run(ctx, which):
    if which == "call":
        return tune.tune_chemistry(ctx, torch.zeros(12, 4), 1e-7)
    return tune.tune_stepper(ctx, None, None, 0.5)


@pytest.mark.parametrize("which", ["call", "steps"])
@pytest.mark.parametrize("times,want", [
    ({}, (4, 17)),                                        # all alike
    ({(4, 17): 98.0}, (4, 17)),                           # it gains less than the margin
    ({(4, 17): 102.0}, (4, 17)),
    ({(4, 17): 60.0}, (4, 17)),
    ({(4, 17): 102.0, (4, 7): 98.0}, (4, 16)),            # 4% behind the fastest, which is 2% ahead of no groups
    ({(4, 3): 60.0}, (4, 3)),                             # a clear winner
    ({(4, 17): 120.0}, (4, 16)),                          # the setting in force is a clear loser
])
def test_what_a_run_leaves(ctx, which, times, want):
    ctx.times = times
    res = run(ctx, which)
    assert res["best"] == want == tune.get_chem_tuning(ctx)


def test_settings_with_groups_that_are_alike(ctx):
    """Whole steps: the setting in force stays; one call: the fastest of them is applied."""
    ctx.times = {(4, 17): 60.0, (4, 5): 59.5}
    assert run(ctx, "steps")["best"] == (4, 17) == tune.get_chem_tuning(ctx)
    assert run(ctx, "call")["best"] == (4, 5)


def test_a_setting_that_is_no_candidate_is_not_kept(ctx):
    ctx.now = [8, 11]
    assert run(ctx, "call")["best"] == tune.CHEM_DEFAULT


def test_the_librarys_start_is_a_candidate():
    assert (4, 17) in tune.CHEM_CANDIDATES and (4, 17) in tune.STEP_CANDIDATES
