"""Cached choices are used while they are current: timed on these kernels and in the grid asked for."""
import json

import pytest

from master_thesis_b200 import autotune

GRID = dict(refill=[4, 8], trace_blocks=[0, 9])


@pytest.fixture
def search(tmp_path, monkeypatch):
    monkeypatch.setattr(autotune, "CACHE", str(tmp_path / "tune.json"))
    calls = []
    monkeypatch.setattr(autotune, "_time", lambda fn, reps: (fn(), float(len(calls)))[1])

    def run(grid=GRID, entry=None):
        if entry is not None:
            (tmp_path / "tune.json").write_text(json.dumps({"k": entry}))
        del calls[:]
        return autotune._search("k", grid, calls.append, 1, False), len(calls)
    return run


def test_current_choice_is_served(search):
    best, timed = search()
    assert timed == 4 and best == dict(refill=4, trace_blocks=0)
    assert search() == (best, 0)


@pytest.mark.parametrize("entry", [
    dict(best=dict(refill=8, trace_blocks=10), ms=1.0),  # before the kernels were counted
    dict(best=dict(refill=8, trace_blocks=9), ms=1.0),
    dict(best=dict(refill=8, trace_blocks=9), ms=1.0, kernels=autotune.KERNELS - 1),
    dict(best=dict(refill=8, trace_blocks=10), ms=1.0, kernels=autotune.KERNELS),  # not in the grid
    dict(best=dict(refill=8), ms=1.0, kernels=autotune.KERNELS),  # without a knob of the grid
])
def test_stale_choice_is_searched_again(search, entry):
    assert search(entry=entry) == (dict(refill=4, trace_blocks=0), 4)
    assert search()[1] == 0


def test_another_grid_is_searched(search):
    search()
    assert search(dict(refill=[16], trace_blocks=[0])) == (dict(refill=16, trace_blocks=0), 1)
