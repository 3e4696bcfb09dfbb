"""The autotuner times the kernel that its launch shapes shape (no GPU: the solver is a stand-in): calls that would
take the cooperative kernel by their size are timed with it switched off, in the tuner and in the sweep."""
import numpy as np
import pytest

from cmaq_gb300 import autotune
from cmaq_gb300.synthetic import make_grid


class Solver:
    """ChemSolver's calls; a step takes as long as the launch shape says, or 1 ms by the cooperative kernel."""

    made = []

    def __init__(self, *a, **kw):
        self.knobs = {}
        Solver.made.append(self)

    def set_tuning(self, **kw):
        self.knobs.update(kw)

    def step(self, *a, **kw):
        coop = self.knobs.get("ros3_coop", -1) != 0
        ms = 1.0 if coop else 10.0 * self.knobs["block_warps"] + self.knobs["lockstep"]
        return {"device_ms": ms, "accepted_steps": 1, "rejected_steps": 0, "sunlit_attempts": 0}

    def steps(self, n, *a, **kw):
        return self.step()

    def close(self):
        pass


@pytest.fixture
def stand_in(monkeypatch):
    import torch
    Solver.made = []
    monkeypatch.setattr(autotune, "ChemSolver", Solver)
    monkeypatch.setattr(torch.Tensor, "cuda", lambda self, *a, **kw: self)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda *a: None)


def test_candidates_are_timed_on_the_work_queue(stand_in, tmp_path):
    g = make_grid(ncols=4, nrows=3, nlays=2, seed=1)
    res = autotune.tune(g, variants=("default",), cache=tmp_path / "c.json")
    assert len({r["ms"] for r in res["table"]}) == len(res["table"])      # each shape its own time
    assert (res["block_warps"], res["lockstep"]) == (2, 1)


def test_the_sweep_times_the_work_queue(stand_in):
    g = make_grid(ncols=4, nrows=3, nlays=2, seed=1)
    out = autotune.sweep(g, ["default:2:1", "default:8:2"], ncalls=1, reps=1, verbose=False)
    assert out["default:2:1"][0]["ms"] == 21.0 and out["default:8:2"][0]["ms"] == 82.0


def test_results_of_earlier_timings_are_not_taken(tmp_path):
    """A cache key names what was timed: entries stored before, under mechanism, GPU and size alone, are not found."""
    assert autotune.cache_key("cb6r5_ae7_aq", 40000).count("|") > 2
