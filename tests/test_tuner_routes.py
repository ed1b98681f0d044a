"""The LIF tuner tells candidates apart that run different kernels, and only those (host logic, no GPU)."""
import pytest
import torch

from flyb200 import autotune


class FakeBrain:
    """As much of a Brain as the tuner touches; per-step kernels only where `defer` or `staged` ask for them."""
    n, B, step_count, pull_group, device = 4096, 64, 0, 4, torch.device("cpu")
    launch, block, items_per_thread, staged, defer, pull = "step", 256, 0, False, False, False

    def __init__(self, honoured):
        self.honoured = honoured

    def can_pull(self):
        return True

    def _make_args(self):
        pass

    def state_dict(self):
        return {}

    def load_state_dict(self, state):
        pass

    def window_steps(self, steps):
        return 0 if self.honoured and not self.pull and (self.staged or self.defer) else steps

    def step(self, steps):
        pass

    def candidate(self):
        kind = ("staged-" if self.staged else "") + ("pull" if self.pull else "defer" if self.defer else "")
        return self.launch, self.block, self.items_per_thread, kind.strip("-") or "fused"


@pytest.mark.parametrize("honoured,fast_run,fast_one,want,timings", [
    (False, ("step", True), ("step", 512, 2, "staged-pull"), ("step", 512, 2, "staged-pull"), 3),
    (False, ("step", False), ("step", 256, 4, "staged-defer"), ("step", 256, 4, "staged-defer"), 3),
    (False, ("persistent", False), ("persistent", 512, 2, "fused"), ("persistent", 512, 2, "fused"), 3),
    (True, ("step", 128, 2, "defer"), ("step", 256, 1, "fused"), ("step", 128, 2, "defer"), 3 + 12),
])
def test_equal_runs_are_timed_once_and_told_apart_by_single_steps(monkeypatch, honoured, fast_run, fast_one, want, timings):
    brain, taken = FakeBrain(honoured), []

    def run_ms(fn, reps):                       # a run's time by what it runs, with noise that favours the last
        c = brain.candidate()
        route = c if not brain.window_steps(10) else (c[0], "pull" in c[3])
        taken.append(route)
        return (1.0 if route == fast_run else 2.0) - 0.001 * len(taken)

    monkeypatch.setattr(autotune, "CACHE", {})
    monkeypatch.setattr(autotune, "graph_key", lambda b: "graph")
    monkeypatch.setattr(autotune, "activity_bucket", lambda b: 0)
    monkeypatch.setattr(autotune, "_time", run_ms)
    monkeypatch.setattr(autotune, "_time_one_by_one", lambda b, steps: 1.0 if b.candidate() == fast_one else 2.0)
    choice = autotune.tune_lif(brain)
    assert (choice["launch"], choice["block"], choice["items_per_thread"], choice["delivery"]) == want == brain.candidate()
    assert len(taken) == timings and len(set(taken)) == timings
    assert len(choice["all"]) == len(autotune.LIF_CANDIDATES)
