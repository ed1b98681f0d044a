"""A brain is tuned while another thread allocates, copies and steps a brain of its own."""
import threading

import pytest
import torch

from flyb200 import autotune
from test_gpu_windows import brain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("single", [False, True])
def test_tuning_beside_another_threads_work(monkeypatch, single):
    monkeypatch.setattr(autotune, "CACHE", {})
    alone, tuned = brain(32, "step", False), brain(32, "step", False)
    done, errors, rounds = threading.Event(), [], []

    def work():
        try:
            other = brain(3, "persistent", False)
            with torch.cuda.stream(torch.cuda.Stream()):
                while not done.is_set() and len(rounds) < 2000:
                    x = torch.empty(1_000_003 + 4096 * len(rounds), device="cuda")
                    x[:3].copy_(torch.ones(3))
                    other.step(7)
                    other.check()
                    rounds.append(float(x[0]))
        except Exception as e:                     # noqa: BLE001 - reported by the test
            errors.append(e)

    thread = threading.Thread(target=work)
    thread.start()
    try:
        tuned.single_steps = single
        choice = autotune.tune_lif(tuned, steps=4)
    finally:
        done.set()
        thread.join()
    assert not errors and rounds and choice["ms_per_step"] > 0
    for b in (alone, tuned):
        b.launch, b.staged, b.defer, b.pull = "step", False, False, False
        b._make_args()
        b.step(9)
        b.check()
    assert torch.equal(alone.v, tuned.v) and torch.equal(alone.ring, tuned.ring)
