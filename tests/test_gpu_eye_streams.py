"""Poses that `column_radiance` queued on one stream reach a trace on another, eager or replayed."""
import numpy as np
import pytest
import torch

from flyb200 import world as W
from flyb200.batch_world import BatchWorld

pytestmark = pytest.mark.gpu

BUSY = 60_000_000        # clock cycles a stream is kept busy with: some 30 ms


def _eye(batch):
    rng = np.random.default_rng(5)
    az, el = rng.uniform(-np.pi, np.pi, (80, 7)), rng.uniform(-1.2, 1.2, (80, 7))
    b = BatchWorld([W.make_room(i)[0] for i in range(batch)], device="cuda")
    b.set_eye(np.stack([np.cos(el) * np.cos(az), np.cos(el) * np.sin(az), np.sin(el)], -1), np.ones(7))
    return b


def _pose(batch, seed):
    rng = np.random.default_rng(seed)
    eye = np.c_[rng.uniform(-1.5, 1.5, (batch, 2)), rng.uniform(0.8, 1.5, batch)]
    h = rng.uniform(-np.pi, np.pi, batch)
    forward, left = np.c_[np.cos(h), np.sin(h), np.zeros(batch)], np.c_[-np.sin(h), np.cos(h), np.zeros(batch)]
    return eye, forward, left, np.cross(forward, left)


@pytest.mark.parametrize("replayed", [False, True])
@pytest.mark.parametrize("batch", [1, 5])
def test_poses_queued_on_a_busy_stream_reach_a_trace_on_another(batch, replayed):
    b = _eye(batch)
    want = b.column_radiance(*_pose(batch, 1)).clone()
    b.set_pose(*_pose(batch, 2))
    other = b.trace_eye()
    busy, free = torch.cuda.Stream(), torch.cuda.Stream()
    if replayed:
        got = torch.zeros_like(want)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=free):
            b.trace_eye(got)
    torch.cuda.synchronize()
    assert not torch.equal(want, other)
    with torch.cuda.stream(busy):
        torch.cuda._sleep(BUSY)
        queued = b.column_radiance(*_pose(batch, 1))
    with torch.cuda.stream(free):
        if replayed:
            graph.replay()
        else:
            got = b.trace_eye()
    torch.cuda.synchronize()
    assert torch.equal(queued, want) and torch.equal(got, want)
