"""Replays of captured steps mixed with ordinary steps, with the launches
recorded on the CPU: whatever numbers of launches the steps take, a replay
advances the state where it is, and the books agree with it."""

import contextlib

import pytest
import torch

from latticeboltzmann_gb300 import solver


class FakeGraph:
    recording = None

    def __init__(self):
        self.launches = []

    def replay(self):
        for launch in self.launches:
            launch()


class FakeLattice:
    """Two buffers that each count the steps in them; a launch takes up to ``most``."""

    device = torch.device("cpu")

    def __init__(self, most):
        self.most, self.buf, self._cur, self.steps_taken = most, [0, 0], 0, 0

    def step(self, n):
        left = n
        while left > 0:
            t = min(left, self.most)
            src, dst = self._cur, 1 - self._cur

            def launch(src=src, dst=dst, t=t):
                self.buf[dst], self.buf[src] = self.buf[src] + t, -1000
            FakeGraph.recording.launches.append(launch) if FakeGraph.recording else launch()
            self._cur = dst
            left -= t
        self.steps_taken += n


@pytest.fixture
def fake_cuda(monkeypatch):
    class Stream:
        def __init__(self, device=None):
            pass

        def wait_stream(self, other):
            pass

    @contextlib.contextmanager
    def graph(g, stream=None):
        FakeGraph.recording = g
        yield
        FakeGraph.recording = None

    monkeypatch.setattr(torch.cuda, "Stream", Stream)
    monkeypatch.setattr(torch.cuda, "current_stream", Stream)
    monkeypatch.setattr(torch.cuda, "CUDAGraph", FakeGraph)
    monkeypatch.setattr(torch.cuda, "graph", graph)
    monkeypatch.setattr(torch.cuda, "stream", lambda s: contextlib.nullcontext())


@pytest.mark.parametrize("most", [1, 2, 4, 6, 8])
@pytest.mark.parametrize("n", [2, 6, 8, 10])
@pytest.mark.parametrize("m", [1, 2, 3, 4])
def test_replay_advances_the_state_where_it_is(fake_cuda, most, n, m):
    lat = FakeLattice(most)
    lat.step(1)
    replay = solver.Replay(lat, n)
    assert lat.steps_taken == 1 and lat.buf[lat._cur] == 1
    total = 1
    for part in (n, m, n, n, m, m, n):
        replay() if part == n else lat.step(part)
        total += part
        assert lat.buf[lat._cur] == lat.steps_taken == total
    cur = lat._cur
    replay.graph.replay()
    assert lat._cur == cur and lat.buf[cur] == total + n
