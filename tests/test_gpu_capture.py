"""Captured steps mixed with ordinary ones against single steps, bit for bit:
lattices and batches whose steps take even and odd numbers of launches."""

import numpy as np
import pytest
import torch

import latticeboltzmann_gb300 as PyLB
from latticeboltzmann_gb300 import _lib
from latticeboltzmann_gb300 import batch as B
from test_gpu_batch_steps import LARGE, SINGLE, SMALL, make
from test_gpu_march import two_step  # noqa: F401

pytestmark = pytest.mark.gpu


def mixed(lat, n, m):
    replay = lat.capture(n)
    for part in (n, m, n, n, m, n):
        replay() if part == n else lat.step(part)
    return replay, 4 * n + 2 * m


@pytest.mark.parametrize("size,storage,rounding", [((256, 256), "f32", "nearest"), ((1237, 1288), "f32", "nearest"),
                                                   ((256, 256), "f16dev", "stochastic"), ((96, 80), "f64", "nearest")])
@pytest.mark.parametrize("n", [8, 10])
@pytest.mark.parametrize("m", [2, 3, 4])
def test_lattice_replays_mixed_with_steps(two_step, cuda, size, storage, rounding, n, m):
    def lattice():
        lat = PyLB.Lattice(*size, 1.4, boundary="cavity", u0=0.05, storage=storage, rounding=rounding, seed=5, device=cuda)
        return lat.equilibrium(1.0, 0.01, 0.02)
    _lib.set_tuning(_lib.TUNE_TWO_STEP, 1)
    lat, ref = lattice(), lattice()
    replay, total = mixed(lat, n, m)
    _lib.set_tuning(_lib.TUNE_TWO_STEP, 0)
    for _ in range(total):
        ref.step(1)
    assert lat.steps_taken == total
    assert torch.equal(lat.state, ref.state)
    # the graph itself keeps the buffer
    replay.graph.replay()
    for _ in range(n):
        ref.step(1)
    assert torch.equal(lat.state, ref.state)


@pytest.mark.parametrize("sizes", [SMALL, LARGE])
@pytest.mark.parametrize("n", [8, 10])
@pytest.mark.parametrize("m", [2, 3, 4])
def test_batch_replays_mixed_with_steps(cuda, sizes, n, m):
    a, b = make(sizes, "f32", "periodic", cuda), make(sizes, "f32", "periodic", cuda)
    _, total = mixed(a, n, m)
    b.step(total, SINGLE)
    assert a.steps_taken == total
    assert torch.equal(a.state, b.state)


def test_state_loaded_between_replays(two_step, cuda):
    _lib.set_tuning(_lib.TUNE_TWO_STEP, 1)
    lat = PyLB.Lattice(256, 256, 1.4, u0=0.05, device=cuda)
    ref = PyLB.Lattice(256, 256, 1.4, u0=0.05, device=cuda)
    replay = lat.capture(2)  # one launch
    replay()
    f = ref.equilibrium(1.01, 0.0, 0.01).populations()
    lat.load(f)
    ref.load(f)
    replay()
    ref.step(2)
    assert torch.equal(lat.state, ref.state)


@pytest.mark.parametrize("sizes", [SMALL, LARGE])
@pytest.mark.parametrize("retired", [False, True])
def test_batch_in_a_graph_of_the_callers(cuda, sizes, retired):
    """After a warm-up of two steps any number of steps can be captured."""
    a, b = make(sizes, "f32", "periodic", cuda), make(sizes, "f32", "periodic", cuda)
    if retired:
        for x in (a, b):
            x.set_active(np.arange(len(sizes)) % 3 != 1)
    a.step(2)
    b.step(2, SINGLE)
    for n in (10, 3, 1, 8, 5):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            a.step(n)
        g.replay()
        b.step(n, SINGLE)
        torch.cuda.synchronize()
        for i in range(len(sizes)):
            assert torch.equal(a.populations(i), b.populations(i))


@pytest.mark.parametrize("sizes", [SMALL, LARGE])
def test_replay_keeps_its_lists(cuda, sizes):
    """A graph of some of the instances stays good when others become active."""
    a, b = make(sizes, "f32", "periodic", cuda), make(sizes, "f32", "periodic", cuda)
    some = np.arange(len(sizes)) % 3 != 1
    for x in (a, b):
        x.set_active(some)
    replay = a.capture(6)
    a.set_active(np.ones(len(sizes), dtype=bool))
    # what the allocator gives out next would lie where the lists were
    rubbish = [torch.full((n,), -1, dtype=torch.int32, device=cuda) for n in (64, 256, 1024, 4096, 16384) for _ in range(50)]
    replay()
    b.step(6, SINGLE)
    for i in range(len(sizes)):
        assert torch.equal(a.populations(i), b.populations(i)), i
    del rubbish
