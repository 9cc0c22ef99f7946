"""Several fused steps of a small lattice per launch (k_tile) against single
steps: bit for bit, since each cell of every intermediate step is computed with
the single-step kernels' operations and stored in the storage's own codes.
Sizes: the smallest, whole rows and strips with a halo, one tile and many,
sides shorter than the halo, tiles that end inside a warp."""

import pytest
import torch

import latticeboltzmann_gb300 as PyLB
from latticeboltzmann_gb300 import _lib
from test_gpu_march import same, two_step  # noqa: F401

pytestmark = pytest.mark.gpu

SIZES = [(2, 2), (3, 2), (2, 9), (5, 7), (16, 128), (33, 17), (64, 250), (300, 200), (7, 3001), (3001, 7), (256, 256)]


@pytest.mark.parametrize("storage", ["f32", "f32dev", "f64", "f16dev", "bf16dev"])
@pytest.mark.parametrize("boundary", ["cavity", "cavity-ladd", "periodic"])
@pytest.mark.parametrize("size", SIZES)
def test_tile_equals_single_steps(two_step, cuda, storage, boundary, size):
    if storage == "f64" and size == (300, 200):
        size = (310, 211)
    same(*size, storage, boundary, (2, 21), cuda)


@pytest.mark.parametrize("storage", ["f16dev", "bf16dev"])
@pytest.mark.parametrize("boundary", ["cavity", "cavity-ladd", "periodic"])
@pytest.mark.parametrize("size", [(2, 9), (33, 17), (64, 250), (300, 200), (1200, 1001)])
def test_tile_stochastic_equals_single_steps(two_step, cuda, storage, boundary, size):
    same(*size, storage, boundary, (3, 13), cuda, "stochastic")


@pytest.mark.parametrize("storage,size", [("f32", (900, 1000)), ("f32", (1023, 1025)), ("f16dev", (1000, 1096))])
def test_tile_largest(two_step, cuda, storage, size):
    same(*size, storage, "cavity", (7,), cuda)


def test_tile_under_capture(two_step, cuda):
    _lib.set_tuning(_lib.TUNE_TWO_STEP, 1)
    for n in (2, 6, 10, 26):
        lat = PyLB.Lattice(60, 50, 1.2, u0=0.05, device=cuda)
        ref = PyLB.Lattice(60, 50, 1.2, u0=0.05, device=cuda)
        replay = lat.capture(n)
        replay()
        replay()
        ref.step(2 * n)
        assert torch.equal(lat.state, ref.state)


def test_tile_from_two_threads(two_step, cuda):
    """Plans are kept per host thread; two threads step different lattices on their own streams."""
    import threading
    _lib.set_tuning(_lib.TUNE_TWO_STEP, 1)
    got = {}

    def work(nx, ny):
        with torch.cuda.stream(torch.cuda.Stream(cuda)):
            lat = PyLB.Lattice(nx, ny, 1.5, u0=0.05, device=cuda)
            for _ in range(20):
                lat.step(9)
            torch.cuda.current_stream(cuda).synchronize()
            got[(nx, ny)] = lat.state.clone()

    ts = [threading.Thread(target=work, args=a) for a in ((90, 130), (130, 90))]
    [t.start() for t in ts]
    [t.join() for t in ts]
    for a in ((90, 130), (130, 90)):
        ref = PyLB.Lattice(*a, 1.5, u0=0.05, device=cuda)
        for _ in range(180):
            ref.step(1)
        assert torch.equal(ref.state, got[a])
