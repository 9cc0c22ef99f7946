"""Several fused steps per launch (k_march) against single steps.

Each cell of every intermediate step is computed with the single-step
kernel's operations and stored in the storage's own codes, so the populations
after any number of steps equal the single-step path's bit for bit.  Sizes:
one strip and several, strips that end inside a warp, within one vector of a
strip's edge and (4-byte codes) inside a vector, one row per chunk and many,
the smallest lattice of each number of steps per launch in both directions."""

import ctypes

import pytest
import torch

import latticeboltzmann_gb300 as PyLB
from latticeboltzmann_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.fixture
def two_step(cuda):
    saved = _lib.get_tuning(_lib.TUNE_TWO_STEP)
    yield
    _lib.set_tuning(_lib.TUNE_TWO_STEP, saved)


def run(nx, ny, storage, boundary, steps, several, rounding, cuda):
    _lib.set_tuning(_lib.TUNE_TWO_STEP, int(several))
    lat = PyLB.Lattice(nx, ny, 1.6, boundary=boundary, u0=0.09, storage=storage, rounding=rounding, seed=5,
                       device=cuda)
    g = torch.Generator(device=cuda).manual_seed(nx + ny)
    noise = [torch.randn(nx, ny, generator=g, dtype=torch.float64, device=cuda) for _ in range(3)]
    lat.equilibrium(1 + 0.02 * noise[0], 0.04 * noise[1], 0.04 * noise[2])
    for n in steps:
        lat.step(n)
    torch.cuda.synchronize()
    return lat.state, int(lat._step_ctr)


def same(nx, ny, storage, boundary, steps, cuda, rounding="nearest"):
    a, na = run(nx, ny, storage, boundary, steps, True, rounding, cuda)
    b, nb = run(nx, ny, storage, boundary, steps, False, rounding, cuda)
    assert na == nb
    assert torch.equal(a, b)


TWO = [(8, 125000), (62504, 16), (1000, 1000), (8180, 120), (7900, 124)]
FOUR = [(8, 187504), (93760, 16), (93751, 17), (8, 187501), (1230, 1240), (1237, 1283)]


@pytest.mark.parametrize("storage", ["f32", "f32dev"])
@pytest.mark.parametrize("boundary", ["cavity", "cavity-ladd", "periodic"])
@pytest.mark.parametrize("size,steps", [(s, (5,)) for s in TWO] + [(s, (4, 11)) for s in FOUR])
def test_march_4_byte_codes_equal_single_steps(two_step, cuda, storage, boundary, size, steps):
    same(*size, storage, boundary, steps, cuda)


@pytest.mark.parametrize("storage", ["f16dev", "bf16dev"])
@pytest.mark.parametrize("rounding", ["nearest", "stochastic"])
@pytest.mark.parametrize("boundary", ["cavity", "cavity-ladd", "periodic"])
@pytest.mark.parametrize("size,steps", [((8, 140000), (5,)), ((70000, 16), (5,)), ((4700, 240), (5,)),
                                        ((4500, 248), (5,)), ((8, 187504), (4, 11)), ((93760, 16), (11,)),
                                        ((1237, 1288), (4, 7))])
def test_march_16_bit_codes_equal_single_steps(two_step, cuda, storage, rounding, boundary, size, steps):
    same(*size, storage, boundary, steps, cuda, rounding)


def test_march_unaligned_buffers(two_step, cuda):
    """Buffers that start on 4 bytes only take the element-by-element form."""
    nx, ny = 1500, 1024
    out = []
    for off in (0, 1):
        for several in (1, 0):
            _lib.set_tuning(_lib.TUNE_TWO_STEP, several)
            store = [torch.zeros(9 * nx * ny + 4, device=cuda) for _ in range(2)]
            a, b = (s[off:off + 9 * nx * ny].view(9, nx, ny) for s in store)
            g = torch.Generator(device=cuda).manual_seed(1)
            a.copy_(0.1 + 0.01 * torch.rand(9, nx, ny, generator=g, device=cuda))
            which = ctypes.c_int(-1)
            _lib.call("lbgb_run_fused", a.data_ptr(), b.data_ptr(), nx, ny, _lib.CAVITY, 1.3, 0.05, _lib.F32, 6,
                      ctypes.byref(which), torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
            out.append((a, b)[which.value].clone())
            assert float(store[0][:off].abs().sum() + store[0][off + 9 * nx * ny:].abs().sum()) == 0.0
            assert float(store[1][:off].abs().sum() + store[1][off + 9 * nx * ny:].abs().sum()) == 0.0
    assert all(torch.equal(out[0], o) for o in out[1:])


def test_march_under_capture_and_max_steps(two_step, cuda):
    _lib.set_tuning(_lib.TUNE_TWO_STEP, 1)
    code = _lib.load().lbgb_max_steps_per_launch
    assert code(4096, 4096, _lib.CAVITY, _lib.F32) == 4
    assert code(1024, 1032, _lib.CAVITY, _lib.F32) == 2
    assert code(4096, 4096, _lib.CAVITY, _lib.F64) == 1
    assert code(1, 1, _lib.PERIODIC, _lib.F32) == 1
    lat = PyLB.Lattice(1024, 1000, 1.2, u0=0.05, device=cuda)
    ref = PyLB.Lattice(1024, 1000, 1.2, u0=0.05, device=cuda)
    replay = lat.capture(6)
    replay()
    replay()
    ref.step(12)
    assert torch.equal(lat.state, ref.state)
