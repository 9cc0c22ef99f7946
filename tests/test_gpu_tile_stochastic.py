"""Stochastic rounding in k_tile against the pipelined single-step kernel that it
stands in for: half and bfloat16 rows of whole vectors from 65,536 cells to the
1.1 M where the march begins, several launches of several steps, other seeds."""

import pytest
import torch

import latticeboltzmann_gb300 as PyLB
from latticeboltzmann_gb300 import _lib
from test_gpu_march import two_step  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["f16dev", "bf16dev"])
@pytest.mark.parametrize("boundary", ["cavity", "cavity-ladd", "periodic"])
@pytest.mark.parametrize("size,seed", [((256, 256), 1), ((512, 520), 77), ((1000, 1096), 2 ** 31 + 5)])
def test_tile_equals_the_pipelined_kernel(two_step, cuda, storage, boundary, size, seed):
    def run(several):
        _lib.set_tuning(_lib.TUNE_TWO_STEP, several)
        lat = PyLB.Lattice(*size, 1.6, boundary=boundary, u0=0.09, storage=storage, rounding="stochastic", seed=seed,
                           device=cuda)
        g = torch.Generator(device=cuda).manual_seed(size[0])
        r = [torch.randn(*size, generator=g, dtype=torch.float64, device=cuda) for _ in range(3)]
        lat.equilibrium(1 + 0.02 * r[0], 0.04 * r[1], 0.04 * r[2])
        for n in (5, 1, 17):
            lat.step(n)
        return lat
    code, bc = _lib.STORAGE_CODES[storage], _lib.BOUNDARY_CODES[boundary]
    assert size[0] * size[1] >= _lib.get_tuning(_lib.TUNE_PIPE_MIN_CELLS) and size[1] % 8 == 0
    _lib.set_tuning(_lib.TUNE_TWO_STEP, 1)
    assert _lib.load().lbgb_max_steps_per_launch(*size, bc, code) > 1
    a, b = run(1), run(0)
    assert torch.equal(a.state, b.state) and int(a._step_ctr) == int(b._step_ctr) == 23
