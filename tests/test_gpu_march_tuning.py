"""Several steps per launch equal single steps also where LBGB_TUNE_PIPE_MIN_CELLS
hands large lattices to the register kernel, which rounds half precision's
wall-density-1 lid once instead of twice."""

import pytest

from latticeboltzmann_gb300 import _lib
from test_gpu_march import same, two_step  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["f16dev", "bf16dev", "f32"])
@pytest.mark.parametrize("size", [(512, 520), (1237, 1288)])
def test_register_kernel_for_large_lattices(two_step, cuda, storage, size):
    saved = _lib.get_tuning(_lib.TUNE_PIPE_MIN_CELLS)
    try:
        _lib.set_tuning(_lib.TUNE_PIPE_MIN_CELLS, 1 << 40)
        same(*size, storage, "cavity-ladd", (4, 7), cuda)
    finally:
        _lib.set_tuning(_lib.TUNE_PIPE_MIN_CELLS, saved)
