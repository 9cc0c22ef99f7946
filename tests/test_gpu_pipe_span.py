"""FP64 tiles of the pipelined step kernel span rows: 15 segments of 64 cells each.

The rows here have one segment (many rows a tile), one less, as many and one
more than a tile's, and a remainder; with a part of the rows as well.  The
register kernel works cell by cell with the same arithmetic: equal bit for bit.
"""

import numpy as np
import pytest
import torch

import latticeboltzmann_gb300 as PyLB
from latticeboltzmann_gb300 import _lib

pytestmark = pytest.mark.gpu

SEG = 64


@pytest.fixture
def kernel(cuda):
    saved = _lib.get_tuning(_lib.TUNE_KERNEL)
    yield lambda name: _lib.set_tuning(_lib.TUNE_KERNEL, _lib.KERNELS[name])
    _lib.set_tuning(_lib.TUNE_KERNEL, saved)


@pytest.mark.parametrize("boundary", ["cavity", "cavity-ladd", "periodic"])
@pytest.mark.parametrize("nx,ny", [(47, 2), (31, SEG - 2), (46, SEG), (29, SEG + 2), (11, 14 * SEG), (7, 15 * SEG),
                                   (13, 16 * SEG), (8, 15 * SEG + 2), (5, 31 * SEG - 2), (700, 7 * SEG)])
def test_spanning_tiles_equal_register_kernel(kernel, cuda, boundary, nx, ny):
    f0 = torch.from_numpy(np.random.default_rng(nx + ny).random((9, nx, ny))) / 9
    out = []
    for name in ("register", "pipelined"):
        kernel(name)
        lat = PyLB.Lattice(nx, ny, 1.3, boundary=boundary, u0=0.05, storage="f64", device=cuda)
        lat.load(f0)
        lat.step(2)
        out.append(lat.state.clone())
    _lib.device_status()
    assert torch.equal(*out)
