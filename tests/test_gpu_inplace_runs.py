"""The in-place streams with runs of one, two and four tiles (the run length
follows from the lattice's size) against the out-of-place kernels: bit for bit."""

import pytest
import torch

import latticeboltzmann_gb300 as PyLB
from latticeboltzmann_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("nx,ny", [(40, 512), (704, 600), (1200, 256), (2432, 1024), (2432, 520), (608, 2060), (17, 4100)])
def test_runs_equal_out_of_place(cuda, dtype, nx, ny):
    f = torch.rand(9, nx, ny, device=cuda, dtype=dtype, generator=torch.Generator(device=cuda).manual_seed(nx))
    code = _lib.F32 if dtype == torch.float32 else _lib.F64
    s = torch.cuda.current_stream().cuda_stream
    ref, walls = torch.empty_like(f), torch.empty_like(f)
    _lib.call("lbgb_stream_periodic", f.data_ptr(), ref.data_ptr(), nx, ny, code, s)
    _lib.call("lbgb_stream_bounce_back", f.data_ptr(), walls.data_ptr(), nx, ny, 0.07, code, s)
    g = f.clone()
    PyLB.stream(g)
    assert torch.equal(g, ref)
    PyLB.Streaming.stream_and_bounce_back(f, 0.07)
    assert torch.equal(f, walls)
    _lib.device_status()
