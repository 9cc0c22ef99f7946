"""The FP64 collision and fields on the GPU (with the GPU's own reciprocal)
against extended precision on the host: no larger error than the FP64
evaluation of the same nodes, at most and in the root mean square of every
population, in the register, pipelined and tiled kernels."""

import numpy as np
import pytest
import torch

import latticeboltzmann_gb300 as PyLB
from test_fix64_host import states
from test_fix64_precision_host import CX, CY, evaluate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(64, 62), (256, 258)])
@pytest.mark.parametrize("u,noise", [(0.01, 1e-3), (0.16, 0.01)])
@pytest.mark.parametrize("omega", [0.25, 0.7, 1.0, 1.9])
def test_step_against_extended_precision(cuda, size, u, noise, omega):
    f = np.ascontiguousarray(states(size[0] * size[1], u, noise, 3).T).reshape(9, *size)
    lat = PyLB.Lattice(*size, omega, boundary="periodic", storage="f64", device=cuda)
    lat.load(torch.from_numpy(f)).step(1)
    got = lat.populations().cpu().numpy().reshape(9, -1).T
    pulled = np.stack([np.roll(f[i], (CX[i], CY[i]), (0, 1)) for i in range(9)]).reshape(9, -1).T
    exact = evaluate(pulled, omega, np.longdouble)
    here = np.abs((got - exact).astype(np.float64))
    fp64 = np.abs((evaluate(pulled, omega, np.float64) - exact).astype(np.float64))
    assert here.max() <= fp64.max()
    assert (np.sqrt((here ** 2).mean(0)) <= np.sqrt((fp64 ** 2).mean(0))).all()
    # several steps per launch do the same arithmetic
    two = PyLB.Lattice(*size, omega, boundary="periodic", storage="f64", device=cuda).load(torch.from_numpy(f))
    one = PyLB.Lattice(*size, omega, boundary="periodic", storage="f64", device=cuda).load(torch.from_numpy(f))
    assert torch.equal(two.step(2).state, one.step(1).step(1).state)


@pytest.mark.parametrize("u,noise", [(1e-6, 0.0), (0.01, 1e-3), (0.16, 0.01)])
def test_velocity_against_extended_precision(cuda, u, noise):
    f = np.ascontiguousarray(states(300 * 200, u, noise, 5).T)
    lat = PyLB.Lattice(300, 200, 1.0, boundary="periodic", storage="f64", device=cuda)
    _, ux, uy = lat.load(torch.from_numpy(f.reshape(9, 300, 200))).macroscopic()
    w = f.astype(np.longdouble)
    r, d = w.sum(0), f[0].copy()
    for c in range(1, 9):
        d += f[c]
    for got, c in ((ux, CX), (uy, CY)):
        exact = (w * c[:, None]).sum(0) / r
        j = np.zeros_like(d)
        for i in (1, 2, 3, 4, 5, 6, 7, 8):
            j += c[i] * f[i]
        here = np.abs((got.cpu().numpy().ravel() - exact).astype(np.float64))
        fp64 = np.abs((j / d - exact).astype(np.float64))
        assert here.max() <= fp64.max()
