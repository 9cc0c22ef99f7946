"""The surrogate's fused layer kernels against float64 products of the same BF16
operands, at the edges of their tiles (128 pixels of a row, 16 and 64 input
channels or modes a block, 16 channels a warp), and the fused network against
the one that runs one pass per operation.

Tolerances.  An FP32 sum of K products is off by at most K 2^-24 sum|x w|; the
sums here have K <= 192, so 2e-5 sum|x w| (doubled by the bias and the
accumulator's own rounding).  tanh.approx is off by 2^-10.99 relative, which
moves gelu(x) and gelu'(x) by at most 2^-11 |x| (1 + x^2) and BF16 rounding by
2^-9 of the value.  Sums over the pixels are held to the separate kernel's bits.
"""

import numpy as np
import pytest
import torch

from latticeboltzmann_gb300 import _lib
from latticeboltzmann_gb300 import fno as F

pytestmark = pytest.mark.gpu

# n, k1, rows, W, k2
SIZES = [(16, 1, 1, 8, 0), (32, 4, 1, 1000, 0), (32, 32, 3, 128, 24), (16, 17, 5, 136, 8), (32, 128, 1, 4096, 0),
         (16, 65, 2, 264, 64), (32, 32, 700, 120, 40), (32, 64, 4, 40, 24),
         (32, 32, 64, 256, 24), (16, 32, 96, 512, 16), (32, 20, 1, 512 * 75, 0)]


def gelu(x):
    return 0.5 * x * (1 + torch.tanh(0.7978845608028654 * (x + 0.044715 * x ** 3)))


def gelu_d(x):
    t = torch.tanh(0.7978845608028654 * (x + 0.044715 * x ** 3))
    return 0.5 * (1 + t) + 0.5 * x * (1 - t * t) * 0.7978845608028654 * (1 + 3 * 0.044715 * x * x)


def near(got, ref, tol):
    assert bool(((got.double() - ref).abs() <= tol).all()), float(((got.double() - ref).abs() - tol).max())


def operands(cuda, n, k1, rows, W, k2):
    g = torch.Generator(device=cuda).manual_seed(n + k1 + W)
    r = lambda *s: torch.randn(*s, generator=g, device=cuda).bfloat16()
    x, b1, bias = r(k1, rows * W), r(n, k1) * k1 ** -0.5, r(n).float()
    a2, b2 = r(max(k2, 1), W), r(n, rows, max(k2, 1)) * 0.1
    D = b1.double() @ x.double()
    S = b1.double().abs() @ x.double().abs()
    if k2:
        D = D + (b2.double() @ a2.double()).view(n, rows * W)
        S = S + (b2.double().abs() @ a2.double().abs()).view(n, rows * W)
    return x, b1, bias, a2, b2, D, 4e-5 * (S + 1)


@pytest.mark.parametrize("n,k1,rows,W,k2", SIZES)
def test_layer_and_its_gradient(cuda, n, k1, rows, W, k2):
    x, b1, bias, a2, b2, D, tol = operands(cuda, n, k1, rows, W, k2)
    N = rows * W
    s = torch.cuda.current_stream().cuda_stream
    z, v = torch.full((n, N), 7.0, device=cuda), torch.zeros(n, N, device=cuda, dtype=torch.bfloat16)
    second = (k2, a2.data_ptr(), b2.data_ptr()) if k2 else (0, None, None)
    _lib.call("lbgb_fno_layer", n, k1, rows, W, x.data_ptr(), b1.data_ptr(), k1, 1, *second, bias.data_ptr(), 1,
              z.data_ptr(), v.data_ptr(), s)
    ref = D + bias.double()[:, None]
    near(z, ref, tol)
    near(v, gelu(z.double()), 2 ** -8 * gelu(z.double()).abs() + 2 ** -11 * z.double().abs() * (1 + z.double() ** 2))
    _lib.call("lbgb_fno_layer", n, k1, rows, W, x.data_ptr(), b1.data_ptr(), k1, 1, *second, None, 0, None,
              v.data_ptr(), s)
    near(v, D, 2 ** -8 * D.abs() + tol)

    bt = b1.t().contiguous()  # (k1, n): the strides of the transposed product
    parts = torch.empty(_lib.load().lbgb_fno_layer_parts(n), device=cuda)
    f32 = torch.empty(n, N, device=cuda)
    ordered = _lib.load().lbgb_fno_layer_sums(rows, W, k2)
    for zz in (z, None):
        sums = [torch.empty(n, device=cuda) for _ in range(3)]
        back = ("lbgb_fno_layer_back", n, k1, rows, W, x.data_ptr(), bt.data_ptr(), 1, n, *second,
                zz.data_ptr() if zz is not None else None, v.data_ptr())
        _lib.call(*back, f32.data_ptr(), sums[0].data_ptr(), parts.data_ptr(), s)
        d = gelu_d(z.double()) if zz is not None else torch.ones_like(D)
        e = 2 ** -11 * (1 + z.double().abs() ** 3) if zz is not None else 0 * D
        near(f32, D * d, D.abs() * e + 2 * tol)
        assert torch.equal(v, f32.bfloat16())
        _lib.call("lbgb_fno_row_sum", f32.data_ptr(), sums[1].data_ptr(), parts.data_ptr(), n, N, s)
        assert torch.equal(sums[0], sums[1])
        if ordered:  # the same additions without the FP32 values in memory
            v.zero_()
            _lib.call(*back, None, sums[2].data_ptr(), parts.data_ptr(), s)
            assert torch.equal(sums[2], sums[1]) and torch.equal(v, f32.bfloat16())
        else:
            with pytest.raises(ValueError):
                _lib.call(*back, None, sums[2].data_ptr(), parts.data_ptr(), s)
    _lib.gemm_status()


@pytest.mark.parametrize("hidden,k1,N,cout", [(128, 32, 1000, 3), (16, 1, 8, 1), (48, 20, 128, 4), (112, 128, 136, 2),
                                              (128, 32, 128 * 700, 3)])
def test_projection_and_its_gradient(cuda, hidden, k1, N, cout):
    x, q1, q1b, _, _, D, tol = operands(cuda, hidden, k1, 1, N, 0)
    g = torch.Generator(device=cuda).manual_seed(N)
    q2 = (torch.randn(cout, hidden, generator=g, device=cuda) / 8).bfloat16()
    q2b = torch.randn(cout, generator=g, device=cuda)
    d = torch.randn(cout, N, generator=g, device=cuda).bfloat16()
    s = torch.cuda.current_stream().cuda_stream
    gb, out, out2 = torch.zeros(hidden, N, device=cuda, dtype=torch.bfloat16), *torch.zeros(2, cout, N, device=cuda)
    args = (hidden, k1, 1, N, x.data_ptr(), q1.data_ptr(), q1b.data_ptr(), cout, q2.data_ptr())
    _lib.call("lbgb_fno_project", *args, q2b.data_ptr(), gb.data_ptr(), out.data_ptr(), s)
    _lib.call("lbgb_fno_project", *args, q2b.data_ptr(), None, out2.data_ptr(), s)
    assert torch.equal(out, out2)
    h = D + q1b.double()[:, None]
    act = 2 ** -11 * (1 + h.abs() ** 3)
    near(gb, gelu(h), 2 ** -8 * gelu(h).abs() + act + 2 * tol)
    near(out, q2.double() @ gb.double() + q2b.double()[:, None], 4e-5 * (q2.double().abs() @ gb.double().abs() + 4))
    dh, f32 = torch.zeros_like(gb), torch.empty(hidden, N, device=cuda)
    sums = [torch.empty(hidden, device=cuda) for _ in range(3)]
    parts = torch.empty(_lib.load().lbgb_fno_layer_parts(hidden), device=cuda)
    _lib.call("lbgb_fno_project_back", *args, d.data_ptr(), dh.data_ptr(), f32.data_ptr(), sums[0].data_ptr(),
              parts.data_ptr(), s)
    dg = q2.double().t() @ d.double()
    ref = dg * gelu_d(h)
    near(f32, ref, dg.abs() * (act + 2 * tol) + 1e-5)
    assert torch.equal(dh, f32.bfloat16())
    _lib.call("lbgb_fno_row_sum", f32.data_ptr(), sums[1].data_ptr(), parts.data_ptr(), hidden, N, s)
    assert torch.equal(sums[0], sums[1])
    if _lib.load().lbgb_fno_layer_sums(1, N, 0):
        dh.zero_()
        _lib.call("lbgb_fno_project_back", *args, d.data_ptr(), dh.data_ptr(), None, sums[2].data_ptr(),
                  parts.data_ptr(), s)
        assert torch.equal(sums[2], sums[1]) and torch.equal(dh, f32.bfloat16())
    _lib.gemm_status()


@pytest.mark.parametrize("B,H,W", [(2, 40, 32), (1, 64, 72), (3, 48, 128), (2, 96, 136), (2, 64, 128)])
def test_fused_network_equals_separate_passes(cuda, B, H, W):
    g = torch.Generator(device=cuda).manual_seed(H)
    a, t = (torch.randn(c, B, H, W, generator=g, device=cuda) for c in (4, 3))
    net = F.FNO2d(device=cuda, seed=H)
    got = []
    for fused in (False, True):
        net.fused_epilogue = fused
        assert net._fused(B, H, W) == fused
        loss = float(net.loss_and_backward(a, t))
        got.append((loss, net.grads(), net.forward(a).double().cpu().numpy()))
    # the same values are rounded to BF16 and the same sums taken, bit for bit
    rel = lambda x, y: np.linalg.norm(x - y) / np.linalg.norm(y)
    assert rel(got[1][2], got[0][2]) < 1e-6  # the output's last product is FP32 sums of 128
    assert got[1][0] == got[0][0]
    for name, ref in got[0][1].items():
        assert np.array_equal(got[1][1][name], ref), name


@pytest.mark.parametrize("n,k1,rows,W,k2", [(33, 4, 1, 64, 0), (24, 4, 1, 64, 0), (32, 129, 1, 64, 0), (32, 4, 1, 12, 0),
                                            (32, 4, 2, 64, 65), (32, 4, 2, 64, 12)])
def test_refused_sizes(cuda, n, k1, rows, W, k2):
    x = torch.zeros(1 << 16, device=cuda, dtype=torch.bfloat16)
    p = x.data_ptr()
    with pytest.raises((ValueError, _lib.LBGBError)):
        _lib.call("lbgb_fno_layer", n, k1, rows, W, p, p, 1, 1, k2, p, p, None, 0, None, p, 0)
