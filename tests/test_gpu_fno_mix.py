"""The surrogate's complex mixing per Fourier mode and its gradients against
float64, with channel, sample and mode counts off the kernels' groups (4
channels a thread; 4 x 32 channels, 8 samples and 16 modes a block).

Tolerance: FP32 sums of K products are off by at most (K + 3) 2^-24 of the sum
of their magnitudes (each complex product is two, of sums of two); BF16 results
by 2^-9 more.
"""

import pytest
import torch

from latticeboltzmann_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,O,B,q,mk", [(32, 32, 16, 24, 12), (1, 1, 1, 2, 1), (5, 33, 3, 6, 17), (6, 30, 9, 8, 16),
                                        (9, 4, 8, 4, 33), (32, 64, 2, 24, 12)])
def test_mixing_and_gradients(cuda, C, O, B, q, mk):
    g = torch.Generator(device=cuda).manual_seed(C + O)
    P = torch.randn(C, B, 2 * mk, 2 * q, generator=g, device=cuda)
    D = torch.randn(O, B, 2 * q, 2 * mk, generator=g, device=cuda)
    Rr, Ri = (torch.randn(C, O, q, mk, generator=g, device=cuda).bfloat16() for _ in range(2))
    Ym = torch.empty(O, B, 2 * q, 2 * mk, device=cuda, dtype=torch.bfloat16)
    dP = torch.empty(C, B, 2 * mk, 2 * q, device=cuda, dtype=torch.bfloat16)
    dR = torch.full((2, C, O, q, mk), 7.0, device=cuda)
    s = torch.cuda.current_stream().cuda_stream
    _lib.call("lbgb_fno_mix", P.data_ptr(), Rr.data_ptr(), Ri.data_ptr(), Ym.data_ptr(), C, O, B, q, mk, s)
    _lib.call("lbgb_fno_mix_back", D.data_ptr(), P.data_ptr(), Rr.data_ptr(), Ri.data_ptr(), dP.data_ptr(),
              dR[0].data_ptr(), dR[1].data_ptr(), C, O, B, q, mk, s)
    p, d = P.double(), D.double()
    x = torch.complex(p[:, :, :mk, :q] + p[:, :, mk:, q:], p[:, :, mk:, :q] - p[:, :, :mk, q:]).transpose(2, 3)
    dy = torch.complex(d[:, :, :q, :mk] + d[:, :, q:, mk:], d[:, :, :q, mk:] - d[:, :, q:, :mk])
    R = torch.complex(Rr.double(), Ri.double())
    mag = lambda z: z.real.abs() + z.imag.abs() + 0j

    def near(got, eq, a, b, n, bf16):
        ref, size = torch.einsum(eq, a, b), torch.einsum(eq, mag(a), mag(b)).real
        for u, v in zip(got, (ref.real, ref.imag)):
            assert bool(((u.double() - v).abs() <= (2 * n + 6) * 2 ** -24 * size + (2 ** -8 * v.abs() if bf16 else 0)).all())

    y = Ym[:, :, :q]
    near((y[..., :mk], y[..., mk:]), "cbyk,coyk->obyk", x, R, C, True)
    assert torch.equal(Ym[:, :, q:, mk:], y[..., :mk]) and torch.equal(Ym[:, :, q:, :mk], -y[..., mk:])
    t = dP.transpose(2, 3)
    near((t[:, :, :q, :mk], t[:, :, :q, mk:]), "obyk,coyk->cbyk", dy, R.conj(), O, True)
    near((dR[0], dR[1]), "obyk,cbyk->coyk", dy, x.conj(), B, False)
