"""Gradients belong to the last training forward, whatever is changed between it
and backward: the parameters, or how the layers run.  Reference: the network
that runs one pass per operation and keeps the hidden layer's values, whose
gradients the fused one equals bit for bit."""

import pytest
import torch

from latticeboltzmann_gb300 import fno as F

pytestmark = pytest.mark.gpu


def net_and_inputs(cuda, fused):
    net = F.FNO2d(width=32, modes=12, layers=2, hidden=128, device=cuda, seed=3)
    net.fused_epilogue = fused
    g = torch.Generator(device=cuda).manual_seed(1)
    a = torch.randn(4, 2, 64, 128, generator=g, device=cuda)
    d = torch.randn(3, 2 * 64 * 128, generator=g, device=cuda)
    assert net._fused(2, 64, 128) == fused
    return net, a, d


def grads(net):
    return net.grad.clone()


def test_parameters_changed_before_backward(cuda):
    out = []
    for fused in (True, False):
        net, a, d = net_and_inputs(cuda, fused)
        net.forward(a, train=True)
        g = torch.Generator(device=cuda).manual_seed(2)
        net.flat.add_(0.05 * torch.randn(net.numel, generator=g, device=cuda))
        net._refresh_bf16()
        net.backward(d)
        out.append(grads(net))
    assert torch.equal(*out)


@pytest.mark.parametrize("first", [True, False])
def test_form_switched_before_backward(cuda, first):
    net, a, d = net_and_inputs(cuda, first)
    net.forward(a, train=True)
    net.backward(d)
    before = grads(net)
    net.forward(a, train=True)
    net.grad.zero_()
    net.fused_epilogue = not first
    net.backward(d)
    assert torch.equal(grads(net), before)
    net.forward(a)  # of the other form, without gradients
    net.grad.zero_()
    net.backward(d)
    assert torch.equal(grads(net), before)


def test_backward_needs_a_training_forward(cuda):
    net, a, d = net_and_inputs(cuda, True)
    net.forward(a)
    with pytest.raises(KeyError):
        net.backward(d)
