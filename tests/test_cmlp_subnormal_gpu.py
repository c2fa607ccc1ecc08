"""Amplitudes exp(-beta) below the normal range of FP32 pass through the complex MLP.
Zero weights and a last bias of i beta make every unit of the third layer exp(-beta);
output weights of 2^120 bring them back: y = 32 * 2^120 * exp(-beta).  bf16(h) +
bf16(h - bf16(h)) leaves at most half a unit of BF16's smallest values, 2^-134, per
unit, and the exponential some 2^-20."""
import math

import pytest
import torch

from test_inr_gpu import pkg  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beta", [86.0, 88.0, 89.5, 91.0])
def test_amplitudes_below_the_normal_range(pkg, beta):  # noqa: F811
    dev = torch.device("cuda")
    mlp = pkg.cmlp.ComplexMLP(32, 64, 2, 1, first_omega_0=1.0, hidden_omega_0=1.0).to(dev)
    with torch.no_grad():
        for layer in list(mlp.net)[:3]:
            layer.linear.weight.zero_()
            layer.linear.bias.zero_()
        mlp.net[2].linear.bias.fill_(1j * beta)
        mlp.net[3].weight.fill_(2.0 ** 120)
        mlp.net[3].bias.zero_()
        y = mlp.net(torch.zeros(200, 32, device=dev))
    h = math.exp(-beta)
    assert (h < 2.0 ** -126) == (beta > 87.5)
    want = 32 * 2.0 ** 120 * h
    assert bool((y.imag.abs() <= 1e-3 * want).all())
    assert bool(((y.real.double() - want).abs() <= want * (2.0 ** -134 / h + 2.0 ** -16)).all())
