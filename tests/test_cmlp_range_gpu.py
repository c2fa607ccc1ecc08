"""Phases of millions of turns through the complex MLP: h = exp(i w z) with w z a float
of the test's own choice (zero weights, biases of that value, omega 1) against cos and
sin of that float in 64 bits.  The reduction by 2 pi = c1 - c2 leaves |w z| / 2 pi times
what the two floats miss of 2 pi and roundings of a unit, the special function unit
2^-21 on [-pi, pi], BF16 halves 2^-16 of each value."""
import cmath
import math

import pytest
import torch

from test_inr_gpu import pkg  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layer", [0, 2])
@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("phase", [3.0, 1.0e5, 2.5e7, 2.7e7, 3.1e7, 6.0e7])
def test_phase(pkg, layer, sign, phase):  # noqa: F811
    dev = torch.device("cuda")
    mlp = pkg.cmlp.ComplexMLP(32, 64, 2, 1, first_omega_0=1.0, hidden_omega_0=1.0).to(dev)
    ref = torch.arange(32, dtype=torch.float32)
    z = sign * (phase + ref * (4.0 if phase > 1e6 else 0.25))  # exact in float32
    with torch.no_grad():
        for l in list(mlp.net)[:3]:
            l.linear.weight.zero_()
            l.linear.bias.zero_()
        mlp.net[3].weight.zero_()
        mlp.net[3].bias.zero_()
        for unit in (0, 5, 31):
            mlp.net[3].weight.zero_()
            mlp.net[3].weight[0, unit] = 1.0
            if layer == 2:
                mlp.net[2].linear.bias.copy_(z.to(dev).to(torch.complex64))
                y = mlp.net(torch.zeros(3, 32, device=dev))
                want = complex(math.cos(float(z[unit])), math.sin(float(z[unit])))
            else:  # h2 = exp(i h1 / 4) and h3 = exp(i h2 / 4) of that unit
                mlp.net[0].linear.bias.copy_(z.to(dev))
                for l in (mlp.net[1], mlp.net[2]):
                    l.linear.weight.zero_()
                    l.linear.weight[unit, unit] = 0.25
                y = mlp.net(torch.zeros(3, 32, device=dev))
                h = complex(math.cos(float(z[unit])), math.sin(float(z[unit])))
                want = cmath.exp(0.25j * cmath.exp(0.25j * h))
            miss = abs(2 * math.pi - (6.28318548202514648 - 1.74845553e-7))
            tol = abs(phase) / (2 * math.pi) * miss + 2.0 ** -21 + 3 * 2.0 ** -16 + 2.0 ** -22 * math.pi
            got = y[:, 0].to(torch.complex128).cpu()
            assert float((got - want).abs().max()) <= tol
