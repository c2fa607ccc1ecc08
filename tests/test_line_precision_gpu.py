"""Intensities of probes whose side has a prime factor of 17 to 113, as close to 64 bits
as FP32 sums over pairs are.  A sum of h = p / 2 pairs of random phase gathers a
relative r.m.s. error of 2^-24 sqrt(p / 12) per axis (partial sums grow as sqrt(k),
each rounded by 2^-24 / sqrt(3) of itself at most), products, twiddles and the other
passes about 2^-24 sqrt(4); intensities carry the amplitude's relative error.  Allowed:
one and a half times that."""
import pytest
import torch

from conftest import load_pkg

pytestmark = pytest.mark.gpu
SIDES = [(34, 34), (68, 68), (92, 51), (119, 119), (145, 145), (148, 148), (161, 64), (221, 255), (282, 282), (284, 296),
         (67, 67), (113, 113), (226, 226), (109, 101), (306, 306), (340, 391)]


def _prime(n):
    p, d = 1, 2
    while n > 1:
        while n % d == 0:
            n, p = n // d, d
        d += 1
    return p


@pytest.mark.parametrize("M,N", SIDES)
def test_intensities(M, N):
    pkg = load_pkg()
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(M * N)
    O = torch.randn(M + 40, N + 40, dtype=torch.complex64, device=dev, generator=g)
    P = torch.randn(M, N, dtype=torch.complex64, device=dev, generator=g)
    tl = torch.randint(0, 41, (6, 2), device=dev, generator=g).to(torch.int32)
    got = pkg.forward_intensity(O, P, tl).double()
    O64, P64 = O.to(torch.complex128), P.to(torch.complex128)
    ref = torch.stack([torch.fft.fftshift(torch.fft.fft2(P64 * O64[y:y + M, x:x + N])).abs().square()
                       for y, x in tl.tolist()])
    err = float((got - ref).square().sum().sqrt() / ref.square().sum().sqrt())
    assert err <= 1.5 * 2.0 ** -24 * ((_prime(M) + _prime(N)) / 12 + 8) ** 0.5
