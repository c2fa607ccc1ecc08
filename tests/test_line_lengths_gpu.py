"""DFTs of any line length inside the general probe path: every pass radix, lengths
of one to four passes, Bluestein's convolution (a prime factor above 13) and the
direct sums that replace it when its tables do not fit (primes above about 2500).

Intensities, loss and gradients against torch's complex128 transforms of the same
FP32 inputs.  FP32 transforms of up to 4096 points: 1e-5 of the largest intensity,
2e-5 on the loss and 2e-4 of the largest gradient entry (the bounds of
test_general_probe_gpu.py)."""
import pytest
import torch

from conftest import load_pkg

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (1, 7), (2, 3), (4, 5), (6, 8), (9, 10), (11, 13), (12, 15), (16, 17), (33, 49), (121, 60),
          (169, 30), (83, 2), (127, 131), (255, 100), (251, 317), (320, 18), (1500, 3), (5, 2187), (1021, 2),
          (2, 1999), (2503, 2), (2, 4093), (4096, 1)]


def _problem(M, N, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.complex(torch.randn(s, generator=g, device="cuda"), torch.randn(s, generator=g, device="cuda"))  # noqa: E731
    O, P = r(M + 9, N + 7), r(M, N) / (M * N) ** 0.5
    tl = torch.tensor([[0, 0], [9, 7], [3, 5], [4, 1], [9, 0]], dtype=torch.int32, device="cuda")
    Im = 4.0 * torch.rand(5, M, N, generator=g, device="cuda")
    return O, P, tl, Im


def _exact(O, P, tl, Im, loss):
    O, P = O.to(torch.complex128).requires_grad_(), P.to(torch.complex128).requires_grad_()
    M, N = P.shape
    I = torch.stack([torch.fft.fftshift(torch.fft.fft2(P * O[y:y + M, x:x + N])).abs().square() for y, x in tl.tolist()])
    m = Im.double()
    if loss == "smooth_L1_loss":
        per = torch.nn.functional.smooth_l1_loss(I, m, reduction="none")
    else:
        d = torch.sqrt(m + 1e-8) - torch.sqrt(I + 1e-8)
        rx, ry = torch.roll(d, -1, -1) - d, torch.roll(d, -1, -2) - d
        per = torch.sqrt(rx * rx + ry * ry + 1e-8)
    total = per.mean(dim=(-2, -1)).sum()
    return I.detach(), total.detach(), *torch.autograd.grad(total, (O, P))


def _rel(a, b):
    return float((a - b).abs().max() / b.abs().max())


@pytest.mark.parametrize("M,N", SHAPES)
def test_any_length(M, N):
    pkg = load_pkg()
    O, P, tl, Im = _problem(M, N, 31 * M + N)
    loss = "FD_loss" if (M + N) % 3 == 0 and min(M, N) > 1 else "smooth_L1_loss"
    I, total, dO, dP = _exact(O, P, tl, Im, loss)
    assert _rel(pkg.forward_intensity(O, P, tl).double(), I) <= 1e-5
    got = pkg.fwd_adj_raw(O, P, tl, Im, pkg.LOSS_CODES[loss])
    only = pkg.fwd_adj_raw(O, P, tl, Im, pkg.LOSS_CODES[loss], want_grad=False)
    assert abs(float(got[0] - total)) <= 2e-5 * float(total) and torch.equal(got[0], only[0])
    tol = 1e-3 if loss == "FD_loss" else 2e-4
    assert _rel(got[2], dO) <= tol and _rel(got[3], dP) <= tol
    again = pkg.fwd_adj_raw(O, P, tl, Im, pkg.LOSS_CODES[loss])
    assert all(torch.equal(a, b) for a, b in zip(got[2:], again[2:]))
