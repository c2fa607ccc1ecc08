"""One NaN or infinity in the input of the Fourier upsampling, or of its adjoint,
reaches every output, as through the FFTs it stands for: each route (power-of-two
lines, lines of any length with and without Bluestein's convolution, the half-bin turn
of odd lengths, more than two phases, scale 1), samples of phase 0 and of the others,
the first and the last of a line.  A finite call on the same shapes stays finite."""
import pytest
import torch

from conftest import load_pkg

pytestmark = pytest.mark.gpu


def _up(x, s):
    h, w = x.shape
    F = torch.fft.fftshift(torch.fft.fft2(x))
    ph, pw = (h * s - h) // 2, (w * s - w) // 2
    F = torch.nn.functional.pad(F, (pw, w * s - w - pw, ph, h * s - h - ph))
    return torch.fft.ifft2(torch.fft.ifftshift(F)) * s ** 2


def _none_finite(z):
    return not bool((torch.isfinite(z.real) & torch.isfinite(z.imag)).any())


@pytest.mark.parametrize("val", [float("nan"), float("inf"), float("-inf")])
@pytest.mark.parametrize("h,w,s", [(256, 512, 2), (256, 300, 4), (1024, 256, 2), (45, 60, 2), (45, 60, 3), (64, 64, 4),
                                   (67, 35, 2), (249, 7, 2), (5, 1, 3), (30, 30, 1), (1, 1, 2)])
def test_reaches_every_output(h, w, s, val):
    pkg = load_pkg()
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(h * w + s)
    draw = lambda *n: torch.randn(n, dtype=torch.complex64, device=dev, generator=g)  # noqa: E731
    x0, g0 = draw(h, w), draw(h * s, w * s)
    x = x0.clone().requires_grad_()
    y = pkg.resample.fourier_upsample(x, s)
    gx, = torch.autograd.grad(y, x, g0, retain_graph=True)
    assert bool(torch.isfinite(torch.view_as_real(y.detach())).all() and torch.isfinite(torch.view_as_real(gx)).all())
    for part in (0, 1):
        for pos in {(0, 0), (h // 2, w // 3), (h - 1, w - 1)}:
            bad = x0.clone()
            torch.view_as_real(bad)[pos][part] = val
            assert _none_finite(_up(bad, s))
            assert _none_finite(pkg.resample.fourier_upsample(bad, s))
        for pos in {(0, 0), (s * (h // 2), s * (w - 1)), (0, s * w - 1), (s * h - 1, s * (w // 2)),
                    (s * h - 1, s * w - 1), (min(2, s * h - 1), min(1, s * w - 1))}:
            bad = g0.clone()
            torch.view_as_real(bad)[pos][part] = val
            got, = torch.autograd.grad(y, x, bad, retain_graph=True)
            leaf = x0.cpu().requires_grad_()
            want, = torch.autograd.grad(_up(leaf, s), leaf, bad.cpu())
            assert _none_finite(want) and _none_finite(got)
