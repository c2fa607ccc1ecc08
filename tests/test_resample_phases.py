"""The phase form of the Fourier upsampling: y[s m + p] is the inverse length-n
transform of X_k exp(2 pi i (k + d) p / N), k the signed frequency.

CPU: the identity itself against the padded form (the FP64 oracle), even and odd
lengths and every scale.  GPU: the kernels that use it at the edges of their
range; FP32 transforms of up to 2048 points, tolerance of test_resample_gpu.py."""
import numpy as np
import pytest
import torch

from conftest import load_pkg
from oracle.inr import fourier_upsample, fourier_upsample_adjoint

TOL = 2e-6


def by_phases(x, s):
    """One axis (the last) of the upsampling, phase by phase."""
    n = x.shape[-1]
    N = n * s
    d = n // 2 + (N - n) // 2 - N // 2  # the band's offset: -1 for odd n and even N
    k = np.fft.fftfreq(n, 1.0 / n)
    k = np.where(k >= (n + 1) // 2, k - n, k)
    X = np.fft.fft(x, axis=-1)
    y = np.empty(x.shape[:-1] + (N,), complex)
    for p in range(s):
        m = np.arange(n)
        y[..., p::s] = np.fft.ifft(X * np.exp(2j * np.pi * k * p / N), axis=-1) * np.exp(2j * np.pi * d * (s * m + p) / N)
    return y


@pytest.mark.parametrize("h,w", [(8, 8), (7, 12), (9, 5), (1, 6), (2, 3), (30, 49)])
@pytest.mark.parametrize("s", [1, 2, 3, 4, 5])
def test_identity(h, w, s):
    rng = np.random.default_rng(h * w + s)
    x = rng.standard_normal((h, w)) + 1j * rng.standard_normal((h, w))
    y = by_phases(by_phases(x, s).T, s).T
    assert np.abs(y - fourier_upsample(x, s)).max() <= 1e-12 * np.abs(y).max()


@pytest.mark.gpu
@pytest.mark.parametrize("h,w,s", [(256, 256, 2), (256, 512, 4), (512, 256, 4), (1024, 1024, 2), (1024, 256, 4),
                                   (2048, 512, 2), (256, 100, 2), (512, 37, 2), (2048, 5, 2), (5, 2048, 2),
                                   (1, 256, 2), (256, 1, 4), (64, 1024, 4), (300, 512, 2)])
@pytest.mark.parametrize("shift", [0, 1])
def test_kernels(h, w, s, shift):
    """shift: the long side starts 8 bytes off a 16-byte boundary (C ABI callers)."""
    pkg = load_pkg()
    dev = torch.device("cuda")
    L, st = pkg.lib(), torch.cuda.current_stream().cuda_stream
    rng = np.random.default_rng(h + w + s)
    x = (rng.standard_normal((h, w)) + 1j * rng.standard_normal((h, w))).astype(np.complex64)
    g = (rng.standard_normal((h * s, w * s)) + 1j * rng.standard_normal((h * s, w * s))).astype(np.complex64)
    place = lambda a: torch.cat([torch.zeros(shift, dtype=torch.complex64), torch.from_numpy(a).reshape(-1)]).to(dev)  # noqa: E731
    xt, gt = place(x), place(g)
    y, gx = torch.zeros_like(gt), torch.zeros_like(xt)
    n = int(L.ptycho_fourier_upsample_workspace_size(h, w, s))
    ws = torch.empty(n, dtype=torch.uint8, device=dev)
    off = 8 * shift
    pkg._lib.check(L.ptycho_fourier_upsample(xt.data_ptr() + off, h, w, s, y.data_ptr() + off, ws.data_ptr(), n, st), "up")
    pkg._lib.check(L.ptycho_fourier_upsample_adjoint(gt.data_ptr() + off, h, w, s, gx.data_ptr() + off, ws.data_ptr(), n,
                                                     st), "adjoint")
    ref = fourier_upsample(x.astype(np.complex128), s)
    ref_g = fourier_upsample_adjoint(g.astype(np.complex128), s, (h, w))
    got, got_g = y[shift:].reshape(h * s, w * s).cpu().numpy(), gx[shift:].reshape(h, w).cpu().numpy()
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()
    assert np.abs(got_g - ref_g).max() <= TOL * np.abs(ref_g).max()
    if shift:
        assert y[0] == 0 and gx[0] == 0
