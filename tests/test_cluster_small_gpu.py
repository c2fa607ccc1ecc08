"""The cluster kernel (a pattern per cluster of M / 16 CTAs) at the edges of its
rule: batches on both sides of each limit give the gradients of one oracle, so the
routes agree with each other and with FP64.  Bounds of test_fwd_adj_gpu.py: loss
2e-5, gradients 2e-4 of the largest entry (FD 1e-3), intensities 1e-5."""
import numpy as np
import pytest
import torch

from conftest import load_pkg

pytestmark = pytest.mark.gpu
LOSSES = ("smooth_L1_loss", "Poisson_likelihood_loss", "FD_loss")


def _problem(M, B, seed):
    rng = np.random.default_rng(seed)
    H, W, F = M + 13, M + 6, 6
    c = lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)  # noqa: E731
    O, P = c(H, W), c(M, M) / M
    tl = np.stack([rng.integers(0, H - M + 1, F), rng.integers(0, W - M + 1, F)], 1).astype(np.int32)
    Im = np.abs(rng.standard_normal((F, M, M))).astype(np.float32) * 3
    return O.astype(np.complex64), P.astype(np.complex64), tl, Im, rng.integers(0, F, B).astype(np.int32)


def _exact(O, P, tl, Im, batch, loss):
    """torch autograd in 64 bits of Recovery.py's formulas; frames counted once."""
    O64 = torch.from_numpy(O).to("cuda", torch.complex128).requires_grad_()
    P64 = torch.from_numpy(P).to("cuda", torch.complex128).requires_grad_()
    M, total, Is = P.shape[0], 0.0, []
    count = np.bincount(batch, minlength=len(tl))
    for f, (y, x) in enumerate(tl):
        I = torch.fft.fftshift(torch.fft.fft2(P64 * O64[y:y + M, x:x + M])).abs().square()
        m = torch.from_numpy(Im[f]).to("cuda", torch.float64)
        if loss == "smooth_L1_loss":
            per = torch.nn.functional.smooth_l1_loss(I, m, reduction="none")
        elif loss == "Poisson_likelihood_loss":
            per = I - m * torch.log(I + 1e-8)
        else:
            d = torch.sqrt(m + 1e-8) - torch.sqrt(I + 1e-8)
            rx, ry = torch.roll(d, -1, 1) - d, torch.roll(d, -1, 0) - d
            per = torch.sqrt(rx * rx + ry * ry + 1e-8)
        total = total + int(count[f]) * per.mean()
        Is.append(I.detach())
    return Is, float(total), *torch.autograd.grad(total, (O64, P64))


def _rel(a, b):
    return float((a - b).abs().max() / b.abs().max())


@pytest.mark.parametrize("loss", LOSSES)
@pytest.mark.parametrize("M,B", [(64, 1), (64, 16), (64, 17), (128, 1), (128, 64), (128, 65), (128, 96), (128, 97),
                                 (256, 1), (256, 4), (256, 5), (256, 40)])
def test_both_sides_of_the_rule(M, B, loss):
    pkg = load_pkg()
    O, P, tl, Im, batch = _problem(M, B, 7 * M + B)
    dev = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    args = (dev(O), dev(P), dev(tl), dev(Im), pkg.LOSS_CODES[loss])
    L, per, dO, dP = pkg.fwd_adj_raw(*args, batch=batch, per_pattern=True)
    Is, total, eO, eP = _exact(O, P, tl, Im, batch, loss)
    assert abs(float(L) - total) <= 2e-5 * abs(total)
    tol = 1e-3 if loss == "FD_loss" else 2e-4
    assert _rel(dO, eO) <= tol and _rel(dP, eP) <= tol
    L2, per2, dO2, dP2 = pkg.fwd_adj_raw(*args, batch=batch, per_pattern=True)
    assert torch.equal(dO, dO2) and torch.equal(dP, dP2) and torch.equal(per, per2)
    only = pkg.fwd_adj_raw(*args, batch=batch, want_grad=False)[0]
    assert abs(float(only) - total) <= 2e-5 * abs(total)
    I = pkg.forward_intensity(args[0], args[1], args[2], batch=torch.from_numpy(batch))
    for b in {0, B // 2, B - 1}:
        assert _rel(I[b].double(), Is[batch[b]]) <= 1e-5


@pytest.mark.parametrize("M", [64, 128, 256])
def test_skipped_windows(M):
    """A window off the canvas and a frame id out of range inside a small batch: NaN
    losses and intensities there, the others' gradients, the status raised."""
    pkg = load_pkg()
    O, P, tl, Im, _ = _problem(M, 4, M)
    tl[1, 0] = 14
    batch = np.array([0, 1, 2, 9], np.int32)
    dev = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    pkg.optics.read_status(torch.device("cuda"))
    for loss in LOSSES:
        _, per, dO, dP = pkg.fwd_adj_raw(dev(O), dev(P), dev(tl), dev(Im), pkg.LOSS_CODES[loss], batch=batch,
                                         per_pattern=True)
        _, good, eO, eP = pkg.fwd_adj_raw(dev(O), dev(P), dev(tl), dev(Im), pkg.LOSS_CODES[loss],
                                          batch=np.array([0, 2], np.int32), per_pattern=True)
        assert per.isnan().tolist() == [False, True, False, True] and torch.equal(per[::2], good)
        assert torch.equal(dO, eO) and torch.equal(dP, eP)
    I = pkg.forward_intensity(dev(O), dev(P), dev(tl), batch=dev(batch))
    assert bool(I[1].isnan().all()) and bool(I[3].isnan().all()) and not bool(I[::2].isnan().any())
    assert pkg.optics.read_status(torch.device("cuda")) == 6
