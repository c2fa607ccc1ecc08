"""The C++ autograd nodes of the complex MLP and the Fourier upsampling
(csrc/torch_ext.cpp) against the Python Functions they stand in for: the same library
calls, so outputs and gradients are bitwise equal, for feature-major, dense and
strided features, frozen inputs and parameters, a graph backed up twice, gradients
with a pending conjugation, saved-tensor hooks, a side stream and no-grad calls."""
import pytest
import torch

from test_inr_gpu import _mlp_from_golden, pkg  # noqa: F401

pytestmark = pytest.mark.gpu


def _both(pkg, fn):  # noqa: F811
    out = []
    for use in (True, False):
        pkg.optics.USE_TORCHEXT = use
        try:
            out.append(fn())
        finally:
            pkg.optics.USE_TORCHEXT = True
    return out


def _same(a, b):
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert (x is None) == (y is None)
        if x is not None:
            assert x.dtype == y.dtype and x.shape == y.shape and torch.equal(x, y)


@pytest.mark.parametrize("layout", ["planar", "dense", "strided", "double"])
@pytest.mark.parametrize("N", [1, 129, 5000])
def test_mlp_routes(pkg, layout, N):  # noqa: F811
    assert pkg._lib.torchext() is not None
    dev = torch.device("cuda")
    mlp, _ = _mlp_from_golden(pkg, 0, dev)
    mlp.net[1].omega_0.requires_grad_(False)
    mlp.net[2].linear.bias.requires_grad_(False)
    ps = [p for p in mlp.parameters() if p.requires_grad]
    g = torch.Generator(device=dev).manual_seed(N)
    base = torch.randn(33, N, device=dev, generator=g) * 0.05
    x = {"planar": base[:32].contiguous().t(), "dense": base[:32].t().contiguous(),
         "strided": base.t().contiguous()[:, 1:], "double": base[:32].t().double()}[layout].requires_grad_()
    gy = torch.randn(N, 1, dtype=torch.complex64, device=dev, generator=g)

    def run():
        y = mlp.net(x)
        first = torch.autograd.grad(y, [x] + ps, gy, retain_graph=True)
        pkg.optics.read_status(dev)  # clears the status word in place between two backwards
        again = torch.autograd.grad(y, [x] + ps, gy.conj().resolve_conj().conj())
        frozen = torch.autograd.grad(mlp.net(x.detach()), ps, gy)
        with torch.no_grad():
            plain = mlp.net(x)
        assert not plain.requires_grad and y.shape == (N, 1)
        _same(first, again)
        _same(first[1:], frozen)
        return [y.detach(), plain, *first]

    if layout == "strided" and N == 1:  # one row is contiguous as it lies: refused for its 4-byte offset
        def refused():
            with pytest.raises(pkg.PtychoError, match="misaligned"):
                mlp.net(x)
            return []
        _both(pkg, refused)
        return
    _same(*_both(pkg, run))


def test_mlp_hooks_and_stream(pkg):  # noqa: F811
    dev = torch.device("cuda")
    mlp, _ = _mlp_from_golden(pkg, 0, dev)
    x = (torch.randn(32, 3000, device=dev) * 0.05).t().requires_grad_()
    gy = torch.randn(3000, 1, dtype=torch.complex64, device=dev)
    ref = torch.autograd.grad(mlp.net(x), [x] + list(mlp.parameters()), gy)
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(1) or t.cpu(), lambda t: t.to(dev)):
        y = mlp.net(x)
    assert packed
    # the features come back from the host in their own (feature-major) strides
    _same(ref, torch.autograd.grad(y, [x] + list(mlp.parameters()), gy))
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        side = torch.autograd.grad(mlp.net(x), [x] + list(mlp.parameters()), gy)
    torch.cuda.current_stream().wait_stream(s)
    _same(ref, side)
    with torch.no_grad():
        x[0, 0] += 1.0
    y = mlp.net(x)
    with torch.no_grad():
        x[0, 0] += 1.0
    with pytest.raises(RuntimeError, match="modified by an inplace"):
        y.backward(gy)


@pytest.mark.parametrize("h,w,s", [(256, 256, 2), (45, 64, 3), (30, 30, 1), (256, 512, 4)])
def test_upsample_routes(pkg, h, w, s):  # noqa: F811
    dev = torch.device("cuda")
    x = torch.randn(w, h, dtype=torch.complex64, device=dev).t().requires_grad_()
    g = torch.randn(h * s, w * s, dtype=torch.complex64, device=dev)

    def run():
        y = pkg.resample.fourier_upsample(x, s)
        gx, = torch.autograd.grad(y, x, g, retain_graph=True)
        g2, = torch.autograd.grad(y.real.sum() + y.imag.square().sum(), x)
        wide = x.detach().to(torch.complex128).requires_grad_()
        g3, = torch.autograd.grad(pkg.resample.fourier_upsample(wide, s), wide, g)
        return [y.detach(), gx, g2, g3]

    _same(*_both(pkg, run))
    with pytest.raises(ValueError):
        pkg.resample.fourier_upsample(x[None], s)
    with pytest.raises(ValueError, match="CUDA"):
        pkg.resample.fourier_upsample(x.detach().cpu(), s)
