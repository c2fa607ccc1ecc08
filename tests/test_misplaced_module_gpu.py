"""A module whose parameters are not where the features are, or not of the shapes the
kernels read, is refused on the host with ValueError, before any launch: the kernels
would read host memory or past the end.  Both autograd routes."""
import pytest
import torch

from conftest import load_pkg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pkg():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    return load_pkg()


class _NoCalls:
    """stands in for the library: any entry point called is the test's failure"""

    def __getattr__(self, name):
        raise AssertionError(f"{name} was called")


@pytest.fixture(params=[True, False], ids=["cpp", "python"])
def route(request, pkg, monkeypatch):
    ext = pkg._lib.torchext()
    assert ext is not None
    monkeypatch.setattr(pkg.optics, "USE_TORCHEXT", request.param)
    monkeypatch.setattr(pkg._lib, "lib", lambda: _NoCalls())
    return request.param


def _mlp(pkg):
    return pkg.cmlp.ComplexMLP(32, 64, 2, 1, hidden_omega_0=1.0)


def test_mlp_on_the_host(pkg, route):
    x = torch.zeros(5, 32, device="cuda")
    with pytest.raises(ValueError, match="is on cpu"):
        _mlp(pkg).net(x)
    one = _mlp(pkg).to("cuda")  # one parameter left behind
    one.net[2].linear.bias.data = one.net[2].linear.bias.data.cpu()
    with pytest.raises(ValueError, match="is on cpu"):
        one.net(x)


@pytest.mark.parametrize("shape", [(5, 16), (32,), (2, 5, 32), (5, 33)])
def test_feature_shape(pkg, route, shape):
    with pytest.raises(ValueError, match="features must be"):
        _mlp(pkg).to("cuda").net(torch.zeros(shape, device="cuda"))


def test_parameter_shapes(pkg, route):
    x = torch.zeros(5, 32, device="cuda")
    for i, p in ((1, torch.zeros(32, 16, dtype=torch.complex64)), (1, torch.zeros(32, 32)),
                 (2, torch.zeros(32, 16, dtype=torch.complex64))):
        m = _mlp(pkg).to("cuda")
        m.net[i].linear.weight = torch.nn.Parameter(p.to("cuda"))
        with pytest.raises(ValueError, match="has shape"):
            m.net(x)
    m = _mlp(pkg).to("cuda")
    m.net[0].linear.weight = torch.nn.Parameter(torch.zeros(32, 31, device="cuda"))
    with pytest.raises(ValueError, match="has shape"):
        m.net(x)


def test_encoder_and_model(pkg, monkeypatch):
    cfg = {"n_levels": 4, "base_resolution": 4}
    enc = pkg.Encoding(2, cfg)
    half = pkg.Encoding(2, cfg).to("cuda").half()
    good = pkg.Encoding(2, cfg).to("cuda")
    model = pkg.ComplexINRModel2D(24, 24, 1, update_probe=False)
    xy = torch.zeros(7, 2, device="cuda")
    monkeypatch.setattr(pkg._lib, "lib", lambda: _NoCalls())
    with pytest.raises(ValueError, match="table is on cpu"):
        enc(xy)
    with pytest.raises(ValueError, match="contiguous float32"):
        half(xy)
    for bad in (torch.zeros(7, 1, device="cuda"), torch.zeros(7, device="cuda"), torch.zeros(7, 3, device="cuda")):
        with pytest.raises(ValueError, match="coordinates must be"):
            good(bad)
    with pytest.raises(ValueError, match="table is on cpu"):
        model()
    with pytest.raises(ValueError, match="initial estimate"):
        pkg.complex_inr._Residual.apply(torch.tensor(1.0), torch.zeros(4, 4, dtype=torch.complex64, device="cuda"),
                                        torch.zeros(4, 3, dtype=torch.complex64), None)
    with pytest.raises(ValueError, match="CUDA"):
        pkg.complex_inr._Residual.apply(torch.tensor(1.0), torch.zeros(4, 4, dtype=torch.complex64),
                                        torch.zeros(4, 4, dtype=torch.complex64), None)


def test_residual_scale_on_the_host(pkg):
    """k as a 0-d host parameter goes along to the device, its gradient comes back."""
    m = torch.randn(6, 5, dtype=torch.complex64, device="cuda")
    ws = torch.zeros(int(pkg.lib().ptycho_residual_workspace_size()), dtype=torch.uint8, device="cuda")
    out = []
    for dev in ("cpu", "cuda"):
        k = torch.tensor(0.5, device=dev, requires_grad=True)
        y = pkg.complex_inr._Residual.apply(k, m, m, ws)
        y.real.sum().backward()
        out.append((y.detach(), k.grad.cpu()))
        assert k.grad.device.type == dev
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
