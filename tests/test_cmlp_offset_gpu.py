"""Feature-major MLP inputs at any 4-byte offset (rows 1 .. 32 of a [33, N] buffer with N
odd) pass through forward and backward, bitwise as an aligned copy does; the C entry
takes such a feature gradient too.  Dense rows at such an offset stay refused."""
import pytest
import torch

from test_inr_gpu import _mlp_from_golden, pkg  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("route", [True, False])
@pytest.mark.parametrize("N", [2, 129, 1001])
def test_offset_features(pkg, N, route, monkeypatch):  # noqa: F811
    monkeypatch.setattr(pkg.optics, "USE_TORCHEXT", route)
    dev = torch.device("cuda")
    mlp, _ = _mlp_from_golden(pkg, 0, dev)
    g = torch.Generator(device=dev).manual_seed(N)
    base = 0.05 * torch.randn(33 * N + 1, device=dev, generator=g)
    gy = torch.randn(N, 1, dtype=torch.complex64, device=dev, generator=g)
    for off in (1, N, N + 1):
        x = base[off:off + 32 * N].view(32, N).t()
        assert pkg.cmlp._is_planar(x)
        out = []
        for v in (x, x.t().clone().t()):
            v = v.detach().requires_grad_()
            y = mlp.net(v)
            out.append([y.detach(), *torch.autograd.grad(y, [v] + list(mlp.parameters()), gy)])
        assert out[0][0].isfinite().all()
        assert all(torch.equal(a, b) for a, b in zip(*out))


def test_offset_feature_gradient(pkg):  # noqa: F811
    dev = torch.device("cuda")
    mlp, _ = _mlp_from_golden(pkg, 0, dev)
    N = 77
    L = pkg.lib()
    flat = [pkg.cmlp._f32(p) for p in pkg.cmlp._params(mlp.net)]
    packed = torch.empty(int(L.ptycho_cmlp_packed_bytes()), dtype=torch.uint8, device=dev)
    pkg._lib.check(L.ptycho_cmlp_pack(*[f.data_ptr() for f in flat], packed.data_ptr(), None), "pack")
    x = 0.05 * torch.randn(32, N, device=dev)
    gy = torch.randn(N, dtype=torch.complex64, device=dev)
    ws = torch.empty(int(L.ptycho_cmlp_backward_workspace_size(N)), dtype=torch.uint8, device=dev)
    st = pkg.optics.device_status(dev)
    got = []
    for off in (0, 1):
        buf = torch.full((32 * N + 2,), 7.0, device=dev)
        gx, grad = buf[off:off + 32 * N], torch.empty(int(L.ptycho_cmlp_grad_floats()), device=dev)
        pkg._lib.check(L.ptycho_cmlp_backward_planar(packed.data_ptr(), x.data_ptr(), gy.data_ptr(), N, gx.data_ptr(),
                                                     grad.data_ptr(), None, ws.data_ptr(), ws.numel(), st.data_ptr(),
                                                     None), "backward")
        torch.cuda.synchronize()
        assert float(buf[off + 32 * N]) == 7.0 and (off == 0 or float(buf[0]) == 7.0)
        got.append((gx.clone(), grad))
        assert L.ptycho_cmlp_backward(packed.data_ptr(), x.data_ptr() + 4, gy.data_ptr(), N - 1, None, grad.data_ptr(),
                                      None, ws.data_ptr(), ws.numel(), st.data_ptr(), None) != 0
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
