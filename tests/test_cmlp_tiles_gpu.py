"""Complex MLP at the edges of its tiling: a tile is 128 coordinates, a CTA (one
per SM) runs four tiles at a time forward and two backward.

Outputs and feature gradients of a coordinate depend on that coordinate alone, so
they are bitwise those of the same coordinates in a call of another size; the
weight gradients are held to the BF16-operand oracle at the bound of
test_inr_gpu.py (rel-to-max 5e-3)."""
import pytest
import torch

from oracle import inr
from test_inr_gpu import _mlp_from_golden, pkg, rel_max  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 127, 128, 129, 148 * 128 - 1, 148 * 128 + 1, 2 * 148 * 128 + 1,
                               4 * 148 * 128 + 129, 9 * 148 * 128 + 130])
def test_tiles(pkg, N):  # noqa: F811
    dev = torch.device("cuda")
    mlp, params = _mlp_from_golden(pkg, 0, dev)
    g = torch.Generator(device=dev).manual_seed(N)
    x = (torch.randn(32, N, device=dev, generator=g) * 0.05).t().requires_grad_(True)
    gy = torch.randn(N, 1, dtype=torch.complex64, device=dev, generator=g)
    ps = list(mlp.parameters())
    y = mlp.net(x)
    dx, *dw = torch.autograd.grad(y, [x] + ps, gy)
    # the last 200 coordinates (the tail of the last tiles) on their own
    k = min(N, 200)
    xs = x[N - k:].detach().clone().requires_grad_(True)
    ys = mlp.net(xs)
    dxs, = torch.autograd.grad(ys, xs, gy[N - k:])
    assert torch.equal(y[N - k:], ys) and torch.equal(dx[N - k:], dxs)
    # feature gradients skipped: the same weight gradients
    for a, b in zip(dw, torch.autograd.grad(mlp.net(x.detach()), ps, gy)):
        assert torch.equal(a, b)
    xn, gn = x.detach().cpu().numpy().astype("float64"), gy.cpu().numpy()[:, 0]
    yq, cq = inr.cmlp_forward(xn, params, q=inr.bf16_round, qh=inr.bf16_split)
    gq = inr.cmlp_backward(gn, params, cq)
    assert rel_max(y.detach().cpu().numpy()[:, 0], yq) <= 5e-3
    # parameters() order: (omega, weight, bias) of three layers, output weight and bias
    ref = [None, gq["W1"], gq["b1"], None, gq["Wh"][0], gq["bh"][0], None, gq["Wh"][1], gq["bh"][1], gq["Wo"], gq["bo"]]
    for i, (d, r) in enumerate(zip(dw, ref)):
        if r is not None:
            assert rel_max(d.cpu().numpy().reshape(-1), r.reshape(-1)) <= 5e-3, i


def test_output_from_the_backward(pkg):  # noqa: F811
    """The backward entry's own y (C ABI, optional) against the forward's."""
    dev = torch.device("cuda")
    mlp, _ = _mlp_from_golden(pkg, 0, dev)
    L, N = pkg.lib(), 3000
    x = torch.randn(32, N, device=dev) * 0.05
    y0 = mlp.net(x.t()).detach()[:, 0]
    flat = [pkg.cmlp._f32(p) for p in pkg.cmlp._params(mlp.net)]
    s = torch.cuda.current_stream().cuda_stream
    packed = torch.empty(int(L.ptycho_cmlp_packed_bytes()), dtype=torch.uint8, device=dev)
    pkg._lib.check(L.ptycho_cmlp_pack(*[f.data_ptr() for f in flat], packed.data_ptr(), s), "pack")
    gy = torch.randn(N, dtype=torch.complex64, device=dev)
    grad = torch.empty(int(L.ptycho_cmlp_grad_floats()), device=dev)
    y = torch.empty(N, dtype=torch.complex64, device=dev)
    ws = torch.empty(int(L.ptycho_cmlp_backward_workspace_size(N)), dtype=torch.uint8, device=dev)
    pkg._lib.check(L.ptycho_cmlp_backward_planar(packed.data_ptr(), x.data_ptr(), gy.data_ptr(), N, None,
                                                 grad.data_ptr(), y.data_ptr(), ws.data_ptr(), ws.numel(), None, s),
                   "backward")
    # FP32 output weights' products against BF16 hi + lo ones: 2^-16 of the terms' size
    assert float((y - y0).abs().max() / y0.abs().max()) <= 64 * 2.0 ** -16
