"""Inputs and gradients with a pending conjugation or negation (``x.conj()`` is a view
that only carries a flag) give bitwise what their resolved copies give, through every
entry that hands a tensor's memory to the library: contiguous and transposed views,
both autograd routes."""
import pytest
import torch

from conftest import load_pkg

pytestmark = pytest.mark.gpu
LOSSES = ("smooth_L1_loss", "FD_loss", "Poisson_likelihood_loss")


@pytest.fixture(scope="module")
def pkg():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    return load_pkg()


def _c(*n, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + sum(n))
    return torch.randn(n, dtype=torch.complex64, device="cuda", generator=g)


def _same(a, b):
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert torch.equal(x.resolve_conj().resolve_neg(), y.resolve_conj().resolve_neg())


def _scan(M, N):
    O, P = 0.3 * _c(M + 40, N + 50), _c(M, N, seed=1) / M
    tl = torch.tensor([[0, 3], [40, 50], [11, 7]], dtype=torch.int32, device="cuda")
    Im = 5.0 * torch.rand(3, M, N, device="cuda", generator=torch.Generator(device="cuda").manual_seed(M))
    return O, P, tl, Im


@pytest.mark.parametrize("M,N", [(64, 64), (128, 128), (256, 256), (90, 77)])
def test_forward_and_losses(pkg, M, N, monkeypatch):
    O, P, tl, Im = _scan(M, N)
    views = [(O.conj(), P.conj()), (O.t().contiguous().t().conj(), P), (O, P.conj())]
    for Ov, Pv in views:
        Or, Pr = Ov.resolve_conj().clone(), Pv.resolve_conj().clone()
        assert (Ov.is_conj() or Pv.is_conj()) and not Or.is_conj()
        _same([pkg.forward_intensity(Ov, Pv, tl)], [pkg.forward_intensity(Or, Pr, tl)])
        for k, loss in enumerate(LOSSES):
            def raw(o, p):
                total, per, dO, dP = pkg.fwd_adj_raw(o, p, tl, Im, pkg.LOSS_CODES[loss], per_pattern=True)
                return [total, per, dO, dP]
            _same(raw(Ov, Pv), raw(Or, Pr))
            for route in (True, False):
                monkeypatch.setattr(pkg.optics, "USE_TORCHEXT", route)

                def grads(o, p):  # with respect to the views themselves
                    o, p = o.detach().requires_grad_(), p.detach().requires_grad_()
                    total = pkg.fused_loss(o, p, tl, Im, loss)
                    return [total.detach(), *torch.autograd.grad(total, (o, p))]
                _same(grads(Ov, Pv), grads(Or, Pr))
        with pytest.raises(ValueError, match="conjugation"):
            pkg.optics.FwdAdjPlan(O, P.conj(), tl, Im, "FD_loss", 3)
        with pytest.raises(ValueError, match="conjugation"):
            pkg.optics.FwdAdjPlan(O, P, tl, torch._neg_view(Im), "FD_loss", 3)


@pytest.mark.parametrize("route", [True, False])
def test_negated_measurements_and_loss_gradients(pkg, route, monkeypatch):
    monkeypatch.setattr(pkg.optics, "USE_TORCHEXT", route)
    O, P, tl, Im = _scan(64, 64)
    O.requires_grad_()
    want = torch.autograd.grad(pkg.fused_loss(O, P, tl, Im, LOSSES[0]), O)
    _same(torch.autograd.grad(pkg.fused_loss(O, P, tl, torch._neg_view(-Im), LOSSES[0]), O), want)
    loss = pkg.fused_loss(O, P, tl, Im, LOSSES[0])
    minus = -torch.ones((), dtype=torch.float64, device="cuda")
    _same(torch.autograd.grad(loss, O, torch._neg_view(minus)), want)
    I = pkg.forward_intensity_batched(O, P, tl)
    _same(torch.autograd.grad(I, O, torch._neg_view(-Im), retain_graph=True), torch.autograd.grad(I, O, Im))


@pytest.mark.parametrize("route", [True, False])
def test_inr_parts(pkg, route, monkeypatch):
    monkeypatch.setattr(pkg.optics, "USE_TORCHEXT", route)
    prep, inr = pkg.probe_prep, pkg.complex_inr

    def both(fn, *args):
        """fn on conjugated views of args, and on resolved copies: outputs and gradients"""
        out = []
        for xs in ([a.conj() for a in args], [a.conj().resolve_conj().clone() for a in args]):
            leaves = [x.detach().requires_grad_() for x in xs]
            y = fn(*leaves)
            g = _c(*y.shape, seed=3) if y.is_complex() else torch.ones_like(y)
            out.append([y.detach(), *torch.autograd.grad(y, leaves, g, retain_graph=True)])
            if y.is_complex():  # a conjugated gradient
                _same(torch.autograd.grad(y, leaves, g.conj().resolve_conj().conj()), out[-1][1:])
        _same(*out)

    both(lambda x: pkg.resample.fourier_upsample(x, 2), _c(256, 64))
    both(prep.center_and_normalize_probe, _c(48, 50))
    both(prep.haar_sparsity, _c(40, 36))
    k = torch.tensor(0.3, device="cuda")
    ws = torch.zeros(int(pkg.lib().ptycho_residual_workspace_size()), dtype=torch.uint8, device="cuda")
    both(lambda m, i: inr._Residual.apply(k, m, i, ws), _c(33, 5), _c(33, 5, seed=9))
    a, b = _c(30, 31), _c(30, 31, seed=2)
    _same([pkg.accuracy.object_error(a.conj(), b)["tensor"]],
          [pkg.accuracy.object_error(a.conj().resolve_conj(), b)["tensor"]])
    mlp = pkg.cmlp.ComplexMLP(32, 64, 2, 1, hidden_omega_0=1.0).to("cuda")
    x = 0.05 * torch.randn(257, 32, device="cuda")
    with torch.no_grad():
        _same([mlp.net(torch._neg_view(-x))], [mlp.net(x)])
    enc = pkg.Encoding(2, {"n_levels": 4, "base_resolution": 4}).to("cuda")
    xy = torch.rand(100, 2, device="cuda")
    f = enc(xy)
    _same([enc(torch._neg_view(-xy)).detach()], [f.detach()])
    g = torch.randn_like(f)
    _same(torch.autograd.grad(f, enc.params, torch._neg_view(-g), retain_graph=True),
          torch.autograd.grad(f, enc.params, g))


def test_adam_takes_a_conjugated_gradient(pkg):
    ps = [_c(20, 7).requires_grad_() for _ in range(2)]
    g = _c(20, 7, seed=5)
    ps[0].grad, ps[1].grad = g.conj(), g.conj().resolve_conj()
    for p in ps:
        pkg.FusedAdam([p], lr=1e-2).step()
    assert torch.equal(ps[0].detach(), ps[1].detach())
