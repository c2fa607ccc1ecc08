"""Functorch transforms and forward-mode differentiation of the C++ autograd nodes are
refused, and a process whose first call of a node was such a one goes on as any other:
the status word that the refused call made is the transform's own and is not kept."""
import subprocess
import sys

import pytest

from conftest import PKG_NAME, ROOT

pytestmark = pytest.mark.gpu

PROGRAM = """
import importlib, sys, torch
import torch.autograd.forward_ad as fwAD
sys.path.insert(0, {root!r})
pkg = importlib.import_module({pkg!r})
dev = "cuda"
torch.manual_seed(0)
mlp = pkg.cmlp.ComplexMLP(32, 64, 2, 1, hidden_omega_0=1.0).to(dev)
x = 0.05 * torch.randn(40, 32, device=dev)
img = torch.randn(30, 32, dtype=torch.complex64, device=dev)
O, P = (torch.randn(n, n, dtype=torch.complex64, device=dev) for n in (90, 64))
tl, Im = torch.tensor([[0, 1]], dtype=torch.int32, device=dev), torch.rand(1, 64, 64, device=dev)
calls = {{"mlp": (lambda z: mlp.net(z).real.sum(), x), "loss": (lambda z: pkg.fused_loss(z, P, tl, Im, "FD_loss"), O),
         "upsample": (lambda z: pkg.resample.fourier_upsample(z, 2).real.sum(), img)}}
first = {first!r}
for name in [first] + [n for n in calls if n != first]:
    fn, a = calls[name]
    def dual():
        with fwAD.dual_level():
            fn(fwAD.make_dual(a, torch.ones_like(a)))
    for refused in (lambda: torch.func.grad(fn)(a), lambda: torch.func.vmap(fn)(torch.stack([a, a])), dual):
        try:
            refused()
        except RuntimeError:
            continue
        raise AssertionError(name + " was not refused")
for name, (fn, a) in calls.items():
    a = a.clone().requires_grad_()
    g, = torch.autograd.grad(fn(a), a)
    assert torch.isfinite(torch.view_as_real(g) if g.is_complex() else g).all() and g.abs().max() > 0, name
assert pkg.read_status(torch.device("cuda", 0)) == 0
print("fine")
"""


@pytest.mark.parametrize("first", ["mlp", "loss", "upsample"])
def test_refusals_leave_nothing_behind(first):
    r = subprocess.run([sys.executable, "-c", PROGRAM.format(root=ROOT, pkg=PKG_NAME, first=first)], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and "fine" in r.stdout, r.stderr[-2000:]
