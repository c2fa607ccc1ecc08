"""The general path's row passes choose their lines per block by the batch
(csrc/general.cu run_rows): batches on both sides of the line give every pattern the
same transform.  Intensities are bitwise those of small batches; the gradients of the
whole batch are the sums of the parts' within 2e-5 of their 2-norm (FP32 sums of at
most 600 terms in another order, sqrt(600) * 2^-24 of the sum expected)."""
import pytest
import torch

from conftest import load_pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,B", [(7, 10, 591), (7, 10, 592), (10, 12, 601), (96, 100, 160)])
def test_batches_agree(M, N, B):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    pkg = load_pkg()
    g = torch.Generator(device="cuda").manual_seed(B)
    O = torch.randn(150, 150, dtype=torch.complex64, device="cuda", generator=g)
    P = torch.randn(M, N, dtype=torch.complex64, device="cuda", generator=g) / M
    tl = torch.randint(0, 50, (B, 2), device="cuda", generator=g, dtype=torch.int32)
    Im = torch.rand(B, M, N, device="cuda", generator=g)
    ids = torch.arange(B, device="cuda", dtype=torch.int32)
    whole = pkg.forward_intensity(O, P, tl)
    parts = torch.cat([pkg.forward_intensity(O, P, tl, batch=ids[i:i + 50]) for i in range(0, B, 50)])
    assert torch.equal(whole, parts)
    code = pkg.LOSS_CODES["smooth_L1_loss"]
    dO, dP = pkg.fwd_adj_raw(O, P, tl, Im, code)[2:]
    sO, sP = torch.zeros_like(dO, dtype=torch.complex128), torch.zeros_like(dP, dtype=torch.complex128)
    for i in range(0, B, 50):
        a, b = pkg.fwd_adj_raw(O, P, tl, Im, code, batch=ids[i:i + 50])[2:]
        sO += a
        sP += b
    for x, y in ((dO, sO), (dP, sP)):
        assert float(torch.linalg.norm(x - y) / torch.linalg.norm(y)) <= 2e-5
