"""M = 256 on clusters of eight CTAs, where a part of the chip cannot hold sixteen
together (csrc/cluster_small.cuh).  A whole chip takes the sixteen, so these kernels
are compiled here: intensities and E' are bitwise those of the larger clusters (each
value goes through the same sums), losses equal to the rounding of an FP64 sum."""
import ctypes
import importlib.util
import os
import subprocess

import pytest
import torch

from conftest import PKG_NAME, ROOT, load_pkg

pytestmark = pytest.mark.gpu
CSRC = os.path.join(ROOT, PKG_NAME, "csrc")
SOURCE = r"""
#include "cluster_small.cuh"
using namespace pty;
extern "C" int run(int mode, const float* O, int H, int W, const float* P, const int* tl, const float* Im, int F, int B,
                   float* out, int* tlb, double* loss, int* status) {
  FusedArgs a{};
  a.O = reinterpret_cast<const float2*>(O);
  a.P = reinterpret_cast<const float2*>(P);
  a.tl = reinterpret_cast<const int2*>(tl);
  a.Imeas = Im;
  a.H = H;
  a.W = W;
  a.F = F;
  a.B = B;
  a.status = status;
  a.loss_pat = loss;
  a.tlb = reinterpret_cast<int2*>(tlb);
  a.I_out = out;
  a.Eout = reinterpret_cast<float2*>(out);
  if (mode == MODE_INTENSITY) return csm::launch<256, 8, MODE_INTENSITY, 0>(a, nullptr);
  if (mode == MODE_ADJ) return csm::launch<256, 8, MODE_ADJ, PTYCHO_LOSS_FD>(a, nullptr);
  return csm::launch<256, 8, MODE_LOSS, PTYCHO_LOSS_FD>(a, nullptr);
}
extern "C" int modes(int i) { return i == 0 ? MODE_INTENSITY : (i == 1 ? MODE_LOSS : MODE_ADJ); }
"""


@pytest.fixture(scope="module")
def kernels(tmp_path_factory):
    spec = importlib.util.spec_from_file_location("ptycho_build", os.path.join(CSRC, "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    d = tmp_path_factory.mktemp("cluster8")
    (d / "t.cu").write_text(SOURCE)
    subprocess.run([build.nvcc(), *build.ARCH, *build.FLAGS, "-shared", str(d / "t.cu"), "-o", str(d / "t.so")], check=True)
    return ctypes.CDLL(str(d / "t.so"))


@pytest.mark.parametrize("B", [1, 3, 20])
def test_bitwise_as_the_large_clusters(kernels, B):
    pkg = load_pkg()
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(B)
    M, H, W = 256, 300, 283
    O = torch.randn(H, W, dtype=torch.complex64, device=dev, generator=g)
    P = torch.randn(M, M, dtype=torch.complex64, device=dev, generator=g) / M
    tl = torch.stack([torch.randint(0, H - M + 1, (B,), generator=g, device=dev),
                      torch.randint(0, W - M + 1, (B,), generator=g, device=dev)], 1).to(torch.int32)
    if B > 1:
        tl[1, 1] = W - M + 1  # leaves the canvas
    good = [b for b in range(B) if b != 1]
    Im = 4.0 * torch.rand(B, M, M, device=dev, generator=g)
    L = pkg.lib()
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    # the library, on clusters of sixteen
    I16 = torch.empty(B, M, M, device=dev)
    pkg._lib.check(L.ptycho_forward_intensity(O.data_ptr(), H, W, P.data_ptr(), M, M, tl.data_ptr(), B, None, B,
                                              I16.data_ptr(), None, None), "intensity")
    ws = pkg.optics.FwdAdjWorkspace()
    pkg.optics.read_status(dev)
    total, per16, _, _ = pkg.fwd_adj_raw(O, P, tl, Im, pkg.LOSS_CODES["FD_loss"], per_pattern=True, workspace=ws)
    torch.cuda.synchronize()
    code = pkg.optics.read_status(dev)
    E16 = ws.buf[:B * M * M * 8].view(torch.float32).view(B, M, M, 2)  # E' comes first in the workspace

    I8, E8 = torch.zeros(B, M, M, device=dev), torch.zeros(B, M, M, 2, device=dev)
    per8, per8l = (torch.zeros(B, dtype=torch.float64, device=dev) for _ in range(2))
    tlb = torch.zeros(B, 2, dtype=torch.int32, device=dev)
    st = torch.zeros(1, dtype=torch.int32, device=dev)
    for k, out, loss in ((0, I8, None), (1, E8, per8l), (2, E8, per8)):
        assert kernels.run(kernels.modes(k), p(O), H, W, p(P), p(tl), p(Im), B, B, p(out), p(tlb),
                           p(loss) if loss is not None else None, p(st)) == 0
        torch.cuda.synchronize()
        if k == 1:
            assert not bool(E8.any())
    assert int(st) == code == (6 if B > 1 else 0)
    assert torch.equal(I8[good], I16[good]) and torch.equal(E8[good], E16[good])
    assert torch.equal(per8, per8l) if B == 1 else torch.equal(per8[good], per8l[good])
    # sums of 65536 positive FP64 terms in another order: at most 65536 units of 2^-53
    assert float(((per8 - per16)[good].abs() / per16[good]).max()) <= 65536 * 2.0 ** -53
    if B > 1:
        assert bool(I8[1].isnan().all()) and bool(per8[1].isnan()) and tlb[1].tolist() == [-1, -1]
    assert torch.equal(tlb[good], tl[good])
