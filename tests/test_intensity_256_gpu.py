"""M = 256 intensities through the row and column kernels (workspace) and through the
cluster kernel (a small or no workspace): both against FP64 (1e-5 of the largest
intensity, test_fwd_adj_256_gpu.py's bound), with frame ids, skipped windows and
batches over one chunk of the scratch."""
import pytest
import torch

from conftest import load_pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 3, 65, 515])
def test_both_routes(B):
    pkg = load_pkg()
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(B)
    r = lambda *s: torch.complex(torch.randn(s, generator=g, device=dev), torch.randn(s, generator=g, device=dev))  # noqa: E731
    H, W, M = 300, 283, 256
    O, P = r(H, W), r(M, M) / M
    tl = torch.stack([torch.randint(0, H - M + 1, (7,), generator=g, device=dev),
                      torch.randint(0, W - M + 1, (7,), generator=g, device=dev)], 1).to(torch.int32)
    tl[5, 0] = H - M + 1  # leaves the canvas
    batch = torch.randint(0, 5, (B,), generator=g, device=dev, dtype=torch.int32)
    if B > 2:
        batch[1], batch[2] = 5, 9  # a bad window, a frame id out of range
    pkg.optics.read_status(dev)
    got = pkg.forward_intensity(O, P, tl, batch=batch)
    assert pkg.optics.read_status(dev) == (6 if B > 2 else 0)
    cluster = torch.empty_like(got)
    L = pkg.lib()
    pkg._lib.check(L.ptycho_forward_intensity(O.data_ptr(), H, W, P.data_ptr(), M, M, tl.data_ptr(), 7, batch.data_ptr(),
                                              B, cluster.data_ptr(), None, torch.cuda.current_stream().cuda_stream), "cluster")
    small = torch.empty_like(got)
    ws = torch.empty(256, dtype=torch.uint8, device=dev)
    pkg._lib.check(L.ptycho_forward_intensity_ws(O.data_ptr(), H, W, P.data_ptr(), M, M, tl.data_ptr(), 7,
                                                 batch.data_ptr(), B, small.data_ptr(), ws.data_ptr(), 256, None,
                                                 torch.cuda.current_stream().cuda_stream), "small workspace")
    assert torch.equal(small.nan_to_num(-1.0), cluster.nan_to_num(-1.0))
    O64, P64 = O.to(torch.complex128), P.to(torch.complex128)
    ref = torch.stack([torch.fft.fftshift(torch.fft.fft2(P64 * O64[y:y + M, x:x + M])).abs().square()
                       for y, x in tl[:5].tolist()])
    for b, f in enumerate(batch.tolist()):
        if f >= 5:
            assert bool(got[b].isnan().all()) and bool(cluster[b].isnan().all())
        else:
            assert float((got[b].double() - ref[f]).abs().max()) <= 1e-5 * float(ref[f].max())
            assert float((cluster[b].double() - ref[f]).abs().max()) <= 1e-5 * float(ref[f].max())
