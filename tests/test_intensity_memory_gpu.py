"""forward_intensity at 256^2 where the scratch of the row and column kernels cannot be
had: the cluster kernel, which needs none, bitwise the entry point without a workspace.
Other shapes need their workspace and raise."""
import pytest
import torch

from conftest import load_pkg

pytestmark = pytest.mark.gpu


def test_without_room_for_scratch(monkeypatch):
    pkg = load_pkg()
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(0)
    O = torch.randn(290, 270, dtype=torch.complex64, device=dev, generator=g)
    P = torch.randn(256, 256, dtype=torch.complex64, device=dev, generator=g) / 256
    B = 60
    tl = torch.stack([torch.arange(B, device=dev) % 35, torch.arange(B, device=dev) % 15], 1).to(torch.int32)
    L = pkg.lib()
    assert int(L.ptycho_forward_intensity_workspace_size(256, 256, B)) > B * 256 * 256 * 8
    want = torch.empty((B, 256, 256), device=dev)
    pkg._lib.check(L.ptycho_forward_intensity(O.data_ptr(), 290, 270, P.data_ptr(), 256, 256, tl.data_ptr(), B, None, B,
                                              want.data_ptr(), None, torch.cuda.current_stream().cuda_stream), "cluster")
    pkg.optics.device_status(dev)
    empty = torch.empty

    def full(*a, **k):
        if k.get("dtype") == torch.uint8:
            raise torch.cuda.OutOfMemoryError("no room for the scratch")
        return empty(*a, **k)

    monkeypatch.setattr(torch, "empty", full)
    assert torch.equal(pkg.forward_intensity(O, P, tl), want)
    with pytest.raises(torch.cuda.OutOfMemoryError):
        pkg.forward_intensity(O, P[:192, :192], tl)
