"""Edges of the hash encoding's kernels (csrc/hashgrid.cu).

Backward on grid coordinates: single rows and columns, cells longer than a fine
tile's tables, cells at the line between the two-pass and the tiled levels, levels
finer than the grid (empty cells), tiles one vertex wider than a block, against the
FP64 oracle with float32 positions.  Tolerance 1e-5 of the largest entry: FP32 sums
of up to a few thousand serial terms of random sign (sqrt(n) rounding errors of
6e-8 of partial sums no larger than the largest entry's).
Forward: coordinates inside [0, 1], on its ends and outside it, both layouts bitwise
equal, against the FP64 bilinear sum at float32 positions: 4 products and 3 sums,
8 * 2^-24 of the largest table value.
"""
import numpy as np
import pytest
import torch

from conftest import load_pkg
from oracle import inr

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pkg():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    return load_pkg()


def _enc(pkg, cfg):
    L, log2T, base, pls = cfg
    return pkg.Encoding(2, {"otype": "HashGrid", "n_levels": L, "n_features_per_level": 2, "log2_hashmap_size": log2T,
                            "base_resolution": base, "per_level_scale": pls}).to("cuda")


@pytest.mark.parametrize("A,Bj,cfg", [
    (2, 3000, (6, 12, 4, 1.9)), (3000, 2, (6, 12, 4, 1.9)), (1000, 5, (5, 10, 3, 2.0)), (1, 5000, (5, 14, 4, 1.8)),
    (3, 4000, (5, 14, 6, 1.9)), (33, 300, (8, 12, 4, 1.7)),
    (256, 256, (5, 16, 63, 1.01)), (257, 130, (4, 16, 255, 1.01)), (70, 70, (8, 14, 16, 1.6)),
    (513, 511, (3, 19, 508, 1.01)), (1030, 64, (6, 14, 16, 1.9))])
def test_grid_backward_edges(pkg, A, Bj, cfg):
    L, log2T, base, pls = cfg
    enc = _enc(pkg, cfg)
    enc.use_grid_plan = True
    xs, ys = torch.linspace(0.5 / A, 1 - 0.5 / A, A), torch.linspace(0.5 / Bj, 1 - 0.5 / Bj, Bj)
    xv, yv = torch.meshgrid([xs, ys], indexing="ij")
    coords = torch.stack((yv.flatten(), xv.flatten())).t().contiguous().cuda()
    g = torch.randn((2 * L, A * Bj), device="cuda", generator=torch.Generator(device="cuda").manual_seed(A))
    got = []
    for gy in (g.t(), g.t().contiguous()):
        got.append(torch.autograd.grad(enc(coords), enc.params, gy)[0])
        assert isinstance(enc._csr[-1][3], pkg.hashgrid.GridPlan)
    assert torch.equal(*got)
    ref = inr.hashgrid_backward(coords.cpu().numpy().astype(np.float64), g.t().cpu().numpy(),
                                inr.hashgrid_levels(L, log2T, base, float(np.float32(pls))), enc.n_entries,
                                fp32_positions=True)
    assert float(np.abs(got[0].cpu().numpy() - ref).max()) <= 1e-5 * np.abs(ref).max()


@pytest.mark.parametrize("cfg", [(16, 14, 16, 1.32), (4, 19, 5, 2.0), (3, 8, 2000, 3.0), (2, 10, 2 ** 19, 3.0)])
def test_forward_edges(pkg, cfg):
    L, log2T, base, pls = cfg
    enc = _enc(pkg, cfg)
    rng = np.random.default_rng(L)
    x = rng.random((1003, 2)).astype(np.float32)
    x[0], x[1], x[2], x[3], x[4], x[5] = (0, 0), (1, 1), (0, 1), (-0.0, 1), (1 - 2.0 ** -24, 2.0 ** -30), (-0.3, 0.5)
    x[6], x[7], x[8] = (1.7, 0.2), (3.0, -2.0), (np.nextafter(np.float32(1), np.float32(2)), 0.5)
    feats = enc(torch.from_numpy(x).cuda()).detach()
    L_ = pkg._lib.lib()
    row = torch.empty((len(x), 2 * L), device="cuda")
    xc = torch.from_numpy(x).cuda()
    assert L_.ptycho_hashgrid_forward(xc.data_ptr(), len(x), enc.params.data_ptr(), *enc.cfg, row.data_ptr(), 0) == 0
    torch.cuda.synchronize()
    assert torch.equal(row, feats)
    tab = enc.params.detach().cpu().numpy().reshape(-1, 2).astype(np.float64)
    for l, (scale, res, n, off, dense) in enumerate(pkg.hashgrid.level_table(*enc.cfg)):
        p = (x.astype(np.float64) * np.float64(np.float32(scale)) + 0.5).astype(np.float32)  # one rounding
        c = np.floor(p)
        f = (p - c).astype(np.float64)
        c = c.astype(np.int64)
        want = np.zeros((len(x), 2))
        for dx in (0, 1):
            for dy in (0, 1):
                u, v = (c[:, 0] + dx) & 0xFFFFFFFF, (c[:, 1] + dy) & 0xFFFFFFFF
                e = ((u + v * res) if dense else (u ^ (v * 2654435761 & 0xFFFFFFFF))) & 0xFFFFFFFF
                w = (f[:, 0] if dx else 1 - f[:, 0]) * (f[:, 1] if dy else 1 - f[:, 1])
                want += w[:, None] * tab[off + e % n]
        err = np.abs(row[:, 2 * l:2 * l + 2].cpu().numpy() - want).max()
        assert err <= 8 * 2.0 ** -24 * np.abs(tab).max()
