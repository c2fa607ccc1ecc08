"""The work a user of this framework has it do, as timed cases.

Six kinds of pass, each through a public entry point, over the sizes of the
framework's own workloads (``synth.WORKLOADS`` c0 to c4, the INR settings of
``bench.py``) and the odd ones a data set brings:

* ``step``: one pixel-grid minibatch, forward + loss + adjoint, as a captured
  training step replays it (``optics.FwdAdjPlan``);
* ``loss``: the same minibatch through the autograd entry (``fused_loss`` and
  its backward), called eagerly;
* ``intensity``: the forward model alone, as the residual evaluation calls it
  (``forward_intensity``);
* ``encode``: a hash encoding's forward and table gradient (``Encoding``);
* ``mlp``: a complex MLP's forward and backward (``ComplexMLP.net``);
* ``upsample``: the Fourier upsampling of the object, both ways
  (``resample.fourier_upsample``);
* ``model``: a whole ``ComplexINRModel2D`` evaluated to object and probe.

``exact`` restates every kind in torch at 64 bits, without the framework.
"""
from __future__ import annotations

import importlib
import math

import numpy as np
import torch

DEV = "cuda"
LOSSES = ("smooth_L1_loss", "Poisson_likelihood_loss", "FD_loss")


def _pkg():
    return importlib.import_module("conventional-ptychography-reconstruction_b200")


# --------------------------------------------------------------------------
# cases
# --------------------------------------------------------------------------
def _scan_case(kind, canvas, M, N, scan, step, jitter, batch, loss, peak):
    return {"kind": kind, "canvas": canvas, "M": M, "N": N, "scan": scan, "step": step, "jitter": jitter,
            "batch": batch, "loss": loss, "peak": peak}


def listed():
    return [
        # the smallest reconstruction and the reference's default batch: launch and latency bound
        {"name": "step_64_b10", **_scan_case("step", 256, 64, 64, 10, 16, 2, 10, "smooth_L1_loss", 1e3)},
        # the default batch of 10 on a 128^2 detector: a tenth of the SMs would hold one pattern each
        {"name": "step_128_b10", **_scan_case("step", 1024, 128, 128, 28, 32, 0, 10, "smooth_L1_loss", 1e3)},
        # the benchmark minibatch: 256 patterns of 128^2
        {"name": "step_128_b256", **_scan_case("step", 1536, 128, 128, 40, 32, 3, 256, "Poisson_likelihood_loss", 1e4)},
        # large probe, low dose
        {"name": "step_256_b64", **_scan_case("step", 2048, 256, 256, 48, 36, 4, 64, "Poisson_likelihood_loss", 1e3)},
        # the largest reconstruction: 512 patterns of 256^2 on a 4096^2 object
        {"name": "step_256_b512", **_scan_case("step", 4096, 256, 256, 96, 40, 0, 512, "Poisson_likelihood_loss", 1e3)},
        # a detector crop that is no power of two
        {"name": "step_192_b64", **_scan_case("step", 1152, 192, 192, 24, 40, 3, 64, "smooth_L1_loss", 1e3)},
        # the third loss, at the default batch, through autograd as an eager program calls it
        {"name": "loss_256_b10_fd", **_scan_case("loss", 1024, 256, 256, 20, 36, 4, 10, "FD_loss", 1e6)},
        # the residual over a stack: intensities of 512 frames, no gradient
        {"name": "intensity_256_b512", **_scan_case("intensity", 2048, 256, 256, 48, 36, 4, 512, "", 1e3)},
        # one INR minibatch's encoder on a 1024^2 object grid
        {"name": "encode_1024", "kind": "encode", "w": 1024, "h": 1024, "log2T": 19, "finest": 1024},
        # one INR minibatch's MLP on the largest object grid
        {"name": "mlp_2048", "kind": "mlp", "n": 2048 * 2048},
        # the largest object's upsampling and its adjoint
        {"name": "upsample_2048x2", "kind": "upsample", "h": 2048, "w": 2048, "s": 2},
        # a whole model evaluated on a canvas of the scan geometry (a multiple of 6, no power of two)
        {"name": "model_3000", "kind": "model", "canvas": 3000, "down": 2, "probe": 256, "log2T": 19, "finest": 1500},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("step", "step", "step", "step", "loss", "intensity", "encode", "mlp", "upsample", "model"))
    if kind in ("step", "loss", "intensity"):
        if rng.random() < 0.65:  # the square sizes detectors are binned to
            M = N = rng.choice((64, 128, 256))
            cap = 512 * 256 * 256
        else:                    # any crop
            M = rng.randint(48, 320)
            N = M if rng.random() < 0.5 else rng.randint(48, 320)
            cap = 128 * 192 * 192
        side = max(M, N)
        batch = max(1, min(_log_int(rng, 1, 512), cap // (M * N)))
        scan = max(math.ceil(math.sqrt(batch)), rng.randint(6, 40))
        jitter = rng.randint(0, 4)
        step = rng.randint(max(8, side // 8), max(9, side // 4))
        canvas = min(4096, (scan - 1) * step + side + 2 * jitter + rng.randint(0, 65))
        while (scan - 1) * step + side + 2 * jitter > canvas:
            step -= 1
        if kind == "intensity":
            return _scan_case(kind, canvas, M, N, scan, step, jitter, batch, "", 1e3)
        loss = rng.choice(LOSSES[:2] if rng.random() < 0.8 else LOSSES[2:])
        peak = 1e6 if loss == "FD_loss" else 1e3
        return _scan_case(kind, canvas, M, N, scan, step, jitter, batch, loss, peak)
    if kind == "encode":
        w, h = _log_int(rng, 64, 1024), _log_int(rng, 64, 1024)
        return {"kind": kind, "w": w, "h": h, "log2T": rng.randint(16, 19), "finest": max(64, max(w, h))}
    if kind == "mlp":
        return {"kind": kind, "n": _log_int(rng, 64 * 64, 2048 * 2048)}
    if kind == "upsample":
        s = rng.choice((1, 2, 2, 2, 3, 4))
        if rng.random() < 0.4:
            h, w = (rng.choice((64, 128, 256, 512, 1024)) for _ in range(2))
        else:
            h, w = (3 * _log_int(rng, 21, 682 // max(1, s - 1)) for _ in range(2))
        return {"kind": kind, "h": h, "w": w, "s": s}
    down = rng.choice((1, 2, 2, 3))
    canvas = 6 * _log_int(rng, 43, 250)
    return {"kind": kind, "canvas": canvas, "down": down, "probe": rng.choice((64, 96, 128, 200, 256)),
            "log2T": rng.randint(16, 19), "finest": max(64, canvas // down)}


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _gen(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed(1000003 * salt + seed)


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device=DEV, dtype=torch.float32)


def _randn(g, *shape):
    return torch.randn(shape, generator=g, device=DEV, dtype=torch.float32)


def _smooth(x, sigma):
    """Gaussian blur of width sigma px with periodic ends."""
    fy = torch.fft.fftfreq(x.shape[0], device=x.device)[:, None]
    fx = torch.fft.rfftfreq(x.shape[1], device=x.device)[None, :]
    k = torch.exp(-2.0 * (math.pi * sigma) ** 2 * (fy * fy + fx * fx))
    return torch.fft.irfft2(torch.fft.rfft2(x) * k, s=x.shape)


def _unit(x):
    return (x - x.min()) / (x.max() - x.min())


def _windows(c, g):
    """[F, 2] int32 (tlY, tlX): an n x n raster with jitter, inside the canvas."""
    n, H = c["scan"], c["canvas"]
    oy = (H - (n - 1) * c["step"] - c["M"]) // 2
    ox = (H - (n - 1) * c["step"] - c["N"]) // 2
    k = torch.arange(n, device=DEV) * c["step"]
    y, x = torch.meshgrid(k + oy, k + ox, indexing="ij")
    tl = torch.stack([y.reshape(-1), x.reshape(-1)], dim=1)
    tl = tl + torch.randint(-c["jitter"], c["jitter"] + 1, tl.shape, generator=g, device=DEV)
    lim = torch.tensor([H - c["M"], H - c["N"]], device=DEV)
    return torch.minimum(tl.clamp_min(0), lim).to(torch.int32).contiguous()


def _crop(O, tl, M, N):
    ry = tl[:, 0].long()[:, None] + torch.arange(M, device=O.device)
    rx = tl[:, 1].long()[:, None] + torch.arange(N, device=O.device)
    return O[ry[:, :, None], rx[:, None, :]]


def _intensities(O, P, tl):
    return torch.fft.fftshift(torch.fft.fft2(P * _crop(O, tl, *P.shape)), dim=(-2, -1)).abs().square()


def _scan_inputs(c, seed):
    """Object and probe estimates, the scan, the measured stack
    (Poisson counts of the true object) and one minibatch of frame ids."""
    g = _gen(seed, 1)
    H, M, N = c["canvas"], c["M"], c["N"]
    amp = 0.6 + 0.4 * _unit(_smooth(_rand(g, H, H), 4.0))
    O = torch.polar(amp, math.pi * (_unit(_smooth(_rand(g, H, H), 4.0)) - 0.5))
    yy = torch.arange(M, device=DEV, dtype=torch.float32)[:, None] - M / 2
    xx = torch.arange(N, device=DEV, dtype=torch.float32)[None, :] - N / 2
    r2 = (yy / M) ** 2 + (xx / N) ** 2
    disk = _smooth((r2 <= 0.35 ** 2).float(), 2.0).clamp_min(0.0)
    haze = 0.4 * disk.mean() * torch.complex(_randn(g, M, N), _randn(g, M, N))
    P = torch.polar(disk, 150.0 * r2) + haze  # a defocused beam with wide-angle scatter
    tl = _windows(c, g)
    ids = torch.randperm(tl.shape[0], generator=g, device=DEV)[:c["batch"]].to(torch.int32)
    Im = torch.cat([_intensities(O, P, tl[s:s + 256]) for s in range(0, tl.shape[0], 256)])
    scale = c["peak"] / Im.max()
    Im = torch.poisson(Im.mul_(scale), generator=g) if c["loss"] else None
    # Poisson refines an estimate whose fringes are right and whose power is not; the others start
    # early: the object's fine detail missing, the probe's defocus and scatter off
    if c["loss"] == "Poisson_likelihood_loss":
        P = 0.8 * P
    else:
        O = torch.complex(_smooth(O.real, 6.0), _smooth(O.imag, 6.0))
        P = torch.polar(disk, 170.0 * r2) + haze.flip(0)
    P = P * scale.sqrt()
    return O.contiguous(), P.contiguous(), tl, Im, ids


def _grid(w, h):
    """The pixel-centre coordinates of an INR's grid, in the model's order."""
    xs = torch.linspace(0.5 / w, 1 - 0.5 / w, w)
    ys = torch.linspace(0.5 / h, 1 - 0.5 / h, h)
    xv, yv = torch.meshgrid([xs, ys], indexing="ij")
    return torch.stack((yv.flatten(), xv.flatten())).t().contiguous().to(DEV)


LEVELS, BASE = 16, 16


def _per_level(finest):
    return math.exp(math.log(finest / BASE) / (LEVELS - 1))


def _encoding_config(c):
    return {"otype": "HashGrid", "n_levels": LEVELS, "n_features_per_level": 2, "log2_hashmap_size": c["log2T"],
            "base_resolution": BASE, "per_level_scale": _per_level(c["finest"])}


def _mlp_weights(mlp, g):
    """Weights as after some training: torch's initial spread."""
    with torch.no_grad():
        for name, p in mlp.named_parameters():
            if not name.endswith("omega_0"):  # those keep their starting values
                k = 1.0 / math.sqrt(32.0)
                r = (2.0 * torch.rand((*p.shape, 2), generator=g, device=DEV) - 1.0) * k
                p.copy_(torch.view_as_complex(r) * 0.7 if p.is_complex() else r[..., 0])


def _model(c, seed):
    g = _gen(seed, 5)
    m = _pkg().ComplexINRModel2D(
        c["canvas"], c["canvas"], c["down"], update_probe=True, probe_width=c["probe"], probe_height=c["probe"],
        n_levels=LEVELS, log2_hashmap_size=c["log2T"], base_resolution=BASE,
        per_level_scale=_per_level(c["finest"]), first_omega_0=10.0, hidden_omega_0=1.0,
        trainable_omega0=True).to(DEV)
    with torch.no_grad():
        for e in (m.xy_hash_encoder, m.probe_hash_encoder):
            e.params.copy_(0.05 * _randn(g, e.params.numel()))
    for mlp in (m.object_complex_mlp, m.probe_complex_mlp):
        _mlp_weights(mlp, g)
    return m


def prepare(case, seed):
    c, k = dict(case), case["kind"]
    pkg = _pkg()
    s = {"kind": k}
    if k == "step":
        O, P, tl, Im, ids = _scan_inputs(c, seed)
        s["plan"] = pkg.optics.FwdAdjPlan(O, P, tl, Im, c["loss"], int(ids.numel()))
        s["ids"] = ids
        s["plan"].set_batch(ids)
        s["plan"].capture()
    elif k == "loss":
        O, P, s["tl"], s["stack"], s["ids"] = _scan_inputs(c, seed)
        s["O"], s["P"], s["loss"] = O.requires_grad_(), P.requires_grad_(), c["loss"]
    elif k == "intensity":
        s["O"], s["P"], s["tl"], _, s["ids"] = _scan_inputs(c, seed)
    elif k == "encode":
        g = _gen(seed, 2)
        s["enc"] = pkg.Encoding(2, _encoding_config(c)).to(DEV)
        s["coords"] = _grid(c["w"], c["h"])
        with torch.no_grad():
            s["enc"].params.copy_(0.05 * _randn(g, s["enc"].params.numel()))
        s["g"] = _randn(g, 2 * LEVELS, c["w"] * c["h"]).t()  # feature-major, as the MLP's backward hands it on
    elif k == "mlp":
        g = _gen(seed, 3)
        s["mlp"] = pkg.cmlp.ComplexMLP(32, 64, 2, 1, first_omega_0=10, hidden_omega_0=1.0,
                                       trainable_omega0=True).to(DEV)
        _mlp_weights(s["mlp"], g)
        s["x"] = (0.05 * _randn(g, 32, c["n"])).t().requires_grad_()
        # the gradient of a fit: the distance from a target near the network's output
        with torch.no_grad():
            net = list(s["mlp"].parameters())
            y = torch.cat([_plain_net(x, net) for x in s["x"].split(1 << 20)])
        s["gy"] = y + 0.3 * torch.complex(_randn(g, c["n"], 1), _randn(g, c["n"], 1))
    elif k == "upsample":
        g = _gen(seed, 4)
        h, w, f = c["h"], c["w"], c["s"]
        s["x"] = torch.complex(_randn(g, h, w), _randn(g, h, w)).requires_grad_()
        s["gy"] = torch.complex(_randn(g, h * f, w * f), _randn(g, h * f, w * f))
        s["s"] = f
    else:
        s["model"] = _model(c, seed)
    return s


def run(s):
    k = s["kind"]
    pkg = _pkg()
    if k == "step":
        p = s["plan"]
        p.set_batch(s["ids"])
        p.replay()
        # the loss as a training loop keeps it (its per-pixel terms are 32-bit)
        return {"loss": p.loss_total.float(), "dO": p.dO, "dP": p.dP}
    if k == "loss":
        loss = pkg.fused_loss(s["O"], s["P"], s["tl"], s["stack"], s["loss"], batch=s["ids"])
        dO, dP = torch.autograd.grad(loss, (s["O"], s["P"]))
        return {"loss": loss.detach().float(), "dO": dO, "dP": dP}
    if k == "intensity":
        return pkg.forward_intensity(s["O"], s["P"], s["tl"], batch=s["ids"])
    if k == "encode":
        f = s["enc"](s["coords"])
        return {"features": f.detach(), "dtable": torch.autograd.grad(f, s["enc"].params, s["g"])[0]}
    if k == "mlp":
        y = s["mlp"].net(s["x"])
        ps = list(s["mlp"].parameters())
        gs = torch.autograd.grad(y, [s["x"]] + ps, s["gy"])
        return {"y": y.detach(), "dx": gs[0], "dw": list(gs[1:])}
    if k == "upsample":
        y = pkg.resample.fourier_upsample(s["x"], s["s"])
        return {"y": y.detach(), "dx": torch.autograd.grad(y, s["x"], s["gy"])[0]}
    with torch.no_grad():
        obj, probe = s["model"]()
    return {"object": obj, "probe": probe}


# --------------------------------------------------------------------------
# the least a pass moves and computes
# --------------------------------------------------------------------------
def _levels(log2T, finest):
    """(scale, vertices per axis, entries, first entry, dense) of every level."""
    b, off, out = float(np.float32(_per_level(finest))), 0, []
    for l in range(LEVELS):
        s = BASE * b ** l - 1.0
        r = int(math.ceil(s)) + 1
        dn = -(-r * r // 8) * 8
        n = min(dn, 1 << log2T)
        out.append((float(np.float32(s)), r, n, off, dn <= 1 << log2T))
        off += n
    return out


def _table_entries(log2T, finest):
    last = _levels(log2T, finest)[-1]
    return last[2] + last[3]


MLP_FLOPS = 2 * (32 * 32 + 2 * 64 * 64 + 2 * 64)  # multiply-adds of one coordinate's forward, as real matrices


def work(case):
    c, k = case, case["kind"]
    if k in ("step", "loss", "intensity"):
        px, B, H = c["M"] * c["N"], c["batch"], c["canvas"]
        fft = 5.0 * px * math.log2(px) + 6.0 * px
        span = min(H, (c["scan"] - 1) * c["step"] + max(c["M"], c["N"]) + 2 * c["jitter"])
        seen = min(B * px, span * span)
        if k == "intensity":
            return {"bytes": 8 * seen + 8 * px + 4 * B * px, "flops": B * (fft + 3.0 * px)}
        # object read where windows fall, object gradient written whole, probe both ways, counts read
        return {"bytes": 8 * seen + 8 * H * H + 16 * px + 4 * B * px, "flops": B * (2 * fft + 20.0 * px + 16.0 * px)}
    if k == "encode":
        n, e = c["w"] * c["h"], _table_entries(c["log2T"], c["finest"])
        return {"bytes": n * (8 + 8 * LEVELS + 8 * LEVELS) + 8 * e * 2, "flops": n * LEVELS * (16 + 16.0)}
    if k == "mlp":  # features and output gradient in, output and feature gradient out
        return {"bytes": c["n"] * (128 + 8 + 8 + 128), "flops": 3.0 * MLP_FLOPS * c["n"]}
    if k == "upsample":
        n, f = c["h"] * c["w"], c["s"]
        N = n * f * f
        one = 5.0 * n * math.log2(max(2, n)) + 5.0 * N * math.log2(max(2, N))
        return {"bytes": 2 * (8 * n + 8 * N), "flops": 2 * one}
    d = c["canvas"] // c["down"]
    n, N, p = d * d, (d * c["down"]) ** 2, c["probe"] ** 2
    e = _table_entries(c["log2T"], c["finest"])
    touched = min(e, 4 * LEVELS * n) + min(e, 4 * LEVELS * p)
    up = 5.0 * n * math.log2(max(2, n)) + 5.0 * N * math.log2(max(2, N))
    return {"bytes": 8 * (n + p) + 8 * touched + 8 * (N + p), "flops": (n + p) * (MLP_FLOPS + 16.0 * LEVELS) + up}


# --------------------------------------------------------------------------
# the same in 64 bits
# --------------------------------------------------------------------------
def _loss_grad(I, Im, name):
    """(sum over patterns of the mean loss, dL/dI) for a block of patterns, torch autograd in 64 bits."""
    I = I.detach().requires_grad_()
    if name == "smooth_L1_loss":
        per = torch.nn.functional.smooth_l1_loss(I, Im, reduction="none")
    elif name == "Poisson_likelihood_loss":
        per = I - Im * torch.log(I + 1e-8)
    else:
        d = torch.sqrt(Im + 1e-8) - torch.sqrt(I + 1e-8)
        rx = torch.roll(d, -1, dims=-1) - d
        ry = torch.roll(d, -1, dims=-2) - d
        per = torch.sqrt(rx * rx + ry * ry + 1e-8)
    loss = per.mean(dim=(-2, -1)).sum()
    return loss.detach(), torch.autograd.grad(loss, I)[0]


def _exact_scan(c, seed):
    O, P, tl, Im, ids = _scan_inputs(c, seed)
    O, P = O.to(torch.complex128), P.to(torch.complex128)
    M, N = P.shape
    if c["kind"] == "intensity":
        return torch.cat([_intensities(O, P, tl[ids[s:s + 64].long()]) for s in range(0, c["batch"], 64)])
    dO, dP = torch.zeros_like(O), torch.zeros_like(P)
    total = torch.zeros((), dtype=torch.float64, device=O.device)
    for s in range(0, c["batch"], 64):
        i = ids[s:s + 64].long()
        w = tl[i]
        win = _crop(O, w, M, N)
        F = torch.fft.fftshift(torch.fft.fft2(P * win), dim=(-2, -1))
        loss, gI = _loss_grad(F.abs().square(), Im[i].double(), c["loss"])
        total += loss
        gpsi = torch.fft.ifft2(torch.fft.ifftshift(2.0 * gI * F, dim=(-2, -1)), norm="forward")
        dP += (gpsi * win.conj()).sum(0)
        gO = gpsi * P.conj()
        for b, (y, x) in enumerate(w.tolist()):
            dO[y:y + M, x:x + N] += gO[b]
    return {"loss": total, "dO": dO, "dP": dP}


def _corners(x, level):
    """(entry, weight) of the four corners of coordinates x [n, 2], 64-bit weights."""
    s, r, n, off, dense = level
    p = x * s + 0.5
    i = p.floor()
    f = p - i
    ix, iy = i[:, 0].long(), i[:, 1].long()
    for dx in (0, 1):
        for dy in (0, 1):
            cx, cy = ix + dx, iy + dy
            e = (cx + cy * r) % n if dense else ((cx ^ (cy * 2654435761 & 0xFFFFFFFF)) & (n - 1))
            yield off + e, (f[:, 0] if dx else 1 - f[:, 0]) * (f[:, 1] if dy else 1 - f[:, 1])


def _exact_features(x, table, log2T, finest):
    out = torch.zeros(x.shape[0], 2 * LEVELS, dtype=torch.float64, device=x.device)
    for l, lev in enumerate(_levels(log2T, finest)):
        for e, w in _corners(x, lev):
            out[:, 2 * l:2 * l + 2] += w[:, None] * table[e]
    return out


def _plain_net(x, net):
    """ComplexMLP.net in plain torch; net: its eleven parameters in order."""
    w1, W1, b1, w2, W2, b2, w3, W3, b3, Wo, bo = net
    h = torch.exp(1j * w1 * (x @ W1.t() + b1).to(Wo.dtype))
    h = torch.exp(1j * w2 * (h @ W2.t() + b2))
    h = torch.exp(1j * w3 * (h @ W3.t() + b3))
    return h @ Wo.t() + bo


def _net64(mlp):
    wide = {torch.float32: torch.float64, torch.complex64: torch.complex128}
    return [p.detach().to(wide[p.dtype]).requires_grad_() for p in mlp.parameters()]


def _up64(x, s):
    h, w = x.shape
    F = torch.fft.fftshift(torch.fft.fft2(x))
    ph, pw = (h * s - h) // 2, (w * s - w) // 2
    F = torch.nn.functional.pad(F, (pw, w * s - w - pw, ph, h * s - h - ph))
    return torch.fft.ifft2(torch.fft.ifftshift(F)) * s ** 2


def exact(case, seed):
    c, k = case, case["kind"]
    if k in ("step", "loss", "intensity"):
        return _exact_scan(c, seed)
    if k == "encode":
        s = prepare(c, seed)
        x, table = s["coords"].double(), s["enc"].params.detach().double().view(-1, 2)
        g = s["g"].double()
        d = torch.zeros_like(table)
        for l, lev in enumerate(_levels(c["log2T"], c["finest"])):
            for e, w in _corners(x, lev):
                d.index_add_(0, e, w[:, None] * g[:, 2 * l:2 * l + 2])
        return {"features": _exact_features(x, table, c["log2T"], c["finest"]), "dtable": d.view(-1)}
    if k == "mlp":
        s = prepare(c, seed)
        net = _net64(s["mlp"])
        y, dx, dw = [], [], None
        for i in range(0, c["n"], 1 << 18):
            x = s["x"][i:i + (1 << 18)].detach().double().requires_grad_()
            out = _plain_net(x, net)
            gs = torch.autograd.grad(out, [x] + net, s["gy"][i:i + (1 << 18)].to(torch.complex128))
            y.append(out.detach())
            dx.append(gs[0])
            dw = [a + b for a, b in zip(dw, gs[1:])] if dw else list(gs[1:])
        return {"y": torch.cat(y), "dx": torch.cat(dx), "dw": dw}
    if k == "upsample":
        s = prepare(c, seed)
        x = s["x"].detach().to(torch.complex128).requires_grad_()
        y = _up64(x, c["s"])
        return {"y": y.detach(), "dx": torch.autograd.grad(y, x, s["gy"].to(torch.complex128))[0]}
    m = _model(c, seed)
    out = []
    with torch.no_grad():
        for enc, mlp, coords in ((m.xy_hash_encoder, m.object_complex_mlp, m.xy_coords),
                                 (m.probe_hash_encoder, m.probe_complex_mlp, m.probe_coords)):
            table, net = enc.params.double().view(-1, 2), _net64(mlp)
            out.append(torch.cat([_plain_net(_exact_features(x.double(), table, c["log2T"], c["finest"]), net)
                                  for x in coords.split(1 << 19)]))
        d = c["canvas"] // c["down"]
        return {"object": _up64(out[0].view(d, d), c["down"]), "probe": out[1].view(c["probe"], c["probe"])}
