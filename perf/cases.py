"""The calls of this library that are timed, with the sizes they are made at.

A case is one call (or one short sequence of calls) that an imaging program
makes through the public entry points: the stateless `vis2dirty` and
`dirty2vis` (a plan and a pass on CUDA tensors, or NumPy arrays through
`rang._core`), the passes of a kept plan (autograd, the fused residual, a few
FISTA iterations), the proposal network's inference and training step, and
the imaging weights. Every observation is the synthetic MeerKAT-shaped one of
`rang.synth`; its visibilities are point sources plus noise, made on the GPU
from the seed.
"""

import math
import sys
from pathlib import Path

import numpy as np
import torch
import torch.nn.functional as F

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "rang-core_b200"))

from rang import fista, gridder, learned, synth, weighting, wgrid_torch  # noqa: E402

DEV = "cuda"

# What a gridding case leaves out: 64 antennas (2016 baselines), 8 s
# integrations, no dropped rows, float32, epsilon 1e-5, w-gridding, no
# weights, no flags, device tensors.
GRID = {"nant": 64, "ntime": 128, "nchan": 64, "drop": 0, "nx": 1024, "ny": 1024, "cell": 1.5, "eps": 1e-5,
        "double": False, "wgt": "none", "flag": 0.0, "wgridding": True, "host": False}


def listed():
    return [
        # A snapshot: two integrations of 17 channels imaged at low
        # resolution, as a real-time monitor or a self-calibration loop does
        # call after call. Latency and launches count.
        {"name": "dirty_snapshot_69k_256", "kind": "dirty", "ntime": 2, "nchan": 17, "nx": 256, "ny": 256, "cell": 2.0,
         "wgt": "f32"},
        # An ordinary observation through the host-array call, the drop-in
        # for the reference's Python function, from NumPy arrays.
        {"name": "dirty_host_16m_1024", "kind": "dirty", "host": True},
        # The same observation in double precision at the tightest accuracy
        # of the benchmark, imaged and predicted.
        {"name": "dirty_f64_16m_1024", "kind": "dirty", "eps": 1e-7, "double": True},
        {"name": "predict_f64_16m_1024", "kind": "predict", "eps": 1e-7, "double": True},
        # The headline round trip: 1.06 G visibilities, a fifth flagged, 4096^2.
        {"name": "roundtrip_1g_4096", "kind": "roundtrip", "ntime": 512, "nchan": 1024, "nx": 4096, "ny": 4096,
         "cell": 1.0, "flag": 0.2},
        # A ragged observation at the widest single-precision support: an odd
        # channel count, rows missing at the end, a rectangular image, weights.
        {"name": "roundtrip_ragged_60m_eps6", "kind": "roundtrip", "ntime": 61, "nchan": 487, "drop": 331,
         "nx": 1998, "ny": 2310, "cell": 1.7, "eps": 1e-6, "wgt": "f32", "flag": 0.1},
        # The differentiable degridder, forward and backward, on a kept plan.
        {"name": "autograd_132m_2048", "kind": "autograd", "ntime": 256, "nchan": 256, "nx": 2048, "ny": 2048},
        # A deconvolution's major cycle on a kept plan: the fused residual.
        {"name": "residual_66m_2048", "kind": "residual", "nchan": 256, "nx": 2048, "ny": 2048, "wgt": "f32"},
        # FISTA iterations through the exact Gram operator.
        {"name": "fista_66m_2048", "kind": "fista", "nchan": 256, "nx": 2048, "ny": 2048, "iterations": 3},
        # The proposal network over a 2048^2 residual (81 overlapping patches).
        {"name": "propose_2048", "kind": "propose", "npix": 2048},
        # One training step's gradients at the training batch.
        {"name": "train_b16_256", "kind": "train", "batch": 16, "height": 256, "width": 256},
        # Briggs weights of an ordinary observation on host arrays.
        {"name": "weights_16m_briggs", "kind": "weights", "ntime": 128, "nchan": 64, "npix": 1024, "cell": 1.5,
         "robust": 0.5},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["dirty", "dirty", "predict", "predict", "roundtrip", "autograd", "residual", "fista", "propose",
                       "train", "weights"])
    if kind == "propose":
        return {"kind": kind, "npix": rng.randint(256, 2048)}
    if kind == "train":
        return {"kind": kind, "batch": rng.randint(1, 16), "height": 8 * rng.randint(8, 32),
                "width": 8 * rng.randint(8, 32)}
    nchan = int(_log(rng, 1, 1024))
    if kind == "weights":
        ntime = max(1, int(_log(rng, 1e5, 6e7) / (2016 * nchan)))
        return {"kind": kind, "ntime": min(ntime, 1024), "nchan": nchan, "npix": 2 * int(_log(rng, 128, 2048)),
                "cell": round(rng.uniform(0.8, 2.2), 3), "robust": round(rng.uniform(-1.0, 1.0), 2)}
    c = {"kind": kind, "nchan": nchan}
    c["double"] = kind in ("dirty", "predict", "roundtrip") and rng.random() < 0.3
    c["nant"] = rng.choice([16, 33, 64])
    nbl = c["nant"] * (c["nant"] - 1) // 2
    if c["double"]:
        c["eps"] = float("%.2g" % _log(rng, 1e-9, 1e-4))
        most = 2e6 if c["eps"] < 1e-7 else 3e7
    else:
        c["eps"] = float("%.2g" % _log(rng, 1e-6, 1e-3))
        most = 1.5e8
    c["ntime"] = max(1, min(2048, int(_log(rng, 3e4, most) / (nbl * nchan))))
    c["drop"] = rng.randint(0, nbl // 2)
    c["nx"], c["ny"] = (2 * int(_log(rng, 64, 2048)) for _ in range(2))
    c["cell"] = round(rng.uniform(0.8, 2.2), 3)
    c["wgt"] = rng.choice(["none", "f32", "f64"] if c["double"] else ["none", "f32"])
    c["flag"] = rng.choice([0.0, round(rng.uniform(0.01, 0.6), 2)])
    c["wgridding"] = rng.random() < 0.85
    if kind in ("dirty", "predict"):
        c["host"] = rng.random() < 0.25
    if kind == "fista":
        c["iterations"] = rng.randint(1, 4)
    return c


# ------------------------------------------------------------------ observations


def _grid_case(case):
    c = dict(GRID)
    c.update(case)
    return c


def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _observation(c, seed):
    """(uvw (nrow, 3) CUDA float64, freq): the field's declination follows the seed."""
    dec = -30.0 + float(np.random.default_rng(seed).uniform(-1.0, 1.0))
    uvw = synth.uvw_tracks(nant=c["nant"], ntime=c["ntime"], tint=8.0, dec_deg=dec)
    uvw = uvw[:max(1, uvw.shape[0] - c["drop"])]
    return torch.from_numpy(np.ascontiguousarray(uvw)).to(DEV), synth.channels(c["nchan"])


def _sources(c, seed, n=8):
    """n sources on pixel centres inside the field: pixel rows and columns, fluxes."""
    rng = np.random.default_rng([seed, 1])
    ix = rng.integers(c["nx"] // 8, c["nx"] - c["nx"] // 8, n)
    iy = rng.integers(c["ny"] // 8, c["ny"] - c["ny"] // 8, n)
    return ix, iy, 10.0 ** rng.uniform(-2.0, 0.0, n)


def _visibilities(c, seed, uvw, freq, g, sigma=0.1):
    """The sources' visibilities plus complex noise of `sigma` per component, complex64."""
    nrow, nchan = uvw.shape[0], len(freq)
    foc = torch.from_numpy(np.asarray(freq) / synth.C_LIGHT).to(DEV)
    cell = c["cell"] * synth.ARCSEC
    vis = torch.empty((nrow, nchan), dtype=torch.complex64, device=DEV)
    step = max(1, (1 << 25) // nchan)
    ix, iy, flux = _sources(c, seed)
    for a in range(0, nrow, step):
        b = min(nrow, a + step)
        part = torch.randn((b - a, nchan), dtype=torch.complex64, device=DEV, generator=g) * (sigma * math.sqrt(2.0))
        for x, y, f in zip(ix, iy, flux):
            l, m = (x - c["nx"] // 2) * cell, (y - c["ny"] // 2) * cell
            n = math.sqrt(1.0 - l * l - m * m) - 1.0 if c["wgridding"] else 0.0
            metres = uvw[a:b, 0] * l + uvw[a:b, 1] * m + uvw[a:b, 2] * n
            turns = metres[:, None] * foc
            turns = (turns - torch.round(turns)).float() * (-2.0 * math.pi)
            part += torch.polar(torch.full_like(turns, float(f)), turns)
        vis[a:b] = part
    return vis


def _per_visibility(shape, g, make):
    """One float per visibility, made in blocks of rows."""
    step = max(1, (1 << 27) // shape[1])
    parts = [make(torch.rand((min(shape[0], a + step) - a, shape[1]), device=DEV, generator=g))
             for a in range(0, shape[0], step)]
    return torch.cat(parts) if len(parts) > 1 else parts[0]


def _weights_and_flags(c, shape, g):
    wgt = mask = None
    if c["wgt"] != "none":
        wgt = _per_visibility(shape, g, lambda r: r + 0.5)
        if c["wgt"] == "f64":
            wgt = wgt.double()
    if c["flag"] > 0:
        mask = _per_visibility(shape, g, lambda r: (r >= c["flag"]).to(torch.uint8))
    return wgt, mask


def _model(c, seed, g, real):
    """A model image: the sources on their pixels over a faint random background."""
    img = torch.randn((c["nx"], c["ny"]), device=DEV, generator=g, dtype=torch.float64) * 1e-4
    ix, iy, flux = _sources(c, seed)
    img.index_put_((torch.from_numpy(ix).to(DEV), torch.from_numpy(iy).to(DEV)),
                   torch.from_numpy(0.9 * flux).to(DEV), accumulate=True)
    return img.to(real)


def _options(c):
    cell = c["cell"] * synth.ARCSEC
    kw = {"pixsize_x": cell, "pixsize_y": cell, "epsilon": c["eps"]}
    if not c["wgridding"]:
        kw["do_wgridding"] = False
    return kw


# ------------------------------------------------------------------ the network


def _network_inputs(case, seed):
    """A residual image (or batch of patches) in units of the PSF peak, targets, and a PSF patch."""
    g = _generator(seed)
    shape = (case["npix"], case["npix"]) if case["kind"] == "propose" else (case["batch"], case["height"], case["width"])
    resid = torch.randn(shape, device=DEV, generator=g) * 0.02
    bright = torch.rand(shape, device=DEV, generator=g) > 0.9995
    resid = resid + bright * torch.rand(shape, device=DEV, generator=g)
    target = bright * torch.rand(shape, device=DEV, generator=g)
    h, w = (learned.PATCH, learned.PATCH) if case["kind"] == "propose" else shape[1:]
    y = (torch.arange(h, device=DEV) - h // 2)[:, None].float()
    x = (torch.arange(w, device=DEV) - w // 2)[None, :].float()
    r = torch.sqrt(x * x + y * y)
    psf = torch.exp(-r * r / 18.0) + 0.05 * torch.cos(r / 3.0) / (1.0 + r / 8.0)
    return resid, target.float(), (psf / psf[h // 2, w // 2]).contiguous()


# ------------------------------------------------------------------ the cases


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("propose", "train"):
        resid, target, psf = _network_inputs(case, seed)
        net = learned.UNet(DEV, seed=seed)
        s = {"kind": kind, "net": net, "resid": resid, "target": target, "psf": psf}
        if kind == "propose":
            s["proposer"] = learned.Proposer(net, case["npix"])
        else:
            s["ws"] = learned.Workspace(net, case["batch"], case["height"], case["width"], training=True)
            s["offsets"] = torch.arange(case["batch"], device=DEV) * (case["height"] * case["width"])
        return s
    if kind == "weights":
        c = dict(case, nant=64, drop=0)
        uvw, freq = _observation(c, seed)
        g = _generator(seed)
        w = _per_visibility((uvw.shape[0], len(freq)), g, lambda r: torch.where(r < 0.1, 0.0, r + 0.5))
        size = weighting.padded_size(case["npix"])
        return {"kind": kind, "uvw": uvw.cpu().numpy(), "wavelength": weighting.wavelengths(freq),
                "w": w.cpu().numpy(), "selected": np.ones(uvw.shape[0], np.uint8),
                "weighting": weighting.ImagingWeights(size, size, case["cell"] * synth.ARCSEC, mode="briggs",
                                                      robust=case["robust"])}
    c = _grid_case(case)
    uvw, freq = _observation(c, seed)
    g = _generator(seed)
    shape = (uvw.shape[0], len(freq))
    real = torch.float64 if c["double"] else torch.float32
    s = {"kind": kind, "host": c["host"], "uvw": uvw, "freq": freq, "options": _options(c),
         "size": {"npix_x": c["nx"], "npix_y": c["ny"]}, "single": not c["double"], "vis": None, "image": None}
    s["wgt"], s["mask"] = _weights_and_flags(c, shape, g)
    if kind in ("dirty", "roundtrip", "residual", "fista"):
        vis = _visibilities(c, seed, uvw, freq, g)
        s["vis"] = vis.to(torch.complex128) if c["double"] else vis
    if kind in ("predict", "roundtrip", "residual"):
        s["image"] = _model(c, seed, g, real)
    if kind == "autograd":
        s["image"] = torch.randn((c["nx"], c["ny"]), device=DEV, generator=g).requires_grad_()
        s["upstream"] = torch.randn(shape, dtype=torch.complex64, device=DEV, generator=g)
    if kind in ("autograd", "residual", "fista"):  # a kept plan
        s["plan"] = wgrid_torch.DevicePlan(uvw, freq, wgt=s["wgt"], mask=s["mask"], single=True, **s["size"],
                                           **s["options"])
        if kind == "fista":
            s["dirty"], s["q"] = s["plan"].residual(s["vis"], s["wgt"])
            top, _ = fista.power_iteration(lambda x: s["plan"].gram(x, s["wgt"]), s["plan"].shape, DEV,
                                           max_iterations=4)
            s["step"], s["lam"], s["iterations"] = 0.8 / top, 1e-4 * float(s["dirty"].max()), c["iterations"]
            s["vis"] = None
    if c["host"]:
        for k in ("uvw", "vis", "image", "wgt", "mask"):
            if s[k] is not None:
                s[k] = s[k].cpu().numpy()
    return s


def run(s):
    kind = s["kind"]
    if kind == "propose":
        return s["proposer"](s["resid"], s["psf"], 1.0)
    if kind == "train":
        net, ws, w = s["net"], s["ws"], s["ws"].width
        net.zero_grad()
        ws.loss.zero_()
        net.pack(ws, s["resid"], s["offsets"], w, s["psf"], w)
        net.forward(ws)
        net.loss_and_grad(ws, s["target"], s["offsets"], w)
        net.backward(ws)
        return {"y": ws.y, "loss": ws.loss, "grad": net.grad}
    if kind == "weights":
        r = s["weighting"](s["uvw"], s["wavelength"], s["w"], s["selected"])
        return {"weights": r.weights, "sums": [r.visibility_weight_sum, r.total_weight, r.max_gridded_weight],
                "count": r.count}
    if kind == "autograd":
        y = wgrid_torch.degrid(s["image"], s["plan"], s["wgt"])
        (grad,) = torch.autograd.grad(y, s["image"], s["upstream"])
        return {"vis": y.detach(), "grad": grad}
    if kind == "residual":
        image, misfit = s["plan"].residual(s["vis"], s["wgt"], model=s["image"])
        return {"image": image, "misfit": misfit}
    if kind == "fista":
        plan, wgt = s["plan"], s["wgt"]
        r = fista.solve(lambda x: plan.gram(x, wgt), s["dirty"], s["lam"], s["step"], s["iterations"], q0=0.5 * s["q"])
        return {"x": r.x, "gx": r.gx, "misfits": r.misfits}
    out = {}
    arrays = {"uvw": s["uvw"], "freq": s["freq"], "wgt": s["wgt"], "mask": s["mask"]}
    if s["host"]:
        if kind == "dirty":
            out["image"] = gridder.vis2dirty(vis=s["vis"], **arrays, **s["size"], **s["options"])
        else:
            out["vis"] = gridder.dirty2vis(dirty=s["image"], **arrays, **s["options"])
        return out
    if kind in ("dirty", "roundtrip"):
        plan = wgrid_torch.DevicePlan(**arrays, vis=s["vis"], single=s["single"], **s["size"], **s["options"])
        out["image"] = plan.grid(s["vis"], s["wgt"], scanned=True)
        plan.close()
    if kind in ("predict", "roundtrip"):
        plan = wgrid_torch.DevicePlan(**arrays, single=s["single"], **s["size"], **s["options"])
        out["vis"] = plan.degrid(s["image"], s["wgt"])
        plan.close()
    return out


def work(case):
    """Each input read once and each output written once; per visibility and
    direction S^3 complex multiply-adds with real taps (4 S^3 operations, S
    the support), per plane and direction one FFT of the oversampled grid."""
    kind = case["kind"]
    if kind == "propose":
        n = case["npix"]
        patches = len(learned.tiles(n)) ** 2
        return {"bytes": 8 * n * n + 2 * 1.95e6, "flops": patches * learned.flops()}
    if kind == "train":
        b, h, w = case["batch"], case["height"], case["width"]
        return {"bytes": 12 * b * h * w + 6 * 1.95e6, "flops": b * learned.flops(h, w, training=True)}
    if kind == "weights":
        n = 2016 * case["ntime"] * case["nchan"]
        return {"bytes": 8 * n + 24 * 2016 * case["ntime"], "flops": 12 * n}
    c = _grid_case(case)
    nrow = max(1, c["nant"] * (c["nant"] - 1) // 2 * c["ntime"] - c["drop"])
    n, pix = nrow * c["nchan"], c["nx"] * c["ny"]
    real = 8 if c["double"] else 4
    supp = max(4, math.ceil(-math.log10(c["eps"])) + 1)
    planes = supp if c["wgridding"] else 1
    per_pass = 4 * supp ** 2 * planes * n * (1.0 - c["flag"])
    per_pass += planes * 5 * 5.3 * pix * math.log2(5.3 * pix)
    per_vis = {"none": 0, "f32": 4, "f64": 8}[c["wgt"]] + (1 if c["flag"] > 0 else 0)
    one = 24 * nrow + n * per_vis + n * 2 * real + pix * real  # one stateless direction
    if kind in ("dirty", "predict"):
        return {"bytes": one, "flops": per_pass}
    if kind in ("roundtrip", "autograd"):
        return {"bytes": 2 * one, "flops": 2 * per_pass}
    if kind == "residual":
        return {"bytes": one + pix * real, "flops": 2 * per_pass}
    applies = c["iterations"] + 1
    return {"bytes": applies * (n * per_vis + 6 * pix * real), "flops": applies * 2 * per_pass}


def tolerance(case):
    kind = case["kind"]
    # bfloat16 activations and gradients through 14 layers.
    if kind == "propose":
        return {"rel": 1e-2, "max": 0.3}
    if kind == "train":
        return {"rel": 3e-2, "max": 0.9}
    if kind == "weights":
        return {"rel": 1e-6, "max": 1e-5, "differ": 0.0}
    c = _grid_case(case)
    if c["double"]:
        return {"rel": 1e-11, "max": 1e-9}
    return {"rel": 1e-5, "max": 1e-3}


# ------------------------------------------------------------------ in 64 bits


def _direct(c, s, direction):
    """The direct sum over visibilities and pixels in float64 (the operator
    that vis2dirty and dirty2vis approximate to epsilon), or None when it
    would take long."""
    uvw = torch.as_tensor(s["uvw"], device=DEV)
    nrow, nchan, pix = uvw.shape[0], len(s["freq"]), c["nx"] * c["ny"]
    if nrow * nchan * pix > 1.5e11:
        return None
    foc = torch.from_numpy(np.asarray(s["freq"]) / synth.C_LIGHT).to(DEV)
    w = torch.ones((nrow, nchan), dtype=torch.float64, device=DEV)
    if s["wgt"] is not None:
        w = torch.as_tensor(s["wgt"], device=DEV).double()
    if s["mask"] is not None:
        w = w * torch.as_tensor(s["mask"], device=DEV)
    cell = c["cell"] * synth.ARCSEC
    l = ((torch.arange(c["nx"], device=DEV) - c["nx"] // 2) * cell)[:, None].double()
    m = ((torch.arange(c["ny"], device=DEV) - c["ny"] // 2) * cell)[None, :].double()
    n = torch.sqrt(1.0 - l * l - m * m) - 1.0 if c["wgridding"] else torch.zeros_like(l * m)
    lmn = torch.stack([(l + 0 * m).reshape(-1), (m + 0 * l).reshape(-1), n.reshape(-1)])
    coords = (uvw[:, None, :] * foc[None, :, None]).reshape(-1, 3)
    w = w.reshape(-1)
    step = max(1, int(2e8 // pix))
    if direction == "dirty":
        v = torch.as_tensor(s["vis"], device=DEV).reshape(-1).to(torch.complex128) * w
        out = torch.zeros(pix, dtype=torch.float64, device=DEV)
        for a in range(0, coords.shape[0], step):
            turns = coords[a:a + step] @ lmn
            turns = (turns - torch.round(turns)).mul_(2.0 * math.pi)
            out += v[a:a + step].real @ torch.cos(turns) - v[a:a + step].imag @ torch.sin(turns)
        return out.reshape(c["nx"], c["ny"])
    img = torch.as_tensor(s["image"], device=DEV).detach().double().reshape(-1)
    out = torch.empty(coords.shape[0], dtype=torch.complex128, device=DEV)
    for a in range(0, coords.shape[0], step):
        turns = coords[a:a + step] @ lmn
        turns = (turns - torch.round(turns)).mul_(2.0 * math.pi)
        out[a:a + step] = torch.complex(torch.cos(turns) @ img, -(torch.sin(turns) @ img))
    return (out * w).reshape(nrow, nchan)


def _exact_network(case, s):
    """The network on its bfloat16 weights and packed inputs, in float64."""
    net = s["net"]
    p = {}
    for key, (o, shape) in net.slots.items():
        buf = net.wb if key.endswith(".w") and len(shape) == 3 else net.master
        t = buf[o:o + int(np.prod(shape))].double().reshape(shape)
        if len(shape) == 3:
            t = t.reshape(shape[0], 3, 3, shape[2]).permute(0, 3, 1, 2).contiguous()
        p[key] = t.requires_grad_(case["kind"] == "train")

    def conv(x, name):
        return F.relu(F.conv2d(x, p[name + ".w"], p[name + ".b"], padding=1))

    def up(x):
        return F.interpolate(x, scale_factor=2, mode="nearest")

    def forward(resid, psf):
        x = torch.zeros((resid.shape[0], learned.IN_CHANNELS) + tuple(resid.shape[1:]), dtype=torch.float64, device=DEV)
        x[:, 0] = resid.bfloat16().double()
        x[:, 1] = psf.bfloat16().double()
        e1 = conv(conv(x, "enc1a"), "enc1b")
        e2 = conv(conv(F.avg_pool2d(e1, 2), "enc2a"), "enc2b")
        e3 = conv(conv(F.avg_pool2d(e2, 2), "enc3a"), "enc3b")
        mid = conv(conv(F.avg_pool2d(e3, 2), "mid_a"), "mid_b")
        d3 = conv(conv(torch.cat([up(mid), e3], 1), "dec3a"), "dec3b")
        d2 = conv(conv(torch.cat([up(d3), e2], 1), "dec2a"), "dec2b")
        d1 = conv(conv(torch.cat([up(d2), e1], 1), "dec1a"), "dec1b")
        return torch.einsum("bchw,c->bhw", d1, p["head.w"]) + p["head.b"]

    if case["kind"] == "propose":
        n, patch = case["npix"], learned.PATCH
        out = torch.empty((n, n), dtype=torch.float64, device=DEV)
        ax = learned.tiles(n)
        with torch.no_grad():
            for a, a0, a1 in ax:
                y = forward(torch.stack([s["resid"][a:a + patch, b:b + patch] for b, _, _ in ax]), s["psf"])
                for k, (b, b0, b1) in enumerate(ax):
                    out[a + a0:a + a1, b + b0:b + b1] = y[k, a0:a1, b0:b1]
        return out
    y = forward(s["resid"], s["psf"])
    loss = ((y - s["target"].double()) ** 2).mean()
    loss.backward()
    grad = torch.zeros(net.size, dtype=torch.float64, device=DEV)
    for key, (o, shape) in net.slots.items():
        gr = p[key].grad
        if len(shape) == 3:
            gr = gr.permute(0, 2, 3, 1).reshape(shape)
        grad[o:o + gr.numel()] = gr.reshape(-1)
    return {"y": y.detach().reshape(-1), "loss": loss.detach().reshape(1), "grad": grad}


def _exact_weights(case, s):
    """Briggs weights with the rank filter (3, 16), the half-plane grid's sums in float64."""
    k = s["weighting"]
    width, height = k.grid_shape()
    uvw = torch.from_numpy(s["uvw"]).to(DEV)
    lam = torch.from_numpy(s["wavelength"]).to(DEV)
    w = torch.from_numpy(s["w"]).to(DEV).double()
    u, v = uvw[:, 0:1] / lam, uvw[:, 1:2] / lam
    u, v = torch.where(v < 0, -u, u), v.abs()
    x = torch.floor(u * width * k.pixel_scale + width // 2).long()
    y = torch.floor(v * height * k.pixel_scale).long()
    inside = (x >= 0) & (x < width) & (y < height // 2)
    at = torch.where(inside, x + y * width, 0)
    grid = torch.zeros(width * (height // 2), dtype=torch.float64, device=DEV)
    grid.index_add_(0, at.reshape(-1), torch.where(inside, w, 0.0).reshape(-1))
    scale = (5.0 * 10.0 ** -k.robust) ** 2 / ((grid * grid).sum() / grid.sum())
    full = torch.where(grid != 0, 1.0 / (1.0 + grid * scale), 0.0).reshape(height // 2, width)
    level, cells = k.rank_filter
    d = cells // 2

    def window(t):
        t = F.pad(t.cumsum(0), (0, 0, 1, 0))
        r = torch.arange(height // 2, device=DEV)
        t = t[(r + d).clamp(max=height // 2)] - t[(r - d).clamp(min=0)]
        t = F.pad(t.cumsum(1), (1, 0))
        r = torch.arange(width, device=DEV)
        return t[:, (r + d).clamp(max=width)] - t[:, (r - d).clamp(min=0)]

    mean = window(full) / window((full != 0).double()).clamp(min=1.0)
    full = torch.where((full != 0) & (full > mean * level), mean * level, full).reshape(-1)
    out = torch.where(inside, full[at], 0.0)
    both = w * out
    return {"weights": out, "sums": [float((w * (both != 0)).sum()), float(both.sum()), float(both.max())],
            "count": None}


def exact(case, seed):
    kind = case["kind"]
    s = prepare(case, seed)
    if kind in ("propose", "train"):
        return _exact_network(case, s)
    if kind == "weights":
        return _exact_weights(case, s)
    c = _grid_case(case)
    if kind == "fista":
        return None
    if kind == "dirty":
        image = _direct(c, s, "dirty")
        return None if image is None else {"image": image}
    vis = _direct(c, s, "predict")
    if vis is None:
        return None
    if kind == "predict":
        return {"vis": vis}
    if kind == "roundtrip":
        return {"image": _direct(c, s, "dirty"), "vis": vis}
    if kind == "autograd":
        grad = _direct(c, dict(s, vis=s["upstream"]), "dirty")
        return {"vis": vis, "grad": grad}
    # The residual: the prediction has no weights, the active set and the sums do.
    bare = _direct(c, dict(s, wgt=None), "predict")
    diff = s["vis"].to(torch.complex128) - bare
    w = torch.ones(diff.shape, dtype=torch.float64, device=DEV) if s["wgt"] is None else s["wgt"].double()
    if s["mask"] is not None:
        w = w * s["mask"]
    return {"image": _direct(c, dict(s, vis=diff), "dirty"), "misfit": (w * diff.abs() ** 2).sum()}
