"""The work that programs have this package do, as cases that can be timed and compared.

Each case is one call a user makes, on inputs made from a seed: a device plane rendered by either
integrator, a whole host image rendered to u8, a batch of uneven images, and the surrogate's layer,
inference and gradient passes.  Sizes and parameters are those of the benchmark workloads and of the
command-line defaults, with odd sizes among them; `draw` spreads the same parameters over their ranges.
"""
from __future__ import annotations

import math
import os

import numpy as np
import torch

import film_grain_gb300 as fg
from film_grain_gb300 import surrogate as sg

LIGHT = {"ramp": 1.0, "blobs": 0.55}  # mean of -ln(1 - u) over the two input families, roughly


# ---------------------------------------------------------------------- cases
def _plane(kind, name, w, h, radius, n, source, sd=0.0, zoom=1.0, seed=42):
    return {"name": name, "kind": kind, "w": w, "h": h, "radius": radius, "sd": sd, "n": n, "zoom": zoom,
            "source": source, "stream": seed}


def _image(name, w, h, radius, n, color, algo, source, sd=0.0, zoom=1.0, roi=False):
    return {"name": name, "kind": "image", "w": w, "h": h, "radius": radius, "sd": sd, "n": n, "zoom": zoom,
            "source": source, "stream": 42, "color": color, "algo": algo, "roi": roi}


def _net(name, kind, nb, h, w):
    return {"name": name, "kind": kind, "nb": nb, "h": h, "w": w}


def listed():
    return [
        # a thumbnail with the command line's defaults (radius 0.10, 32 samples): latency of one call
        _plane("pixel", "pixel_thumb_96x64", 96, 64, 0.10, 32, "ramp"),
        # the 256^2 luma pixel-wise benchmark: a viewer's preview of a plane
        _plane("pixel", "pixel_ramp_256", 256, 256, 0.12, 64, "ramp"),
        # fine grain with few samples on an odd size: the per-sample kernel's range
        _plane("pixel", "pixel_fine_1021x763", 1021, 763, 0.025, 64, "blobs"),
        # the large frame's grain (log-normal 0.025 / 0.01, 256 samples) on a megapixel plane
        _plane("pixel", "pixel_lognormal_1024", 1024, 1024, 0.025, 256, "blobs", sd=0.01),
        # one plane of the grain-wise benchmark: log-normal 0.05 / 0.025, 128 samples, 2x output
        _plane("grain", "grain_lognormal_1024_x2", 1024, 1024, 0.05, 128, "blobs", sd=0.025, zoom=2.0),
        # a small odd crop at high quality: more samples than one mask filter holds
        _plane("grain", "grain_crop_311x205_n400", 311, 205, 0.08, 400, "ramp", zoom=1.5),
        # a photograph-sized image with the command line's defaults, host floats in, host bytes out
        _image("image_luma_1920x1080", 1920, 1080, 0.10, 32, "luma", "auto", "blobs"),
        # the large-frame benchmark end to end: 4096^2 RGB, the longest call users make
        _image("image_rgb_4096", 4096, 4096, 0.025, 256, "rgb", "pixel", "blobs", sd=0.01),
        # a batch of uneven luma images, pixel-wise and grain-wise mixed, behind one graph
        {"name": "batch_uneven_16", "kind": "batch", "count": 16, "largest": 1024, "mix": 7},
        # the surrogate: one residual layer over a megapixel RGB frame's three planes
        _net("surrogate_layer_3x1024x1024", "layer", 3, 1024, 1024),
        # the surrogate's whole preview of an RGB frame
        _net("surrogate_infer_3x720x1280", "infer", 3, 720, 1280),
        # forward and backward of the surrogate on a training batch of 64^2 tiles
        _net("surrogate_gradients_256x64x64", "gradients", 256, 64, 64),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["pixel", "pixel", "pixel", "grain", "grain", "image", "image", "batch", "layer", "infer",
                       "gradients"])
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(2, 24), "largest": rng.choice([256, 512, 1024]),
                "mix": rng.randrange(1 << 20)}
    if kind == "gradients":
        side = rng.randint(24, 96)
        return {"kind": kind, "nb": max(1, int(_log(rng, 16, 256) * 4096 / max(4096, side * side))), "h": side,
                "w": rng.randint(24, 96)}
    if kind in ("layer", "infer"):
        return {"kind": kind, "nb": rng.choice([1, 3]), "h": int(_log(rng, 60, 1400)), "w": int(_log(rng, 60, 1400))}
    c = {"kind": kind, "w": int(_log(rng, 48, 1400)), "h": int(_log(rng, 48, 1400)),
         "radius": round(_log(rng, 0.025, 0.2), 4), "sd": 0.0, "n": int(_log(rng, 12, 256)),
         "zoom": rng.choice([0.5, 1.0, 1.0, 1.0, 1.5, 2.0]), "source": rng.choice(["ramp", "blobs"]),
         "stream": rng.randrange(1 << 31)}
    if rng.random() < 0.5:
        c["sd"] = round(c["radius"] * rng.uniform(0.2, 0.5), 5)
    if kind == "grain" and rng.random() < 0.25:
        c["n"] = rng.randint(257, 512)
    if kind == "image":
        c.update(color=rng.choice(["luma", "rgb"]), algo=rng.choice(["auto", "auto", "grain", "pixel"]),
                 roi=rng.random() < 0.3)
    return c


# ---------------------------------------------------------------------- inputs
def _light(w, h, source, seed):
    """A plane in [0, 1] on the GPU: a noisy horizontal ramp, or Gaussian blobs over a 0.1 background (the
    benchmark's two families; blobs shrink with planes under 1536 px, which they would saturate)."""
    g = torch.Generator().manual_seed(seed)
    if source == "ramp":
        noise = torch.rand((h, w), generator=g) * 0.1 - 0.05
        return (torch.linspace(0.0, 1.0, w)[None, :] + noise).clamp_(0.0, 1.0).cuda()
    u = torch.rand((4, 16), generator=g, dtype=torch.float64)
    scale = min(1.0, max(w, h) / 1536.0)
    amp, sig = 0.2 + 0.7 * u[0], (30.0 + 120.0 * u[1]) * scale
    ax = [torch.exp(-((torch.arange(n, dtype=torch.float64)[None, :] + 0.5 - n * c[:, None]) ** 2) /
                    (2 * sig[:, None] ** 2)).cuda() for n, c in ((w, u[2]), (h, u[3]))]
    v = 0.1 + torch.einsum("b,by,bx->yx", amp.cuda(), ax[1], ax[0])
    return v.clamp_(0.0, 1.0).float()


def _params(case, **more):
    sd = case["sd"]
    return fg.ParamsBuilder(radius_mean=case["radius"], radius_stddev=sd,
                            radius_dist=fg.RadiusDist.Lognorm if sd > 0 else fg.RadiusDist.Const, zoom=case["zoom"],
                            n_samples=case["n"], seed=case["stream"], **more).build()


def _lambda(plane, derived):
    return fg.lambda_from_plane(plane.cpu().numpy(), derived.inv_e_pi_r2)[0]


def _batch_members(case):
    """Sizes, radii and sample counts of the benchmark's sweep, up to the case's largest size."""
    rng = np.random.default_rng(case["mix"])
    sizes = [s for s in (128, 256, 512, 1024) if s <= case["largest"]]
    return [dict(kind="batch", w=int(rng.choice(sizes)) - int(rng.integers(0, 8)), h=int(rng.choice(sizes)), sd=0.0,
                 zoom=1.0, radius=float(rng.choice((0.025, 0.05, 0.1, 0.2))), n=int(rng.choice((16, 64, 256))),
                 source="blobs", stream=int(rng.integers(0, 2**32))) for _ in range(case["count"])]


def _net_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    nb, h, w = case["nb"], case["h"], case["w"]
    if case["kind"] == "layer":
        x = torch.randn((nb, h, w, 32), generator=g, device="cuda").relu_().to(torch.bfloat16)
        wt = (torch.randn((32, 9, 32), generator=g, device="cuda") * 0.03).to(torch.bfloat16)
        return {"x": x, "w": wt, "b": torch.randn(32, generator=g, device="cuda") * 0.05}
    if h * w > 96 * 96:
        u = torch.stack([_light(w, h, "blobs", seed * 8 + c) for c in range(nb)])
    else:  # training tiles: coarse textures with fine noise
        u = torch.nn.functional.interpolate(torch.rand((nb, 1, 8, 8), generator=g, device="cuda"), size=(h, w),
                                            mode="bilinear")[:, 0]
        u = (u + 0.05 * torch.randn((nb, h, w), generator=g, device="cuda")).clamp_(0.0, 0.99)
    radius = torch.rand(nb, generator=g, device="cuda") * 0.17 + 0.03
    target = (u + 0.1 * torch.randn((nb, h, w), generator=g, device="cuda")).clamp_(0.0, 1.0)
    return {"u": u.contiguous(), "radius": radius, "target": target, "noise": seed * 977 + 5}


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind in ("pixel", "grain"):
        s["params"] = _params(case)
        s["derived"] = fg.derive_common(s["params"], (case["w"], case["h"]))
        plane = _light(case["w"], case["h"], case["source"], seed)
        s["lam"] = torch.from_numpy(_lambda(plane, s["derived"])).cuda()
    elif kind == "image":
        w, h = case["w"], case["h"]
        roi = fg.Roi(w // 8, h // 8, w - w // 16, h - h // 16) if case["roi"] else None
        algo = {"auto": fg.Algo.Auto, "grain": fg.Algo.Grain, "pixel": fg.Algo.Pixel}[case["algo"]]
        s["params"] = _params(case, color_mode=fg.ColorMode.Rgb if case["color"] == "rgb" else fg.ColorMode.Luma,
                              algo=algo, roi=roi)
        s["rgb"] = torch.stack([_light(w, h, case["source"], seed * 3 + c) for c in range(3)], dim=-1).cpu().numpy()
    elif kind == "batch":
        items = []
        for k, m in enumerate(_batch_members(case)):
            p = _params(m)
            d = fg.derive_common(p, (m["w"], m["h"]))
            lam = _lambda(_light(m["w"], m["h"], m["source"], seed * 64 + k), d)
            items.append((torch.from_numpy(lam).cuda(), p, d, fg.choose_algorithm(p, d), lam))
        s["batch"] = fg.Batch(items)
    else:
        s.update(_net_inputs(case, seed))
        if kind == "layer":
            s["out"] = torch.empty_like(s["x"])
        else:
            s["net"] = sg.load_default()
    return s


# ---------------------------------------------------------------------- one pass
def run(s):
    kind = s["kind"]
    if kind == "pixel":
        return fg.render_pixelwise(s["lam"], s["params"], s["derived"])
    if kind == "grain":
        return fg.render_grainwise(s["lam"], s["params"], s["derived"])
    if kind == "image":
        return fg.render_with_input_image(s["rgb"], s["params"])[0]
    if kind == "batch":
        s["batch"].run()
        return s["batch"].outputs
    if kind == "layer":
        x, nb, h, w = s["x"], *s["x"].shape[:3]
        rc = fg.lib().fg_sg_conv_forward(sg.CONV_RESIDUAL, x.data_ptr(), 32, s["w"].data_ptr(), s["b"].data_ptr(),
                                         x.data_ptr(), None, s["out"].data_ptr(), None, None, nb, h, w,
                                         torch.cuda.current_stream().cuda_stream)
        if rc:
            raise RuntimeError(fg.lib().fg_last_error_message().decode())
        return s["out"]
    net = s["net"]
    if kind == "infer":
        return net.infer(s["u"], s["radius"], seed=s["noise"])
    y = net.forward(s["u"], s["radius"], seed=s["noise"], keep=True)
    loss = net.backward(s["u"], s["target"])
    return {"y": y, "loss": loss, "grad": net.grad}


# ---------------------------------------------------------------------- what a pass cannot do without
def _plane_work(c):
    """Each sample's point and cell range (30 operations), each grain's draws (70, or 150 with a log-normal
    radius), and for the grain-wise integrator the bit of each covered sample (12)."""
    px, out = c["w"] * c["h"], c["w"] * c["h"] * c["zoom"] ** 2
    per_px = LIGHT[c["source"]] / (math.pi * (c["radius"] ** 2 + c["sd"] ** 2))
    grains = px * per_px
    ops = grains * (150 if c["sd"] > 0 else 70)
    if c["kind"] == "grain":
        ops += 12 * out * c["n"] * LIGHT[c["source"]]
    else:
        ops += 30 * out * c["n"]
    return {"bytes": 4.0 * (px + out), "flops": ops}


def work(case):
    kind = case["kind"]
    if kind in ("pixel", "grain"):
        return _plane_work(case)
    if kind == "image":
        c = dict(case, kind="pixel" if case["algo"] == "pixel" else "grain")
        if case["roi"]:
            c.update(w=case["w"] * 13 // 16, h=case["h"] * 13 // 16)
        one = _plane_work(c)
        px = c["w"] * c["h"]
        return {"bytes": 12.0 * px + 3.0 * px * c["zoom"] ** 2, "flops": one["flops"] * (3 if c["color"] == "rgb" else 1)}
    if kind == "batch":
        parts = [_plane_work(m) for m in _batch_members(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    px = case["nb"] * case["h"] * case["w"]
    if kind == "layer":
        return {"bytes": 128.0 * px, "flops": 2.0 * 9 * 32 * 32 * px}
    forward = 2.0 * 9 * (3 * 32 + 8 * 32 * 32 + 32) * px
    if kind == "infer":
        return {"bytes": 8.0 * px, "flops": forward}
    return {"bytes": 12.0 * px, "flops": 3.0 * forward}


# ---------------------------------------------------------------------- the same results in 64 bits
def _conv64(x, w):
    """3x3 zero-padded conv of x [n, h, w, ci] with w [co, 9, ci], both float64."""
    n, h, wd, ci = x.shape
    xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    z = torch.zeros((n, h, wd, w.shape[0]), dtype=torch.float64, device=x.device)
    for tap in range(9):
        ky, kx = divmod(tap, 3)
        z += xp[:, ky:ky + h, kx:kx + wd] @ w[:, tap].T
    return z


def _weights64():
    z = np.load(os.path.join(os.path.dirname(sg.__file__), "weights", "surrogate_c4.npz"))
    flat = torch.from_numpy(z["w32"]).cuda()
    out, at = {}, 0
    for name, shape in (("w_in", (32, 9, 16)), ("w_res", (8, 32, 9, 32)), ("w_out", (8, 9, 32)), ("b_in", (32,)),
                        ("b_res", (8, 32)), ("b_out", (8,))):
        k = math.prod(shape)
        part = flat[at:at + k].reshape(shape)
        out[name] = (part.to(torch.bfloat16) if name[0] == "w" else part).double()
        at += k
    return out, float(z["radius_scale"])


def _mul(a, b):
    """a * b mod 2^64 on int64 tensors."""
    return a * (b - (1 << 64) if b >= 1 << 63 else b)


def _shr(a, k):
    return (a >> k) & ((1 << (64 - k)) - 1)


def _network_input(u, radius, scale, seed):
    """(u, N(0, 1) noise, radius) per pixel; the noise is a Box-Muller transform of two 24-bit uniforms from a
    64-bit hash of the seed and the pixel's index."""
    n = u.numel()
    i = torch.arange(1, n + 1, dtype=torch.int64, device=u.device)
    z = _mul(i, 0x9E3779B97F4A7C15) + seed
    z = _mul(z ^ _shr(z, 30), 0xBF58476D1CE4E5B9)
    z = _mul(z ^ _shr(z, 27), 0x94D049BB133111EB)
    z = z ^ _shr(z, 31)
    u1 = (_shr(z, 40).double() + 0.5) / 2**24
    u2 = ((_shr(z, 8) & 0xFFFFFF).double() + 0.5) / 2**24
    noise = torch.sqrt(-2.0 * torch.log(u1)) * torch.cos(2.0 * math.pi * u2)
    x = torch.zeros(tuple(u.shape) + (16,), dtype=torch.float64, device=u.device)
    x[..., 0] = u.double()
    x[..., 1] = noise.reshape(u.shape)
    x[..., 2] = radius.double()[:, None, None] * scale
    return x


def exact(case, seed):
    """The surrogate's results in float64.  The renders have none: their counts are defined by 32-bit draws
    and comparisons."""
    kind = case["kind"]
    if kind == "layer":
        s = _net_inputs(case, seed)
        x = s["x"].double()
        return x + torch.relu(_conv64(x, s["w"].double()) + s["b"].double())
    if kind not in ("infer", "gradients"):
        return None
    s = _net_inputs(case, seed)
    W, scale = _weights64()
    x = _network_input(s["u"], s["radius"], scale, s["noise"])
    h = torch.relu(_conv64(x, W["w_in"]) + W["b_in"])
    hs, rs = [h], []
    for l in range(8):
        rs.append(torch.relu(_conv64(h, W["w_res"][l]) + W["b_res"][l]))
        h = h + rs[-1]
        hs.append(h)
        if kind == "infer":
            hs, rs = [h], []
    y = s["u"].double() + _conv64(h, W["w_out"])[..., 0] + W["b_out"][0]
    if kind == "infer":
        return y
    e = y - s["target"].double()
    g = torch.zeros(tuple(y.shape) + (8,), dtype=torch.float64, device=y.device)
    g[..., 0] = e * (2.0 / e.numel())

    def weight_grad(g, x):
        n, h, wd, ci = x.shape
        xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
        gf = g.reshape(-1, g.shape[-1]).T
        return torch.stack([gf @ xp[:, t // 3:t // 3 + h, t % 3:t % 3 + wd].reshape(-1, ci) for t in range(9)], dim=1)

    def data_grad(g, w):
        return _conv64(g, w.flip(1).permute(2, 1, 0).contiguous())

    grads = {"w_out": weight_grad(g, hs[8]), "b_out": g.sum((0, 1, 2)), "w_res": [], "b_res": []}
    dh = data_grad(g, W["w_out"])
    for l in range(7, -1, -1):
        dz = dh * (rs[l] > 0)
        grads["w_res"].insert(0, weight_grad(dz, hs[l]))
        grads["b_res"].insert(0, dz.sum((0, 1, 2)))
        dh = dh + data_grad(dz, W["w_res"][l])
    dz = dh * (hs[0] > 0)
    flat = [weight_grad(dz, x), torch.stack(grads["w_res"]), grads["w_out"], dz.sum((0, 1, 2)),
            torch.stack(grads["b_res"]), grads["b_out"]]
    return {"y": y, "loss": (e * e).sum().reshape(1), "grad": torch.cat([t.reshape(-1) for t in flat])}
