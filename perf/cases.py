"""Timed workloads of the texture path: what a program that uses this package asks of it.

Each case is one call (or the two calls of a quality check) through the public Python binding:
whole mip chains of single images from the smallest icon to a 4096x4096 albedo map, a mixed batch,
one float level, mip levels alone, a host-buffer call, decoding with error sums, and one
forward + backward pass of the proposal network. Images are synthetic, of the same kinds as
`ntg.synth` (sinusoid octaves, hard-edged rectangles and +-8 noise; a value-noise alpha with 30% of
its texels snapped to 0 or 255; an fBm normal map), generated on the GPU.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nvidia-texture-tools_gb300"))

import ntg  # noqa: E402

FORMATS = {"bc1": ntg.FORMAT_BC1, "bc1a": ntg.FORMAT_BC1A, "bc3": ntg.FORMAT_BC3, "bc4": ntg.FORMAT_BC4,
           "bc5": ntg.FORMAT_BC5}
QUALITIES = {"fastest": ntg.QUALITY_FASTEST, "normal": ntg.QUALITY_NORMAL, "production": ntg.QUALITY_PRODUCTION}
FILTERS = {"box": ntg.FILTER_BOX, "triangle": ntg.FILTER_TRIANGLE, "kaiser": ntg.FILTER_KAISER}
WRAPS = {"clamp": ntg.WRAP_CLAMP, "repeat": ntg.WRAP_REPEAT, "mirror": ntg.WRAP_MIRROR}
XFORMS = {"none": ntg.XFORM_NONE, "gamma": ntg.XFORM_GAMMA, "srgb": ntg.XFORM_SRGB}


def chain(name, kind, w, h, fmt="bc1", quality="normal", filt="box", wrap="mirror", transparency=False, xform="none"):
    case = {"kind": kind, "w": w, "h": h, "format": fmt, "quality": quality, "filter": filt, "wrap": wrap,
            "transparency": transparency, "xform": xform}
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # an icon or a glyph page: the smallest call, all launches and latency
        chain("icon_bc1_64", "chain", 64, 64, "bc1", filt="box"),
        # the reference's CPU-runnable configuration: one 512x512 opaque texture, linear, box mips
        chain("texture_bc1_512", "chain", 512, 512, "bc1", filt="box"),
        # a screenshot or a user's upload: odd extents on every level, sRGB, Kaiser mips
        chain("upload_bc1_1366x769", "chain", 1366, 769, "bc1", filt="kaiser", xform="srgb"),
        # a decal with alpha: small BC3 in gamma space, tiled
        chain("decal_bc3_256", "chain", 256, 256, "bc3", filt="triangle", wrap="repeat", transparency=True, xform="gamma"),
        # the large single-image configuration: 4096x4096 sRGB albedo with alpha, Kaiser mips
        chain("albedo_bc3_4096", "chain", 4096, 4096, "bc3", filt="kaiser", transparency=True, xform="srgb"),
        # a normal map of a model
        chain("normals_bc5_1024", "chain", 1024, 1024, "bc5", filt="triangle"),
        # an asset build: textures of uneven power-of-two sizes, 50/30/20 BC1/BC3/BC5, one graph
        {"name": "batch_mixed_40", "kind": "batch", "count": 40, "kmin": 6, "kmax": 10, "filter": "triangle"},
        # one float level at Production quality with colour weights, as the Surface loop encodes it
        chain("level_bc1_production_640x360", "level", 640, 360, "bc1", quality="production", xform="srgb"),
        # mip levels for a program that encodes them elsewhere: float levels out
        chain("levels_kaiser_2048", "levels", 2048, 2048, filt="kaiser", xform="srgb"),
        # Compressor::process as most programs call it: host image in, host blocks out
        chain("host_bc1_1024", "host", 1024, 1024, "bc1", filt="kaiser"),
        # a quality check: decode a compressed image and sum its errors against the source
        {"name": "check_bc3_2048", "kind": "check", "w": 2048, "h": 2048, "transparency": True},
        # training the proposal network: one batch of the configured size, forward and backward
        {"name": "train_8192", "kind": "train", "rows": 8192},
    ]


def _extent(rng, lo, hi):
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 0.4:  # power-of-two textures are common, and odd ones happen
        return 1 << max(0, round(math.log2(v)))
    return v | 1 if rng.random() < 0.5 else v


def draw(rng):
    u = rng.random()
    filt = rng.choice(["box", "triangle", "kaiser"])
    wrap = rng.choice(["clamp", "repeat", "mirror"])
    xform = rng.choice(["none", "srgb", "srgb", "gamma"])
    if u < 0.5:
        fmt = rng.choice(["bc1", "bc1", "bc1", "bc3", "bc3", "bc5", "bc4", "bc1a"])
        w = _extent(rng, 32, 3000)
        h = w if rng.random() < 0.5 else _extent(rng, 32, 3000)
        quality = "normal"
        if rng.random() < 0.25 and fmt != "bc1a":
            quality = "fastest"
        if fmt in ("bc5", "bc4"):
            xform = "none"
        return chain(None, "chain", w, h, fmt, quality, filt, wrap, fmt != "bc5" and rng.random() < 0.5, xform)
    if u < 0.6:
        return {"kind": "batch", "count": rng.randint(4, 40), "kmin": rng.randint(5, 7), "kmax": rng.randint(8, 10),
                "filter": rng.choice(["triangle", "kaiser"])}
    if u < 0.7:
        fmt = rng.choice(["bc1", "bc1", "bc3"])
        return chain(None, "level", _extent(rng, 32, 1000), _extent(rng, 32, 1000), fmt,
                     rng.choice(["normal", "production"]), transparency=rng.random() < 0.3, xform=xform)
    if u < 0.8:
        return chain(None, "levels", _extent(rng, 64, 3000), _extent(rng, 64, 3000), filt=rng.choice(["triangle", "kaiser"]),
                     wrap=wrap, xform=rng.choice(["none", "srgb"]))
    if u < 0.88:
        return chain(None, "host", _extent(rng, 64, 1500), _extent(rng, 64, 1500), rng.choice(["bc1", "bc3", "bc5"]),
                     filt=filt, wrap=wrap)
    if u < 0.94:
        return {"kind": "check", "w": _extent(rng, 64, 3000), "h": _extent(rng, 64, 3000), "transparency": rng.random() < 0.5}
    return {"kind": "train", "rows": 8 * int(round(math.exp(rng.uniform(math.log(64), math.log(4096)))))}


# ---- inputs ----

_ctx = None


def _context():
    """The context that a program keeps for its lifetime."""
    global _ctx
    if _ctx is None:
        _ctx = ntg.Context(0)
    return _ctx


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _smooth(g, h, w, cell):
    """Value noise: a random lattice of `cell` texels, interpolated."""
    lattice = torch.rand((1, 1, int(h / cell) + 2, int(w / cell) + 2), generator=g, device="cuda")
    return torch.nn.functional.interpolate(lattice, size=(h, w), mode="bilinear", align_corners=True)[0, 0]


def _colour(g, w, h, with_alpha):
    """(h, w, 4) float texels in 0..255, BGRA."""
    scale = max(1.0, min(w, h) / 512.0)
    p = torch.rand((4, 4), generator=g, device="cuda").mul_(2 * math.pi).cpu().numpy()
    xs = torch.arange(w, device="cuda", dtype=torch.float32)[None, :]
    ys = torch.arange(h, device="cuda", dtype=torch.float32)[:, None]
    phase = torch.tensor(p[:, 1:], device="cuda", dtype=torch.float32)
    rgb = torch.full((h, w, 3), 128.0, device="cuda")
    for o in range(4):
        f = 2 * math.pi * (2 ** o) / (256.0 * scale)
        along = (xs * math.cos(p[o, 0]) + ys * math.sin(p[o, 0])) * f
        rgb += (56.0 / 2 ** o) * torch.sin(along[..., None] + phase[o])
    r = torch.rand((12, 7), generator=g, device="cuda").cpu().numpy()
    for q in r:
        rw, rh = int((16 + 113 * q[0]) * scale), int((16 + 113 * q[1]) * scale)
        x0, y0 = int(q[2] * max(1, w - min(rw, w) + 1)), int(q[3] * max(1, h - min(rh, h) + 1))
        rgb[y0:y0 + rh, x0:x0 + rw] = torch.tensor([float(int(255 * v)) for v in q[4:7]], device="cuda")
    rgb += torch.rand(rgb.shape, generator=g, device="cuda") * 16.0 - 8.0
    alpha = torch.full((h, w, 1), 255.0, device="cuda")
    if with_alpha:
        v = 0.65 * _smooth(g, h, w, 32.0 * scale) + 0.35 * _smooth(g, h, w, 8.0 * scale)
        v = torch.round(v * 255.0)
        snap = torch.rand(v.shape, generator=g, device="cuda") < 0.3
        alpha = torch.where(snap, torch.where(v < 128, 0.0, 255.0), v)[..., None]
    return torch.cat([rgb.clamp(0, 255), alpha], dim=2)


def _normals(g, w, h):
    height = torch.zeros((h, w), device="cuda")
    for o in range(5):
        height += (0.5 ** o) * _smooth(g, h, w, max(2.0, min(w, h) / (4.0 * 2 ** o)))
    dx = 4.0 * (torch.roll(height, -1, 1) - torch.roll(height, 1, 1))
    dy = 4.0 * (torch.roll(height, -1, 0) - torch.roll(height, 1, 0))
    inv = torch.rsqrt(dx * dx + dy * dy + 1.0)
    full = torch.full_like(dx, 255.0)
    return torch.stack([torch.zeros_like(dx), (-dy * inv * 0.5 + 0.5) * 255.0, (-dx * inv * 0.5 + 0.5) * 255.0, full], dim=2)


def _image(g, w, h, fmt):
    """(h, w, 4) BGRA8 on the GPU."""
    texels = _normals(g, w, h) if fmt == "bc5" else _colour(g, w, h, fmt in ("bc3", "bc4", "bc1a"))
    return torch.round(texels).clamp(0, 255).to(torch.uint8).contiguous()


def _options(case):
    x = XFORMS[case["xform"]]
    return ntg.ChainOptions.make(format=FORMATS[case["format"]], quality=QUALITIES[case["quality"]],
                                 filter=FILTERS[case["filter"]], wrap=WRAPS[case["wrap"]],
                                 alpha_mode=ntg.ALPHA_TRANSPARENCY if case["transparency"] else ntg.ALPHA_NONE,
                                 in_xform=x, out_xform=x)


def _batch_textures(case, seed):
    """(w, h, format, seed) per texture: powers of two, 80% square, 50/30/20 BC1/BC3/BC5. The sizes and
    formats belong to the case, the images to the seed."""
    rng = np.random.default_rng(case["count"] * 1000 + case["kmin"] * 10 + case["kmax"])
    out = []
    for i in range(case["count"]):
        kw = int(rng.integers(case["kmin"], case["kmax"] + 1))
        kh = kw if rng.random() < 0.8 else int(rng.integers(case["kmin"], case["kmax"] + 1))
        u = rng.random()
        out.append((1 << kw, 1 << kh, "bc1" if u < 0.5 else ("bc3" if u < 0.8 else "bc5"), seed * 1009 + i))
    return out


def _compressed(img):
    """A bounding-box BC3 encoding of an image whose extents are padded to fours: (blocks, 16) bytes."""
    h, w = img.shape[0], img.shape[1]
    ph, pw = -h % 4, -w % 4
    x = torch.nn.functional.pad(img.permute(2, 0, 1).float()[None], (0, pw, 0, ph), mode="replicate")[0].long()
    bh, bw = (h + ph) // 4, (w + pw) // 4
    x = x.reshape(4, bh, 4, bw, 4).permute(1, 3, 2, 4, 0).reshape(bh * bw, 16, 4)
    rgb, a = x[..., [2, 1, 0]], x[..., 3]
    shift, top = torch.tensor([3, 2, 3], device="cuda"), torch.tensor([11, 5, 0], device="cuda")
    c0 = ((rgb.amax(1) >> shift) << top).sum(1)
    c1 = ((rgb.amin(1) >> shift) << top).sum(1)
    pal = _colour_palette(c0, c1)
    d = ((rgb[:, :, None, :] - pal[:, None]) ** 2).sum(3)
    index = torch.where((c0 > c1)[:, None], d.argmin(2), torch.zeros_like(a))
    a0, a1 = a.amax(1), a.amin(1)
    ai = (a[:, :, None] - _alpha_palette(a0, a1)[:, None]).abs().argmin(2)
    weights = torch.arange(16, device="cuda")
    bits = (index << (2 * weights)).sum(1)
    lo, hi = (ai[:, :8] << (3 * weights[:8])).sum(1), (ai[:, 8:] << (3 * weights[:8])).sum(1)
    out = [a0, a1] + [(v >> s) & 255 for v in (lo, hi) for s in (0, 8, 16)]
    out += [c0 & 255, c0 >> 8, c1 & 255, c1 >> 8] + [(bits >> s) & 255 for s in (0, 8, 16, 24)]
    return torch.stack(out, 1).to(torch.uint8).contiguous()


def _colour_palette(c0, c1):
    """(n, 4, 3) RGB of the two 5:6:5 endpoints as the D3D10 decoder expands them."""
    def expand(c):
        r, g, b = (c >> 11) & 31, (c >> 5) & 63, c & 31
        return torch.stack([(r << 3) | (r >> 2), (g << 2) | (g >> 4), (b << 3) | (b >> 2)], 1)
    p0, p1 = expand(c0), expand(c1)
    four = (c0 > c1)[:, None]
    p2 = torch.where(four, (2 * p0 + p1) // 3, (p0 + p1) // 2)
    p3 = torch.where(four, (2 * p1 + p0) // 3, torch.zeros_like(p0))
    return torch.stack([p0, p1, p2, p3], 1)


def _alpha_palette(a0, a1):
    eight = a0 > a1
    pal = [a0, a1]
    for k in range(1, 7):
        six = (((5 - k) * a0 + k * a1) // 5) if k < 5 else torch.full_like(a0, 0 if k == 5 else 255)
        pal.append(torch.where(eight, ((7 - k) * a0 + k * a1) // 7, six))
    return torch.stack(pal, 1)


def _network(seed):
    """The network's flat parameters: W1, b1, W2, b2, W3, b3, uniform in +-sqrt(3 / fan in)."""
    rng = np.random.default_rng(seed ^ 0x4E4554)
    parts = []
    for out, inp in ((256, 48), (256, 256), (8, 256)):
        r = math.sqrt(3.0 / inp)
        parts += [rng.uniform(-r, r, out * inp), rng.uniform(-0.1, 0.1, out)]
    return np.concatenate(parts).astype(np.float32)


def _samples(seed, rows):
    """Block texels in [0, 1] (a colour ramp with noise, sorted along it) and targets of the trained kind."""
    g = _generator(seed)
    ends = torch.rand((rows, 2, 1, 3), generator=g, device="cuda")
    t = torch.sort(torch.rand((rows, 16, 1), generator=g, device="cuda"), dim=1).values
    x = ends[:, 0] + (ends[:, 1] - ends[:, 0]) * 0.3 * t + (torch.rand((rows, 16, 3), generator=g, device="cuda") - 0.5) / 16
    y = torch.rand((rows, 8), generator=g, device="cuda")
    y[:, :3] = torch.sort(y[:, :3], dim=1).values
    y[:, 5] = -3.0 * y[:, 5]
    y[:, 6:] = 0.0
    return x.clamp(0, 1).reshape(rows, 48).contiguous(), y.contiguous()


def prepare(case, seed):
    kind, ctx, g = case["kind"], _context(), _generator(seed)
    if kind in ("chain", "levels"):
        return {"kind": kind, "ctx": ctx, "image": _image(g, case["w"], case["h"], case["format"]), "w": case["w"],
                "h": case["h"], "opt": _options(case)}
    if kind == "host":
        return {"kind": kind, "ctx": ctx, "image": _image(g, case["w"], case["h"], case["format"]).cpu().numpy(),
                "w": case["w"], "h": case["h"], "opt": _options(case)}
    if kind == "batch":
        items = []
        for w, h, fmt, s in _batch_textures(case, seed):
            opt = ntg.ChainOptions.make(format=FORMATS[fmt], filter=FILTERS[case["filter"]],
                                        alpha_mode=ntg.ALPHA_TRANSPARENCY if fmt == "bc3" else ntg.ALPHA_NONE)
            out = torch.empty(ntg.chain_bytes(w, h, opt), dtype=torch.uint8, device="cuda")
            items.append((_image(_generator(s), w, h, fmt), w, h, opt, out))
        return {"kind": kind, "batch": ntg.Batch(ctx, items), "outs": [i[4] for i in items]}
    if kind == "level":
        # a filtered level: each texel the mean of four of a twice larger image, in linear light
        texels = _colour(g, 2 * case["w"], 2 * case["h"], case["transparency"])[..., [2, 1, 0, 3]] / 255.0
        texels[..., :3] = texels[..., :3] ** 2.2
        level = torch.nn.functional.avg_pool2d(texels.permute(2, 0, 1)[None], 2)[0].contiguous()
        return {"kind": kind, "ctx": ctx, "level": level, "case": case}
    if kind == "check":
        img = _image(g, case["w"], case["h"], "bc3")
        source = (img.permute(2, 0, 1)[[2, 1, 0, 3]].float() / 255.0).contiguous()
        return {"kind": kind, "ctx": ctx, "blocks": _compressed(img), "source": source, "case": case}
    net = ntg.MLP(0)
    net.set_params(_network(seed))
    x, t = _samples(seed, case["rows"])
    return {"kind": kind, "net": net, "x": x, "t": t}


def run(state):
    kind = state["kind"]
    if kind == "chain":
        return state["ctx"].compress_chain(state["image"], state["w"], state["h"], state["opt"])
    if kind == "levels":
        return state["ctx"].mip_chain(state["image"], state["w"], state["h"], state["opt"])
    if kind == "host":
        return state["ctx"].compress_chain_host(state["image"], state["w"], state["h"], state["opt"])
    if kind == "batch":
        state["batch"].launch()
        return state["outs"]
    if kind == "level":
        c = state["case"]
        return state["ctx"].encode(FORMATS[c["format"]], state["level"], c["w"], c["h"], QUALITIES[c["quality"]],
                                   ntg.ALPHA_TRANSPARENCY if c["transparency"] else ntg.ALPHA_NONE, XFORMS[c["xform"]],
                                   cw=(0.6, 1.0, 0.4))
    if kind == "check":
        c = state["case"]
        mode = ntg.ALPHA_TRANSPARENCY if c["transparency"] else ntg.ALPHA_NONE
        decoded = state["ctx"].decode(ntg.FORMAT_BC3, state["blocks"], c["w"], c["h"])
        return {"decoded": decoded, "sums": state["ctx"].error_sums(state["source"], decoded, c["w"], c["h"], mode)}
    grads, loss = state["net"].gradients(state["x"], state["t"])
    return {"grads": grads, "loss": loss}


# ---- the work a pass cannot do without ----

def _levels(w, h):
    out = [(w, h)]
    while (w, h) != (1, 1):
        w, h = max(1, w // 2), max(1, h // 2)
        out.append((w, h))
    return out


# Multiplies and adds per block: an interpolated channel's palette search and least squares; for a
# colour fit, 16 operations to rank each of the 968 + 152 cluster orderings by its least-squares
# error (sums of three cumulative colours, their square, the determinant), which no exact search
# over 16 colours avoids.
BLOCK_FLOPS = {"bc1": 16 * 1120, "bc1a": 16 * 1120, "bc3": 16 * 969 + 16 * 8 * 2, "bc4": 16 * 8 * 2, "bc5": 2 * 16 * 8 * 2}
BLOCK_BYTES = {"bc1": 8, "bc1a": 8, "bc3": 16, "bc4": 8, "bc5": 16}
TAPS = {"box": 2, "triangle": 5, "kaiser": 13}


def _chain_work(w, h, fmt, filt, fit=True):
    levels = _levels(w, h)
    blocks = sum(((a + 3) // 4) * ((b + 3) // 4) for a, b in levels)
    outputs = sum(a * b for a, b in levels[1:])
    # per output texel and channel: the X taps of two source rows, the Y taps of one column
    flops = outputs * 4 * 2 * TAPS[filt] * 3 + (blocks * BLOCK_FLOPS[fmt] if fit else 0)
    return levels, blocks, flops


def work(case):
    kind = case["kind"]
    if kind in ("chain", "host"):
        _, blocks, flops = _chain_work(case["w"], case["h"], case["format"], case["filter"])
        return {"bytes": 4 * case["w"] * case["h"] + blocks * BLOCK_BYTES[case["format"]], "flops": flops}
    if kind == "batch":
        total = {"bytes": 0, "flops": 0}
        for w, h, fmt, _s in _batch_textures(case, 0):
            _, blocks, flops = _chain_work(w, h, fmt, case["filter"])
            total["bytes"] += 4 * w * h + blocks * BLOCK_BYTES[fmt]
            total["flops"] += flops
        return total
    if kind == "levels":
        levels, _, flops = _chain_work(case["w"], case["h"], "bc1", case["filter"], fit=False)
        return {"bytes": 4 * case["w"] * case["h"] + 16 * sum(a * b for a, b in levels), "flops": flops}
    if kind == "level":
        blocks = ((case["w"] + 3) // 4) * ((case["h"] + 3) // 4)
        return {"bytes": 16 * case["w"] * case["h"] + blocks * BLOCK_BYTES[case["format"]],
                "flops": blocks * BLOCK_FLOPS[case["format"]]}
    if kind == "check":
        n = case["w"] * case["h"]
        blocks = ((case["w"] + 3) // 4) * ((case["h"] + 3) // 4)
        # blocks in, decoded image out; source and decoded image into the sums
        return {"bytes": 16 * blocks + 48 * n, "flops": 14 * n}
    rows, params = case["rows"], 256 * 48 + 256 + 256 * 256 + 256 + 8 * 256 + 8
    macs = 48 * 256 + 256 * 256 + 256 * 8
    return {"bytes": rows * (48 + 8) * 4 + params * 8, "flops": rows * 2 * (3 * macs - 48 * 256)}


# ---- the same results in 64 bits ----

def _filter_value(filt, x):
    """The filter's value at numpy positions x (unit scale): triangle of width 1, Kaiser of width 3, alpha 4."""
    x = np.abs(x)
    if filt == "triangle":
        return np.where(x < 1.0, 1.0 - x, 0.0)
    t = x / 3.0
    inside = 1.0 - t * t
    return np.where(inside >= 0, np.sinc(x) * np.i0(4.0 * np.sqrt(np.maximum(inside, 0.0))) / np.i0(4.0), 0.0)


def _axis(filt, wrap, n, m):
    """(weights (m, taps), source positions (m, taps)) of a resampling of n texels to m."""
    width = 1.0 if filt == "triangle" else 3.0
    inv = n / m
    taps = math.ceil(width * inv * 2) + 1
    centre = (0.5 + np.arange(m)) * inv
    left = np.floor(centre - width * inv)
    at = left[:, None] + np.arange(taps)
    sub = (np.arange(32) + 0.5) / 32.0
    weights = _filter_value(filt, ((at - centre[:, None])[..., None] + sub) / inv).mean(-1)
    weights /= weights.sum(1, keepdims=True)
    at = at.astype(np.int64)
    if wrap == "clamp":
        at = np.clip(at, 0, n - 1)
    elif wrap == "repeat":
        at = at % n
    elif n == 1:
        at = np.zeros_like(at)
    else:
        period = 2 * n - 2
        at = np.abs(at) % period
        at = np.where(at >= n, period - at, at)
    return torch.from_numpy(weights).cuda(), torch.from_numpy(at).cuda()


def _filtered(img, filt, wrap, m, dim):
    weights, at = _axis(filt, wrap, img.shape[dim], m)
    shape = [1, 1, 1]
    shape[dim] = m
    out = 0
    for j in range(weights.shape[1]):
        out = out + img.index_select(dim, at[:, j]) * weights[:, j].reshape(shape)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "levels":
        if case["filter"] == "box" or case["xform"] == "gamma":
            return None
        img = _image(_generator(seed), case["w"], case["h"], case["format"]).permute(2, 0, 1)[[2, 1, 0, 3]].double() / 255.0
        if case["xform"] == "srgb":
            rgb = img[:3]
            img[:3] = torch.where(rgb < 0.04045, rgb / 12.92, ((rgb + 0.055) / 1.055) ** 2.4)
        levels = [img]
        for w, h in _levels(case["w"], case["h"])[1:]:
            img = _filtered(_filtered(img, case["filter"], case["wrap"], w, 2), case["filter"], case["wrap"], h, 1)
            levels.append(img)
        return torch.cat([lv.reshape(-1) for lv in levels])
    if kind == "check":
        img = _image(_generator(seed), case["w"], case["h"], "bc3")
        w, h = case["w"], case["h"]
        b = _compressed(img).long()
        c0, c1 = b[:, 8] | (b[:, 9] << 8), b[:, 10] | (b[:, 11] << 8)
        k = torch.arange(16, device="cuda")
        index = ((b[:, 12] | (b[:, 13] << 8) | (b[:, 14] << 16) | (b[:, 15] << 24))[:, None] >> (2 * k)) & 3
        rgb = torch.gather(_colour_palette(c0, c1), 1, index[..., None].expand(-1, -1, 3))
        words = [b[:, 2] | (b[:, 3] << 8) | (b[:, 4] << 16), b[:, 5] | (b[:, 6] << 8) | (b[:, 7] << 16)]
        ai = torch.cat([(v[:, None] >> (3 * k[:8])) & 7 for v in words], 1)
        a = torch.gather(_alpha_palette(b[:, 0], b[:, 1]), 1, ai)
        bw, bh = (w + 3) // 4, (h + 3) // 4
        out = torch.cat([rgb, a[..., None]], 2).reshape(bh, bw, 4, 4, 4).permute(4, 0, 2, 1, 3).reshape(4, 4 * bh, 4 * bw)
        out = out[:, :h, :w].double() / 255.0
        source = img.permute(2, 0, 1)[[2, 1, 0, 3]].double() / 255.0
        weight = source[3] ** 2 if case["transparency"] else torch.ones_like(source[3])
        sums = torch.stack([(((source - out)[:3] ** 2).sum(0) * weight).sum(), ((source - out)[3] ** 2).sum()])
        return {"decoded": out.reshape(-1), "sums": sums}
    if kind == "train":
        p = torch.from_numpy(_network(seed)).cuda().double()
        parts, at = [], 0
        for shape in ((256, 48), (256,), (256, 256), (256,), (8, 256), (8,)):
            n = math.prod(shape)
            parts.append(p[at:at + n].reshape(shape).requires_grad_())
            at += n
        w1, b1, w2, b2, w3, b3 = parts
        x, t = (v.double() for v in _samples(seed, case["rows"]))
        hidden = torch.nn.functional.gelu(x @ w1.T + b1, approximate="tanh")
        hidden = torch.nn.functional.gelu(hidden @ w2.T + b2, approximate="tanh")
        weight = torch.tensor([1, 1, 1, 1, 1, 0.25, 0, 0], device="cuda", dtype=torch.float64) / (case["rows"] * 8)
        loss = (weight * (hidden @ w3.T + b3 - t) ** 2).sum()
        grads = torch.autograd.grad(loss, parts)
        return {"grads": torch.cat([v.reshape(-1) for v in grads]), "loss": float(loss.detach())}
    return None
