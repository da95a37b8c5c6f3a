"""Timed cases of the depth stage: what a host program calls it for, through the package's own entry points.

A case is a dict of plain values; `kind` says what is called:

  pair      a rectified grey pair solved as one layer (box filter, cost, eight-path aggregation, winner-take-all), 8-bit
            images or 12-bit camera samples, depth read back into pinned host memory;
  capture   one reference and several module cameras with their own crops and focal lengths summed into one grey layer;
  resume    one ragged layer of a pyramid continued from a stored depth map (its pixels search their own plane ranges);
  pyramid   the whole dense job of a colour capture: six layers, then the upsample to twice the size;
  upsample  the guided upsample of a depth map and its confidence, on device buffers;
  cache     the depth image cache: Set of a full depth map, then one Fetch at an export level;
  stereo    the stereo image of one module after the ISP (warp, YUV, 8-bit store), YUV floats kept;
  census    the census mode on a rectified grey pair (subpixel, left/right check).

Inputs are made on the GPU from the seed: 1/f textures, planar scenes, views warped by their parallax, sensor noise.
"""
import ctypes
import math

import numpy as np
import torch

from lux_b200 import _lib, api

DEV = "cuda:0"


def listed():
    return [
        # half of a served stream: a preview solved while the user frames the shot; latency is all that counts
        {"name": "pair_preview", "kind": "pair", "w": 520, "h": 390, "d": 32, "bits": 8, "tile": 64},
        # the plain pair at the size a CPU can still run
        {"name": "pair_1mp", "kind": "pair", "w": 1040, "h": 780, "d": 64, "bits": 8, "tile": 64},
        # a crop of no round size, planes that fill no power of two, a tile that does not divide it
        {"name": "pair_odd_crop", "kind": "pair", "w": 1431, "h": 1073, "d": 120, "bits": 8, "tile": 32},
        # binned 12-bit sensors at the full disparity range
        {"name": "pair_3mp", "kind": "pair", "w": 2080, "h": 1560, "d": 256, "bits": 12, "tile": 64},
        # the full-resolution 12-bit pair: the largest single solve
        {"name": "pair_13mp", "kind": "pair", "w": 4160, "h": 3120, "d": 256, "bits": 12, "tile": 64},
        # a capture of ten modules fused at cost level
        {"name": "capture_10", "kind": "capture", "w": 2080, "h": 1560, "others": 10, "tile": 64},
        # an interrupted pyramid taken up again at its second-finest layer
        {"name": "resume_layer", "kind": "resume", "w": 2080, "h": 1560, "cams": 5, "level": 4},
        # the whole job of a five-camera colour capture
        {"name": "pyramid_5", "kind": "pyramid", "w": 2080, "h": 1560, "cams": 5},
        # the last step before the renderer, at capture size
        {"name": "upsample_13mp", "kind": "upsample", "w": 2080, "h": 1560},
        # the renderer's and exporter's reads: full depth into the cache, then a region at the largest export level
        {"name": "cache_export", "kind": "cache", "w": 4160, "h": 3120, "cw": 5216, "ch": 3912, "ratio": 2.0},
        # one module's stereo image, ten of which a capture makes
        {"name": "stereo_image", "kind": "stereo", "sw": 2104, "sh": 1560, "w": 2080, "h": 1560},
        # the census mode at the size of a binned sensor
        {"name": "census_3mp", "kind": "census", "w": 2080, "h": 1560, "d": 128},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pair"] * 5 + ["capture", "resume", "pyramid", "upsample", "cache", "stereo", "census"])
    w = _log_int(rng, 420, 4160)
    h = max(200, min(3120, int(w * rng.uniform(0.6, 0.8)) + rng.randrange(3)))
    if kind == "pair":
        return {"kind": kind, "w": w, "h": h, "d": 8 * _log_int(rng, 2, 32), "bits": rng.choice([8, 12]),
                "tile": rng.choice([64, 64, 32, 16])}
    if kind == "upsample":
        return {"kind": kind, "w": w // 2, "h": h // 2}
    if kind == "cache":
        up = rng.uniform(1.0, 1.3)
        return {"kind": kind, "w": w, "h": h, "cw": int(w * up), "ch": int(h * up), "ratio": rng.choice([0.5, 1.0, 2.0])}
    w, h = max(520, w // 2), max(390, h // 2)
    if kind == "capture":
        return {"kind": kind, "w": w, "h": h, "others": rng.randrange(2, 11), "tile": rng.choice([64, 32])}
    if kind == "resume":
        return {"kind": kind, "w": w, "h": h, "cams": rng.randrange(2, 6), "level": rng.choice([2, 3, 4])}
    if kind == "pyramid":  # multiples of four, as sensors are: the skip mask of an odd second layer can leave a pixel no range
        return {"kind": kind, "w": w // 4 * 4, "h": h // 4 * 4, "cams": rng.randrange(2, 6)}
    if kind == "stereo":
        return {"kind": kind, "sw": w + rng.randrange(1, 60), "sh": h + rng.randrange(1, 40), "w": w, "h": h}
    return {"kind": kind, "w": w, "h": h, "d": _log_int(rng, 24, 192)}


# ---------------- inputs ----------------

def _gen(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed((seed * 1000003 + salt * 7919 + 17) & 0x7FFFFFFF)
    return g


def _texture(h, w, g, top):
    """A 1/f-spectrum texture in [0, top] (2.5 standard deviations to either side of the middle)."""
    spec = torch.fft.rfft2(torch.randn((h, w), generator=g, device=DEV))
    f = torch.sqrt(torch.fft.fftfreq(h, device=DEV)[:, None] ** 2 + torch.fft.rfftfreq(w, device=DEV)[None, :] ** 2)
    f[0, 0] = 1.0
    spec = spec / f
    spec[0, 0] = 0.0
    img = torch.fft.irfft2(spec, s=(h, w))
    return (img / (5.0 * img.std()) + 0.5).clamp_(0.0, 1.0) * top


def _planar(h, w, g, segments=6):
    """Six planar segments (Voronoi cells) with values in [0, 1]."""
    r = torch.rand((segments, 5), generator=g, device=DEV).tolist()
    yy = torch.arange(h, device=DEV, dtype=torch.float32)[:, None]
    xx = torch.arange(w, device=DEV, dtype=torch.float32)[None, :]
    best = torch.full((h, w), float("inf"), device=DEV)
    out = torch.zeros((h, w), device=DEV)
    for cy, cx, a, b, c in r:
        d2 = (yy - cy * h) ** 2 + (xx - cx * w) ** 2
        val = (0.1 + 0.8 * a) + 0.2 * (b - 0.5) * (xx / w - cx) + 0.2 * (c - 0.5) * (yy / h - cy)
        near = d2 < best
        best = torch.where(near, d2, best)
        out = torch.where(near, val, out)
    return out.clamp_(0.0, 1.0)


def _pair(h, w, d, seed, top):
    """Left and right views of a planar scene whose disparities span [0, d - 1]: the nearest surface wins, holes repeat the
    last pixel, both views with noise of two digital numbers."""
    g = _gen(seed)
    left = _texture(h, w, g, top).round_()
    disp = (_planar(h, w, g) * (d - 1)).round_().to(torch.int64)
    xr = torch.arange(w, device=DEV)[None, :] - disp
    key = torch.where(xr >= 0, disp * 8192 + left.to(torch.int64), torch.full_like(disp, -1))
    right = torch.full((h, w), -1, dtype=torch.int64, device=DEV)
    right.scatter_reduce_(1, xr.clamp_(min=0), key, "amax")
    idx = torch.where(right >= 0, torch.arange(w, device=DEV)[None, :], torch.zeros_like(right))
    idx = torch.cummax(idx, dim=1).values
    right = torch.gather(right, 1, idx).clamp_(min=0) % 8192
    noise = torch.randn((2, h, w), generator=g, device=DEV) * 2.0
    return [(v + n).round_().clamp_(0, top) for v, n in zip((left, right.to(torch.float32)), noise)]


def _rgba_grey(y):
    out = torch.full((*y.shape, 4), 128, dtype=torch.uint8, device=DEV)
    out[..., 0] = y.to(torch.uint8)
    out[..., 3] = 255
    return out


def _calib(f, cx, cy, t):
    return api.CalibData(np.array([f, 0, cx, 0, f, cy, 0, 0, 1], np.float32), np.asarray(t, np.float32),
                         np.eye(3, dtype=np.float32).reshape(9))


def _colour_capture(case, seed):
    """A colour capture: reference camera and translated cameras, textures per channel, a planar scene at 0.4-6 m with its
    right border at the far end."""
    w, h, cams = case["w"], case["h"], case["cams"]
    g = _gen(seed)
    rnd = np.random.default_rng(seed)
    f = 0.75 * w
    z = _planar(h, w, g) * 5600.0 + 400.0
    z[:, int(w * 0.9):] = 6000.0
    z_inv = 1.0 / z.clamp_(400.0, 6000.0)
    chans = [_texture(h, w, g, 255.0) for _ in range(3)]
    yy = torch.arange(h, device=DEV, dtype=torch.float32)[:, None]
    xx = torch.arange(w, device=DEV, dtype=torch.float32)[None, :]
    images, calibs = [], []
    for k in range(cams):
        b, ang = (0.0, 0.0) if k == 0 else (rnd.uniform(8.0, 40.0), rnd.uniform(0.0, 2.0 * math.pi))
        t = np.array([b * math.cos(ang), b * math.sin(ang), 0.0], np.float32)
        sx = (xx - f * float(t[0]) * z_inv).round_().clamp_(0, w - 1).to(torch.int64)
        sy = (yy - f * float(t[1]) * z_inv).round_().clamp_(0, h - 1).to(torch.int64)
        img = torch.full((h, w, 4), 255, dtype=torch.uint8, device=DEV)
        for c in range(3):
            v = chans[c][sy, sx] + torch.randn((h, w), generator=g, device=DEV) * 1.5
            img[..., c] = v.round_().clamp_(0, 255).to(torch.uint8)
        images.append(img)
        calibs.append(_calib(f, w / 2.0, h / 2.0, -t))
    return images, calibs, z


def _module_capture(case, seed):
    """A reference module and others, half wide (1.0-1.3x its focal length) and half tele (2.2-2.7x), crops of 1-6 MP for a
    2080x1560 reference and in proportion otherwise, disparity ranges of 64 to 192 planes in random directions."""
    w, h, others = case["w"], case["h"], case["others"]
    g = _gen(seed)
    rnd = np.random.default_rng(seed)
    near, f0, cx0, cy0 = 400.0, 0.9 * w, (w - 1) / 2.0, (h - 1) / 2.0
    H3, W3 = 3 * h, 3 * w
    tex = _texture(H3, W3, g, 255.0)
    z_inv = 1.0 / (_planar(H3, W3, g) * (6000.0 - near) + near).clamp_(near, 6000.0)

    def scene(x, y):
        xi, yi = (x + w).round().clamp_(0, W3 - 1).to(torch.int64), (y + h).round().clamp_(0, H3 - 1).to(torch.int64)
        return tex[yi, xi], z_inv[yi, xi]

    def noisy(v):
        return _rgba_grey((v + torch.randn(v.shape, generator=g, device=DEV) * 1.5).round_().clamp_(0, 255))

    def grid(hh, ww):
        return (torch.arange(ww, device=DEV, dtype=torch.float32)[None, :].expand(hh, ww),
                torch.arange(hh, device=DEV, dtype=torch.float32)[:, None].expand(hh, ww))

    images, calibs = [noisy(scene(*grid(h, w))[0])], [_calib(f0, cx0, cy0, np.zeros(3))]
    for k in range(others):
        s = rnd.uniform(2.2, 2.7) if k >= others // 2 else rnd.uniform(1.0, 1.3)
        hk = max(8, int(round(math.sqrt(rnd.uniform(1.0, 6.0) * 0.75e6 * w * h / (2080.0 * 1560.0)))))
        wk, fk = max(8, int(round(hk * 4.0 / 3.0))), f0 * s
        b, ang = float(rnd.choice([64, 96, 128, 192])) * near / fk, rnd.uniform(0, 2 * math.pi)
        t = np.array([b * math.cos(ang), b * math.sin(ang), 0.0], np.float32)
        cxk, cyk = (wk - 1) / 2.0, (hk - 1) / 2.0
        u, v = grid(hk, wk)
        x, y = cx0 + f0 * (u - cxk) / fk, cy0 + f0 * (v - cyk) / fk
        for _ in range(2):
            zi = scene(x, y)[1]
            x = cx0 + f0 * ((u - cxk) / fk - float(t[0]) * zi)
            y = cy0 + f0 * ((v - cyk) / fk - float(t[1]) * zi)
        images.append(noisy(scene(x, y)[0]))
        calibs.append(_calib(fk, cxk, cyk, -t))
    return images, calibs, near


def _smooth_depth(h, w, g):
    """A depth map in mm as the stage leaves it: planar patches at 0.4-6 m."""
    return _planar(h, w, g) * 5600.0 + 400.0


def _aligned(sw, sh, dw, dh, seed):
    """A small rotation and tilt between a dw x dh view and a sw x sh module, and a radial lens table."""
    rnd = np.random.default_rng(seed)
    fa = 1.1 * dw
    ka = np.array([[fa, 0, dw / 2.0], [0, fa, dh / 2.0], [0, 0, 1]])
    kb = np.array([[fa * 1.02, 0, sw / 2.0 + 3.5], [0, fa * 1.02, sh / 2.0 - 2.25], [0, 0, 1]])
    a, tx, ty = np.deg2rad(rnd.uniform(-0.8, 0.8)), *np.deg2rad(rnd.uniform(-0.3, 0.3, 2))
    rz = np.array([[math.cos(a), -math.sin(a), 0], [math.sin(a), math.cos(a), 0], [0, 0, 1]])
    rx = np.array([[1, 0, 0], [0, math.cos(tx), -math.sin(tx)], [0, math.sin(tx), math.cos(tx)]])
    ry = np.array([[math.cos(ty), 0, math.sin(ty)], [0, 1, 0], [-math.sin(ty), 0, math.cos(ty)]])
    lut = (1.0 + 4e-9 * np.arange(4096, dtype=np.float64) ** 2).astype(np.float32)
    s = np.float32(3000.0 / (0.5 * math.hypot(sw, sh)))
    return api.AlignedCalib(H=(kb @ rz @ rx @ ry @ np.linalg.inv(ka)).astype(np.float32), lut=lut, cx=np.float32(sw / 2.0),
                            cy=np.float32(sh / 2.0), sx=s, sy=s)


def _upsample_inputs(case, seed):
    w, h, g = case["w"], case["h"], _gen(seed)
    guide = torch.stack([_texture(2 * h, 2 * w, g, 255.0) for _ in range(3)] + [torch.full((2 * h, 2 * w), 255.0, device=DEV)], -1)
    depth = _smooth_depth(h, w, g) + torch.randn((h, w), generator=g, device=DEV) * 5.0
    return depth.contiguous(), torch.rand((h, w), generator=g, device=DEV), guide.round_().to(torch.uint8).contiguous()


def _cache_inputs(case, seed):
    g = _gen(seed)
    depth = _smooth_depth(case["h"], case["w"], g) + torch.randn((case["h"], case["w"]), generator=g, device=DEV) * 5.0
    dims = (max(8, int(case["cw"] * case["ratio"])), max(8, int(case["ch"] * case["ratio"])))
    # the region of an export: the whole level but for a border
    rect = (dims[0] // 50, dims[1] // 40, dims[0] - dims[0] // 60, dims[1] - dims[1] // 70)
    return depth.contiguous(), rect, dims


def _stereo_inputs(case, seed):
    g = _gen(seed)
    src = torch.ones((case["sh"], case["sw"], 4), device=DEV)
    for c in range(3):
        src[..., c] = _texture(case["sh"], case["sw"], g, 1.0) * (0.4 + 0.2 * c)
    return src, _aligned(case["sw"], case["sh"], case["w"], case["h"], seed), [0.52, 1.0, 0.61], 1.37


def _census_inputs(case, seed):
    return [_rgba_grey(v) for v in _pair(case["h"], case["w"], case["d"], seed, 255.0)]


def _pinned(h, w):
    return torch.empty((h, w), dtype=torch.float32).pin_memory()


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "ctx": api.Context(0)}
    if kind == "pair":
        w, h, d = case["w"], case["h"], case["d"]
        views = _pair(h, w, d, seed, 255.0 if case["bits"] == 8 else 4095.0)
        if case["bits"] == 8:
            s["images"] = [_rgba_grey(v) for v in views]
        else:  # the cameras' samples; the byte images are made from them in every pass
            s["samples"] = [v.to(torch.int16) for v in views]
            s["images"] = [torch.empty((h, w, 4), dtype=torch.uint8, device=DEV) for _ in views]
        f, base = 1000.0, 100.0
        s.update(gray=[1, 1], calibs=[_calib(f, w / 2.0, h / 2.0, [0, 0, 0]), _calib(f, w / 2.0, h / 2.0, [-base, 0, 0])],
                 near=float(np.float32(f * base / (d - 1))), far=1e30, index=0, prev=None, out=_pinned(h, w),
                 params=api.StereoParams(scale=1, tile=case["tile"], skip_mode=0, plane_density=1.0))
    elif kind == "capture":
        s["images"], s["calibs"], s["near"] = _module_capture(case, seed)
        s.update(gray=[1] * len(s["images"]), far=1e30, index=0, prev=None, out=_pinned(case["h"], case["w"]),
                 params=api.StereoParams(scale=1, tile=case["tile"], skip_mode=0, plane_density=1.0))
    elif kind == "resume":
        s["images"], s["calibs"], z = _colour_capture(case, seed)
        p = api.StereoParams.l16_pyramid()[case["level"]]
        ph, pw = -(-case["h"] // (2 * p.scale)), -(-case["w"] // (2 * p.scale))
        ys = (torch.arange(ph, device=DEV) * 2 * p.scale + p.scale).clamp_(max=case["h"] - 1)
        xs = (torch.arange(pw, device=DEV) * 2 * p.scale + p.scale).clamp_(max=case["w"] - 1)
        g = _gen(seed, 1)
        prev = z[ys][:, xs] * (1.0 + 0.02 * torch.randn((ph, pw), generator=g, device=DEV))
        wrong = torch.rand((2, ph, pw), generator=g, device=DEV)  # a few mismatches, as a coarse layer leaves them
        prev = torch.where(wrong[0] < 0.02, 400.0 + 5600.0 * wrong[1], prev)
        s.update(gray=[0] * case["cams"], near=200.0, far=640000.0, index=case["level"], params=p,
                 prev=api.DenseLayer.from_depth(prev.clamp_(min=300.0).cpu().numpy(), ctx=s["ctx"]),
                 out=_pinned(-(-case["h"] // p.scale), -(-case["w"] // p.scale)))
    elif kind == "pyramid":
        s["images"], s["calibs"], _ = _colour_capture(case, seed)
        h, w = case["h"], case["w"]
        g = _gen(seed, 2)
        guide = torch.stack([_texture(2 * h, 2 * w, g, 255.0) for _ in range(4)], -1).round_().to(torch.uint8).contiguous()
        s.update(gray=[0] * case["cams"], guide=guide, depth=_pinned(h, w), out=_pinned(2 * h, 2 * w))
    elif kind == "upsample":
        s["depth"], s["conf"], s["guide"] = _upsample_inputs(case, seed)
        s["outs"] = [torch.empty((2 * case["h"], 2 * case["w"]), device=DEV) for _ in range(2)]
    elif kind == "cache":
        s["depth"], s["rect"], s["dims"] = _cache_inputs(case, seed)
        s["cache"] = api.DepthImageCache((case["cw"], case["ch"]), device=True, ctx=s["ctx"])
    elif kind == "stereo":
        s["src"], s["ac"], s["neutral"], s["gain"] = _stereo_inputs(case, seed)
    else:
        s["left"], s["right"] = _census_inputs(case, seed)
    torch.cuda.synchronize()
    return s


def _read_depth(s, layer, out):
    s["ctx"].check(s["ctx"].lib.lux_layer_read(layer.handle, _lib.FIELD_DEPTH, out.data_ptr(), out.numel() * 4))
    return out


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind in ("pair", "capture", "resume"):
        if "samples" in s:
            for v, im in zip(s["samples"], s["images"]):
                api.image_from_grey16(v, 12, ctx=ctx, out=im)
        layer = api.DenseLayer.compute(s["images"], s["gray"], s["calibs"], s["near"], s["far"], s["params"], index=s["index"],
                                       prev=s["prev"], prefilter=True, ctx=ctx)
        out = _read_depth(s, layer, s["out"])
        layer.close()
        return out
    if kind == "pyramid":
        layers = api.DenseStereoPyramid.run(s["images"], s["gray"], s["calibs"], ctx=ctx)
        h, w = case["h"], case["w"]
        g = _lib.Img(s["guide"].data_ptr(), 2 * w, 2 * h, 2 * w, 1)
        ctx.check(ctx.lib.lux_sgm_upsample(ctx.handle, layers[5].device_ptr(_lib.FIELD_DEPTH), w, h, 1, ctypes.byref(g), w, h, 12.0,
                                           2, None, s["out"].data_ptr(), None))
        _read_depth(s, layers[5], s["depth"])
        for layer in layers:
            layer.close()
        return {"layer": s["depth"], "full": s["out"]}
    if kind == "upsample":
        h, w = case["h"], case["w"]
        g = _lib.Img(s["guide"].data_ptr(), 2 * w, 2 * h, 2 * w, 1)
        ctx.check(ctx.lib.lux_sgm_upsample_noalloc(ctx.handle, s["depth"].data_ptr(), w, h, ctypes.byref(g), w, h, 12.0, 2,
                                                   s["conf"].data_ptr(), s["outs"][0].data_ptr(), s["outs"][1].data_ptr()))
        return {"depth": s["outs"][0], "confidence": s["outs"][1]}
    if kind == "cache":
        s["cache"].Set(s["depth"])
        return {"cache": s["cache"].Current, "region": s["cache"].Fetch(s["rect"], s["dims"])}
    if kind == "stereo":
        image, yuv = api.StereoImage.create(s["src"], case["w"], case["h"], s["ac"], 3, s["neutral"], gain=s["gain"], keep_yuv=True,
                                            ctx=ctx)
        return {"image": image, "yuv": yuv}
    return api.CensusStereo.compute(s["left"], s["right"], case["d"], ctx=ctx)


# ---------------- the work a pass cannot do without ----------------

# integer operations of a pixel and plane: the 3x3 block's differences, caps and sums; a path's minima, sums and minimum
COST_OPS, PATH_OPS, CENSUS_OPS = 28, 9, 2


def work(case):
    kind, w, h = case["kind"], case["w"], case["h"]
    px = w * h
    if kind == "pair":
        return {"bytes": px * (2 * (4 if case["bits"] == 8 else 2) + 4), "flops": px * case["d"] * (COST_OPS + 8 * PATH_OPS)}
    if kind == "capture":  # module crops average 3.5 MP for a 3.24 MP reference; about 160 planes
        return {"bytes": px * (4 + 4 * 1.08 * case["others"] + 4), "flops": px * 160 * (COST_OPS * case["others"] + 8 * PATH_OPS)}
    if kind == "resume":  # about 60 planes a pixel are searched; the cameras are read whole by the box filter
        lp = (w >> (5 - case["level"])) * (h >> (5 - case["level"]))
        return {"bytes": px * 4 * case["cams"] + lp * 8, "flops": lp * 60 * (3 * COST_OPS * (case["cams"] - 1) + 8 * PATH_OPS)}
    if kind == "pyramid":
        return {"bytes": px * 4 * case["cams"] + 4 * px * 8 + px * 4,
                "flops": px * 1.34 * 100 * (3 * COST_OPS * (case["cams"] - 1) + 8 * PATH_OPS)}
    if kind == "upsample":
        return {"bytes": px * (4 + 4 + 16 + 32), "flops": px * 4 * 120}
    if kind == "cache":
        rect, cache = _rect_of(case), case["cw"] * case["ch"]
        out = (rect[2] - rect[0]) * (rect[3] - rect[1])
        return {"bytes": 4 * (px + 2 * cache + out), "flops": 4 * (cache + out)}
    if kind == "stereo":
        return {"bytes": 16 * case["sw"] * case["sh"] + px * 20, "flops": px * 400}
    return {"bytes": px * 12, "flops": px * case["d"] * (CENSUS_OPS + 8 * PATH_OPS)}


def _rect_of(case):
    dims = (max(8, int(case["cw"] * case["ratio"])), max(8, int(case["ch"] * case["ratio"])))
    return (dims[0] // 50, dims[1] // 40, dims[0] - dims[0] // 60, dims[1] - dims[1] // 70)


# ---------------- the same results in 64 bits ----------------

def exact(case, seed):
    """None for the dense solves: their depths are the planes that minimise sums of quantised costs along a fixed traversal
    of the image, choices among given values rather than computed numbers."""
    kind = case["kind"]
    if kind == "upsample":
        return _exact_upsample(case, seed)
    if kind == "cache":
        return _exact_cache(case, seed)
    if kind == "stereo":
        return {"image": None, "yuv": _exact_stereo(case, seed)}
    if kind == "census":
        return _exact_census(case, seed)
    return None


def _exact_upsample(case, seed):
    depth, conf, guide = _upsample_inputs(case, seed)
    h, w = case["h"], case["w"]
    g = guide.to(torch.float64)
    taps = [-0.0625, 0.5625, 0.5625, -0.0625]  # the cubic at half a pixel
    rows = [(2 * torch.arange(h, device=DEV) - 1 + i).clamp_(0, 2 * h - 1) for i in range(4)]
    cols = [(2 * torch.arange(w, device=DEV) - 1 + i).clamp_(0, 2 * w - 1) for i in range(4)]
    v = sum(t * g[r] for t, r in zip(taps, rows))
    low = sum(t * v[:, c] for t, c in zip(taps, cols)).round().clamp_(0, 255)[..., :3]
    k = 0.5 / 144.0
    y, x = torch.arange(2 * h, device=DEV), torch.arange(2 * w, device=DEV)

    def weight(pos, i):
        return torch.where((pos - 0.5 - 2 * i).abs() >= 1.0, 1.0 / 3.0, 1.0).to(torch.float64)

    y0, x0 = torch.where(y > 0, (y - 1) // 2, 0), torch.where(x > 0, (x - 1) // 2, 0)
    num = {"depth": 0.0, "confidence": 0.0}
    den = torch.zeros((2 * h, 2 * w), dtype=torch.float64, device=DEV)
    maps = {"depth": 1.0 / depth.to(torch.float64), "confidence": conf.to(torch.float64)}
    for j in range(2):
        iy = (y0 + j).clamp(0, h - 1)
        for i in range(2):
            ix = (x0 + i).clamp(0, w - 1)
            d = g[..., :3] - low[iy][:, ix]
            e = torch.exp2(torch.clamp(-(d * d).sum(-1) * k, min=-126.0)) + 1e-8
            wt = e * weight(y, iy)[:, None] * weight(x, ix)[None, :]
            den = den + wt
            for n in num:
                num[n] = num[n] + wt * maps[n][iy][:, ix]
    return {"depth": den / num["depth"], "confidence": num["confidence"] / den}


def _exact_cache(case, seed):
    depth, rect, dims = _cache_inputs(case, seed)
    d, (h, w), (cw, ch) = depth.to(torch.float64), (case["h"], case["w"]), (case["cw"], case["ch"])

    def nearest(step, off, n_out, n_in):
        i = torch.arange(n_out, device=DEV, dtype=torch.int64)
        return ((int(step * 65536.0) * i + int(off * 65536.0)) >> 16).clamp_(0, n_in - 1)

    cache = d[nearest(h / ch, 0.0, ch, h)][:, nearest(w / cw, 0.0, cw, w)].clamp(max=100000.0)
    sx, sy = cw / dims[0], ch / dims[1]
    x0, y0, x1, y1 = rect
    if sx == 1.0 and sy == 1.0:
        return {"cache": cache, "region": cache[y0:y1, x0:x1]}
    wx0, wy0 = max(math.floor(x0 * sx), 0), max(math.floor(y0 * sy), 0)
    wx1, wy1 = min(math.ceil(x1 * sx), cw), min(math.ceil(y1 * sy), ch)
    win = cache[wy0:wy1, wx0:wx1]
    ys = nearest(sy, (y0 + 0.5) * sy - wy0, y1 - y0, wy1 - wy0)
    xs = nearest(sx, (x0 + 0.5) * sx - wx0, x1 - x0, wx1 - wx0)
    return {"cache": cache, "region": win[ys][:, xs]}


def _exact_stereo(case, seed):
    src, ac, neutral, gain = _stereo_inputs(case, seed)
    w, h, sw, sh = case["w"], case["h"], case["sw"], case["sh"]
    H = torch.tensor(np.asarray(ac.H, np.float64).reshape(9), device=DEV)
    lut = torch.tensor(np.asarray(ac.lut, np.float64), device=DEV)
    yy = torch.arange(h, device=DEV, dtype=torch.float64)[:, None]
    xx = torch.arange(w, device=DEV, dtype=torch.float64)[None, :]
    den = H[6] * xx + H[7] * yy + H[8]
    dx = (H[0] * xx + H[1] * yy + H[2]) / den - float(ac.cx)
    dy = (H[3] * xx + H[4] * yy + H[5]) / den - float(ac.cy)
    r = torch.sqrt((float(ac.sx) * dx) ** 2 + (float(ac.sy) * dy) ** 2)
    lu = lut[r.to(torch.int64).clamp_(max=4095)]
    px = torch.trunc((float(ac.cx) - 2.0 + lu * dx) * 64.0).to(torch.int64)
    py = torch.trunc((float(ac.cy) - 2.0 + lu * dy) * 64.0).to(torch.int64)
    p = np.arange(64)[:, None] / 64.0 - (np.arange(6)[None, :] - 2.0)
    taps = np.sinc(p) * np.sinc(p / 3.0) * (np.abs(p) < 3.0)
    taps = torch.tensor(taps / taps.sum(1, keepdims=True), device=DEV)
    i, j = px >> 6, py >> 6
    s = src.to(torch.float64) * gain
    acc = torch.zeros((h, w, 4), dtype=torch.float64, device=DEV)
    for b in range(6):
        row = torch.zeros_like(acc)
        yb = (j + b).clamp(0, sh - 1)
        for a in range(6):
            row += s[yb, (i + a).clamp(0, sw - 1)] * taps[px & 63, a][..., None]
        acc += row * taps[py & 63, b][..., None]
    inside = (j < sh) & (j + 6 > 0) & (i < sw) & (i + 6 > 0)
    acc = torch.where(inside[..., None], acc, torch.zeros_like(acc))
    # the luma basis of the AR1335 and the two chroma rows scaled to its length
    a, b, c = (float(np.uint32(u).view(np.float32)) for u in (0x3E5CB924, 0x3EDD5758, 0x3EB44C16))
    ix, iy, iz = (1.0 / v for v in neutral)
    u = np.array([(-b * b - (c + a) * c) * ix, (a - c) * b * iy, ((c + a) * a + b * b) * iz])
    t = np.array([-b * ix, (c + a) * iy, -b * iz])
    luma = np.array([a, b, c])
    n = np.linalg.norm(luma)
    m = torch.tensor(np.stack([luma, u / np.linalg.norm(u) * n, t / np.linalg.norm(t) * n]), device=DEV)
    yuv = acc[..., :3] @ m.T
    yuv = 255.0 * torch.sign(yuv) * yuv.abs() ** (1.0 / 2.2)
    yuv[..., 1:] += 128.0
    return torch.cat([yuv, torch.ones((h, w, 1), dtype=torch.float64, device=DEV)], -1)


def _exact_census(case, seed):
    left, right = [v[..., 0].to(torch.int32) for v in _census_inputs(case, seed)]
    h, w, D = case["h"], case["w"], case["d"]
    P1, P2, big = 10, 120, 1 << 14
    ys, xs = torch.arange(h, device=DEV), torch.arange(w, device=DEV)

    def census(im):
        out = torch.zeros((h, w), dtype=torch.int64, device=DEV)
        bit = 0
        for dy in range(-3, 4):
            for dx in range(-4, 5):
                if dx == 0 and dy == 0:
                    continue
                nb = im[(ys + dy).clamp(0, h - 1)][:, (xs + dx).clamp(0, w - 1)]
                out |= (nb < im).to(torch.int64) << bit
                bit += 1
        return out

    ones = torch.tensor([bin(i).count("1") for i in range(1 << 16)], dtype=torch.uint8, device=DEV)
    cl, cr = census(left), census(right)
    cost = torch.full((h, w, D), 62, dtype=torch.int16, device=DEV)
    for d in range(min(D, w)):
        x = cl[:, d:] ^ cr[:, : w - d]
        cost[:, d:, d] = sum(ones[(x >> (16 * k)) & 0xFFFF] for k in range(4)).to(torch.int16)
    total = torch.zeros((h, w, D), dtype=torch.int16, device=DEV)

    def step(q, c):
        m = q.amin(1, keepdim=True)
        n = torch.minimum(q, m + P2)
        n[:, 1:] = torch.minimum(n[:, 1:], q[:, :-1] + P1)
        n[:, :-1] = torch.minimum(n[:, :-1], q[:, 1:] + P1)
        return c + n - m

    for dx, dy in ((1, 0), (-1, 0), (0, 1), (0, -1), (1, 1), (-1, -1), (1, -1), (-1, 1)):
        prev = None
        along_rows = dy != 0
        count = h if along_rows else w
        order = range(count) if (dy if along_rows else dx) > 0 else range(count - 1, -1, -1)
        for k in order:
            c = cost[k] if along_rows else cost[:, k]
            if prev is None:
                new = c.clone()
            elif dx == 0 or not along_rows:
                new = step(prev, c)
            else:
                new = c.clone()
                if dx > 0:
                    new[1:] = step(prev[:-1], c[1:])
                else:
                    new[:-1] = step(prev[1:], c[:-1])
            if along_rows:
                total[k] += new
            else:
                total[:, k] += new
            prev = new
    key = total.to(torch.int32) * 512 + torch.arange(D, device=DEV, dtype=torch.int32)
    best = key.amin(2)
    dl, sb = (best & 511).to(torch.int64), (best >> 9).to(torch.float64)
    lo = torch.gather(total, 2, (dl - 1).clamp(min=0)[..., None])[..., 0].to(torch.float64)
    hi = torch.gather(total, 2, (dl + 1).clamp(max=D - 1)[..., None])[..., 0].to(torch.float64)
    den = 2.0 * (lo - 2.0 * sb + hi)
    out = dl.to(torch.float64) + torch.where((dl > 0) & (dl < D - 1) & (den > 0), (lo - hi) / den.clamp(min=1e-9), 0.0)
    dr = torch.full((h, w), big * 512, dtype=torch.int32, device=DEV)
    for d in range(min(D, w)):
        dr[:, : w - d] = torch.minimum(dr[:, : w - d], key[:, d:, d])
    xr = xs[None, :] - dl
    back = torch.gather((dr & 511).to(torch.int64), 1, xr.clamp(min=0))
    return torch.where((xr < 0) | ((dl - back).abs() > 1), -1.0, out)
