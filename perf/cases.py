"""The workloads whose speed this repository is measured by, through its public entry points.

A case is a dict of plain values: `kind` says which calls a pass makes, the rest are sizes and
options. The kinds are the calls a renderer makes per frame:

    frame    Denoiser.Denoise + Tonemapping.CalculateExposure of one camera stream
    batch    Context.submit_batch over one frame each of several camera streams
    scatter  Volumetric.ProcessScattering (the froxel volume handed over first, as its
             producer does every frame)
    post     ImageComposition.Finalize + Bloom.Apply
    full     all of them in a renderer's order

The inputs are a small ray-cast scene (ground, wall, sky, spheres; the camera translates, some
spheres move) with log-normal path-tracer noise and fireflies, in the G-buffer's own formats, and
the history a stream has after some frames. Everything is made on the GPU from the seed.

`exact` evaluates the same chain in 64 bits with plain torch, without this repository's code; it
rounds only what the chain stores as 8-bit codes (the gradients).
"""
import math
import weakref

import numpy as np
import torch

from raytracedgl1_gb300 import _native as N
from raytracedgl1_gb300.denoiser import Bloom, Context, Denoiser, ImageComposition, Stream, Tonemapping, Volumetric

DEV = "cuda"
F64 = torch.float64
MAX_RAY = 10000.0
SKY_DEPTH = 20000.0
NEAR, FAR = 0.1, 1000.0
# noise sigma, firefly share and factor; "tame" keeps squared luminances inside the reference formats' fp16 moments
SIGMA = {"tame": (0.6, 0.001, 5.0), "mild": (1.0, 0.001, 100.0), "harsh": (1.5, 0.01, 50.0)}


# ------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------
def _frame(name, w, h, storage, iterations=4, **more):
    return {"name": name, "kind": "frame", "width": w, "height": h, "storage": storage, "iterations": iterations,
            "flags": 0, "noise": "mild", **more}


def listed():
    return [
        # a thumbnail or inset view: launches and latency count
        _frame("frame 320x180 fp16", 320, 180, "fp16"),
        # the parity configuration: full precision, five a-trous passes
        _frame("frame 640x360 fp32", 640, 360, "fp32", 5),
        # a laptop window with an odd height, bf16 storage
        _frame("frame 1366x767 bf16", 1366, 767, "bf16"),
        # the everyday case and the benchmark's: 1080p in 16-bit storage
        _frame("frame 1920x1080 fp16", 1920, 1080, "fp16", 5),
        # the reference's own formats, the default of a stream
        _frame("frame 1920x1080 ref", 1920, 1080, "ref", noise="tame"),
        # IEEE arithmetic asked for: bit-reproducible frames
        _frame("frame 1280x720 exact", 1280, 720, "fp32", 4, flags=N.FLAG_EXACT_MATH),
        # the largest: 4K with heavy noise, bf16 storage
        _frame("frame 3840x2160 bf16", 3840, 2160, "bf16", 5, noise="harsh"),
        # a server's step: cameras of mixed sizes in one call
        {"name": "batch of 8 fp16", "kind": "batch", "sizes": "640x360 640x360 640x360 640x360 1280x720 1280x720 1920x1080 2560x1440",
         "storage": "fp16", "iterations": 5, "flags": 0, "noise": "mild"},
        # volumetric lighting at 1080p
        {"name": "scatter 1920x1080", "kind": "scatter", "width": 1920, "height": 1080, "mode": "volumetric"},
        # exposure, tonemapping and bloom at 1440p
        {"name": "post 2560x1440 fp16", "kind": "post", "width": 2560, "height": 1440, "storage": "fp16"},
        # a whole frame of a renderer at 1440p, an ultrawide with an odd height
        {"name": "full 2560x1079 fp16", "kind": "full", "width": 2560, "height": 1079, "storage": "fp16", "iterations": 4, "flags": 0,
         "noise": "mild", "mode": "volumetric"},
    ]


def _draw_size(rng, lo, hi):
    px = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    aspect = rng.choice([16 / 9, 16 / 9, 4 / 3, 21 / 9, 1.0, 9 / 16])
    w = max(64, int(math.sqrt(px * aspect)) // 2 * 2)
    return w, max(36, min(int(px / w), hi // w))


def draw(rng):
    kind = rng.choice(["frame"] * 6 + ["batch", "scatter", "post", "full"])
    storage = rng.choice(["ref", "fp32", "fp16", "fp16", "bf16"])
    noise = "tame" if storage == "ref" else rng.choice(["mild", "harsh"])
    iterations = rng.choice([3, 4, 4, 5, 5])
    if kind == "batch":
        sizes = ["%dx%d" % _draw_size(rng, 320 * 180, 1920 * 1080) for _ in range(rng.randint(2, 8))]
        return {"kind": kind, "sizes": " ".join(sizes), "storage": storage, "iterations": iterations, "flags": 0, "noise": noise}
    w, h = _draw_size(rng, 320 * 180, 3840 * 2160 // 2)
    if kind == "scatter":
        return {"kind": kind, "width": w, "height": h, "mode": rng.choice(["volumetric", "volumetric", "simple"])}
    if kind == "post":
        return {"kind": kind, "width": w, "height": h, "storage": storage}
    if kind == "full":
        w, h = _draw_size(rng, 320 * 180, 2560 * 1440)
        return {"kind": kind, "width": w, "height": h, "storage": storage, "iterations": iterations, "flags": 0, "noise": noise,
                "mode": "volumetric"}
    flags = rng.choice([0, 0, 0, 0, N.FLAG_EXACT_MATH, N.FLAG_SKIP_GRADIENTS])
    return {"kind": kind, "width": w, "height": h, "storage": storage, "iterations": iterations, "flags": flags, "noise": noise}


# ------------------------------------------------------------------------------------------
# texel codecs of the planes, in torch
# ------------------------------------------------------------------------------------------
def _e5_encode(c):
    """EXT_texture_shared_exponent (9-bit mantissas, bias 15) of non-negative (..., 3) floats, as int32."""
    c = c.double().clamp(0.0, 65408.0)
    m = c.amax(-1).clamp_min(2.0 ** -40)
    e = (torch.floor(torch.log2(m)).clamp_min(-16.0) + 16.0).clamp(0.0, 31.0)
    e = torch.where(torch.floor(m * torch.exp2(24.0 - e) + 0.5) >= 512.0, e + 1.0, e)
    q = torch.floor(c * torch.exp2(24.0 - e).unsqueeze(-1) + 0.5).long()
    v = (e.long() << 27) | (q[..., 2] << 18) | (q[..., 1] << 9) | q[..., 0]
    return torch.where(v >= 2 ** 31, v - 2 ** 32, v).int()


def _e5_decode(v):
    v = v.long() & 0xFFFFFFFF
    s = torch.exp2((v >> 27).double() - 24.0)
    return torch.stack([(v & 511).double() * s, ((v >> 9) & 511).double() * s, ((v >> 18) & 511).double() * s], -1)


def _b10_encode(c):
    """B10G11R11: the upper bits of the fp16 pattern (same exponent), truncated."""
    h = c.clamp(0.0, 60000.0).half().view(torch.int16).long()
    v = (h[..., 0] >> 4) | ((h[..., 1] >> 4) << 11) | ((h[..., 2] >> 5) << 22)
    return torch.where(v >= 2 ** 31, v - 2 ** 32, v).int()


def _b10_decode(v):
    v = v.long() & 0xFFFFFFFF
    ch = [((v & 0x7FF) << 4), (((v >> 11) & 0x7FF) << 4), (((v >> 22) & 0x3FF) << 5)]
    return torch.stack([x.short().view(torch.float16).double() for x in ch], -1)


def _normal_encode(n):
    phi = torch.acos(n[..., 2].double().clamp(-1.0, 1.0))
    theta = torch.atan2(n[..., 1].double(), n[..., 0].double()) % (2.0 * math.pi)
    j = torch.floor(phi * 65535.0 / math.pi + 0.5).long().clamp(0, 65535)
    k = torch.floor(theta * 65536.0 / (2.0 * math.pi) + 0.5).long() & 0xFFFF
    v = (j << 16) | k
    return torch.where(v >= 2 ** 31, v - 2 ** 32, v).int()


def _normal_decode(v):
    v = v.long() & 0xFFFFFFFF
    phi = (v >> 16).double() * (math.pi / 65535.0)
    theta = (v & 0xFFFF).double() * (2.0 * math.pi / 65536.0)
    return torch.stack([torch.sin(phi) * torch.cos(theta), torch.sin(phi) * torch.sin(theta), torch.cos(phi)], -1)


def _rgba(c, a=None):
    a = torch.zeros_like(c[..., :1]) if a is None else a.unsqueeze(-1)
    return torch.cat([c, a], -1)


_TEXEL = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}


def _colour(storage, c):
    return _e5_encode(c) if storage == "ref" else _rgba(c).to(_TEXEL[storage])


def _colour64(storage, t):
    return _e5_decode(t) if storage == "ref" else t[..., :3].double()


def _image(storage, c):
    """PRE_FINAL's format."""
    return _b10_encode(c) if storage == "ref" else _rgba(c).to(torch.float32 if storage == "fp32" else torch.float16)


def _image64(storage, t):
    return _b10_decode(t) if storage == "ref" else t[..., :3].double()


# ------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------
def _camera(w, h):
    f = 1.0 / math.tan(math.radians(30.0))
    aspect = w / h
    proj = np.zeros((4, 4))
    proj[0, 0], proj[1, 1], proj[3, 2] = f / aspect, f, -1.0
    proj[2, 2], proj[2, 3] = -FAR / (FAR - NEAR), -FAR * NEAR / (FAR - NEAR)
    step = 2.0 * 20.0 * aspect / (f * w)   # the camera's translation: 2 pixels at distance 10
    return proj, step


def _regular(w, h):
    """Column of the regular layout for every checkerboard texel (the left half holds one colour
    of the checkerboard, the right half the other)."""
    cx = torch.arange(w, device=DEV).view(1, w)
    cy = torch.arange(h, device=DEV).view(h, 1)
    odd = (cx >= w // 2).long()
    return (cx - odd * (w // 2)) * 2 + (odd + cy) % 2, cy.expand(h, w)


def _scene(w, h, seed, noise):
    """Every producer-written plane of one frame, in its storage format, and the clean lighting."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    proj, step = _camera(w, h)
    rx, ry = _regular(w, h)
    f = proj[1, 1]
    dx = ((rx + 0.5) / w * 2.0 - 1.0) / proj[0, 0]
    dy = ((ry + 0.5) / h * 2.0 - 1.0) / f
    d = torch.stack([dx, dy, torch.full_like(dx, -1.0)], -1).float()
    d = d / d.norm(dim=-1, keepdim=True)
    t = torch.full((h, w), SKY_DEPTH, device=DEV)
    n = torch.zeros(h, w, 3, device=DEV)
    n[..., 2] = 1.0
    obj = torch.zeros(h, w, dtype=torch.long, device=DEV)

    def hit(where, tt, nn, k):
        nonlocal t, n, obj
        near = where & (tt > 0.05) & (tt < t)
        t = torch.where(near, tt, t)
        n = torch.where(near.unsqueeze(-1), nn, n)
        obj = torch.where(near, torch.full_like(obj, k), obj)

    tg = 1.5 / d[..., 1].clamp_min(1e-4)
    hit((d[..., 1] > 0.02) & (tg < 60.0), tg, torch.tensor([0.0, -1.0, 0.0], device=DEV), 1)
    tw = -20.0 / d[..., 2]
    hit(d[..., 1] * tw > -5.0, tw, torch.tensor([0.0, 0.0, 1.0], device=DEV), 2)
    balls = torch.rand(10, 5, generator=g, device=DEV)
    lim = float(proj[0, 0])
    for k in range(10):
        b = balls[k]
        z = -5.0 - 11.0 * b[2]
        c = torch.stack([(b[0] * 2.0 - 1.0) * 0.8 * -z / lim, b[1] * 2.5 - 1.2, z])
        r = 0.4 + 0.9 * b[3]
        bq = (d * c).sum(-1)
        disc = bq * bq - ((c * c).sum() - r * r)
        tt = bq - disc.clamp_min(0.0).sqrt()
        p = d * tt.unsqueeze(-1)
        hit(disc > 0.0, tt, (p - c) / r, 3 + k)
    sky = obj == 0
    t = t.half().float()
    pos = d * t.unsqueeze(-1)
    # what the previous frame saw: the camera one step to the left, every fourth object 4 steps on
    moved = torch.where((obj > 2) & (obj % 4 == 0), 4.0 * step, 0.0)
    motion = torch.zeros(h, w, 4, device=DEV)
    motion[..., 0] = torch.where(sky, torch.zeros_like(t), 0.5 * proj[0, 0] * (step + moved) / (-pos[..., 2]))
    mat = torch.rand(16, 4, generator=g, device=DEV)
    m = mat[obj]
    checker = ((torch.floor(pos[..., 0] * 1.5) + torch.floor(pos[..., 2] * 1.5)) % 2.0).abs()
    rough = (0.05 + 0.9 * m[..., 0] * (0.6 + 0.4 * checker)).clamp(0.0, 1.0)
    metal = torch.where(m[..., 1] > 0.7, m[..., 1], torch.zeros_like(rough))
    albedo_cb = (0.15 + 0.8 * m[..., 1:4] * (0.7 + 0.3 * checker.unsqueeze(-1))).clamp(0.0, 1.0)
    light = torch.tensor([0.48, -0.64, 0.6], device=DEV)
    lam = (n * light).sum(-1).clamp_min(0.0)
    clean = {
        "D": (0.1 + 2.0 * lam).unsqueeze(-1) * torch.tensor([1.0, 0.9, 0.75], device=DEV),
        "S": (0.05 + 1.5 * lam * (1.0 - rough)).unsqueeze(-1) * torch.tensor([1.0, 0.95, 0.9], device=DEV),
        "I": (0.15 + 0.3 * (0.5 - 0.5 * n[..., 1])).unsqueeze(-1) * torch.tensor([0.6, 0.8, 1.0], device=DEV),
    }
    sigma, share, factor = SIGMA[noise]

    def noisy(c):
        v = torch.randn(h, w, 3, generator=g, device=DEV).mul_(sigma).exp_()
        fire = torch.where(torch.rand(h, w, 1, generator=g, device=DEV) < share, factor, 1.0)
        return torch.where(sky.unsqueeze(-1), torch.zeros_like(c), c * v * fire)

    unf = {k: _e5_encode(noisy(c)) for k, c in clean.items()}
    albedo = torch.empty(h, w, 3, device=DEV)
    albedo[ry, rx] = torch.where(sky.unsqueeze(-1), torch.tensor([0.4, 0.6, 1.0], device=DEV), albedo_cb)
    ndv = -(n * d).sum(-1)
    grad = torch.where(sky, torch.zeros_like(t), 2.0 / (f * h) * t / ndv.clamp_min(0.05))
    lum = torch.tensor([0.2125, 0.7154, 0.0721], device=DEV)
    gi = torch.stack([(clean["D"] * lum).sum(-1), (clean["S"] * lum).sum(-1)], -1)
    gi = torch.where(sky.unsqueeze(-1), torch.zeros_like(gi), gi * torch.exp(0.3 * torch.randn(h, w, 2, generator=g, device=DEV)))
    # a light that changed on part of the screen
    relit = torch.where(((rx > w * 0.3) & (rx < w * 0.5)).unsqueeze(-1), 1.7, 1.0) * gi
    hit_dist = 0.5 + 15.0 * torch.rand(h, w, generator=g, device=DEV)
    glass = (obj == 5) | (obj == 9)   # split rays: resolved from their neighbours in the final pass
    tp = torch.ones(h, w, 4, device=DEV)
    tp[..., 3] = glass.float()
    emis = torch.zeros(h, w, 3, device=DEV)
    emis[ry, rx] = torch.where((obj == 6).unsqueeze(-1), mat[6, 1:4] * 2.0, torch.zeros(3, device=DEV))
    ndc = torch.empty(h, w, device=DEV)
    ndc[ry, rx] = torch.where(sky, torch.ones_like(t), FAR / (FAR - NEAR) * (1.0 + NEAR / pos[..., 2]))
    mr = torch.stack([torch.floor(metal * 255.0 + 0.5), torch.floor(rough * 255.0 + 0.5)], -1).to(torch.uint8)
    planes = {
        "ALBEDO": _b10_encode(albedo), "IS_SKY": sky.to(torch.uint8), "NORMAL": _normal_encode(n), "METALLIC_ROUGHNESS": mr,
        "DEPTH_WORLD": t.half(), "DEPTH_GRAD": grad.half(), "MOTION": motion.half(), "UNFILTERED_DIRECT": unf["D"],
        "UNFILTERED_SPECULAR": unf["S"], "UNFILTERED_INDIR": unf["I"], "SURFACE_POSITION": _rgba(pos),
        "VIEW_DIRECTION": _rgba(d, hit_dist).half(), "THROUGHPUT": tp.half(), "GRADIENT_INPUTS": gi.half(),
        "GRADIENT_RESHADED": relit.contiguous(), "SCREEN_EMIS_RT": _b10_encode(emis), "DEPTH_NDC": ndc,
    }
    return planes, clean, sky, g


_BOTH_SLOTS = ("NORMAL", "METALLIC_ROUGHNESS", "DEPTH_WORLD", "SURFACE_POSITION", "GRADIENT_INPUTS")


def _history(storage, clean, sky, g):
    """What a stream keeps from the frame before: accumulated colours, moments, history lengths."""
    h, w = sky.shape
    jitter = lambda c: torch.where(sky.unsqueeze(-1), torch.zeros_like(c), c * torch.exp(0.15 * torch.randn(h, w, 3, generator=g, device=DEV)))  # noqa: E731
    dif, spec, ind = jitter(clean["D"]), jitter(clean["S"]), jitter(clean["I"])
    lum = (dif * torch.tensor([0.2125, 0.7154, 0.0721], device=DEV)).sum(-1)
    spread = 0.05 + 0.5 * torch.rand(h, w, generator=g, device=DEV)
    length = torch.floor(torch.exp(5.0 * torch.rand(h, w, 3, generator=g, device=DEV)))   # 1 .. 148
    hl = torch.cat([length, 0.5 + 10.0 * torch.rand(h, w, 1, generator=g, device=DEV)], -1)
    var = lum * lum * spread / length[..., 0]
    mom = torch.stack([lum, lum * lum * (1.0 + spread)], -1)
    texel = torch.float16 if storage == "ref" else _TEXEL[storage]
    out = {
        "DIFF_ACCUM_MOMENTS": mom.to(torch.float16 if storage == "ref" else torch.float32), "ACCUM_HISTORY_LENGTH": hl.to(texel),
        "SPEC_ACCUM_COLOR": _colour(storage, spec), "INDIR_ACCUM": _colour(storage, ind),
        "DIFF_COLOR_HISTORY": _rgba(dif, var if storage in ("ref", "fp32") else None).to(texel),
    }
    gw, gh = (w + 1) // 3, (h + 1) // 3
    out["DIS_GRADIENT_HISTORY"] = torch.randint(0, 40, (gh, gw, 4), generator=g, device=DEV).to(torch.uint8)
    out["GRADIENT_PREV_PIX"] = torch.full((gh, gw), 10, dtype=torch.uint8, device=DEV)
    return out


def _fog(w, h, g):
    x, y, z = N.VOLUME_SIZE
    vol = torch.rand(z * y, x, 4, generator=g, device=DEV) * torch.tensor([0.03, 0.035, 0.04, 0.02], device=DEV)
    prev = torch.rand(h, w, 4, generator=g, device=DEV) * torch.tensor([0.3, 0.35, 0.4, 0.5], device=DEV)
    prev[..., 3] += 0.4
    hist = torch.floor(1.0 + 15.0 * torch.rand(h, w, generator=g, device=DEV))
    return {"SCATTER_VOLUME": vol.half(), "SCATTERING": prev.half(), "SCATTERING_HISTORY": hist.half()}


def _column_major(a, into):
    into[:] = [float(v) for v in np.asarray(a).T.reshape(-1)]


def _frame_params(case, w, h):
    p = N.FrameParams()
    proj, step = _camera(w, h)
    _column_major(np.eye(4), p.view)
    prev = np.eye(4)
    prev[0, 3] = step
    _column_major(prev, p.viewPrev)
    _column_major(proj, p.projection)
    _column_major(proj, p.projectionPrev)
    p.cameraPosition[:] = (0.0, 0.0, 0.0, 1.0)
    p.cameraPositionPrev[:] = (-step, 0.0, 0.0, 1.0)
    p.timeDelta = 1.0 / 60.0
    p.minLogLuminance, p.maxLogLuminance = math.log2(2.0 ** -6 * 0.125), math.log2(2.0 ** 10 * 0.125)
    p.gradientMultDiffuse, p.gradientMultIndirect, p.gradientMultSpecular = 0.5, 0.2, 0.5
    p.antiFireflyEnabled = 1
    p.atrousIterations = case["iterations"]
    p.flags = case["flags"]
    return p


def _volume_params(case, w, h):
    p = N.VolumetricParams()
    proj, _ = _camera(w, h)
    _column_major(np.eye(4), p.invView)
    _column_major(np.linalg.inv(proj), p.invProjection)
    _column_major(proj, p.volumeViewProj)
    p.cameraPosition[:] = (0.0, 0.0, 0.0, 1.0)
    p.volumeCameraNear, p.volumeCameraFar = 0.1, 40.0
    p.volumeAmbient[:] = (0.1, 0.2, 0.4)
    p.volumeScattering, p.maxHistoryLength, p.frameId = 500.0, 16.0, 7
    p.volumeEnableType = N.VOLUME_ENABLE_VOLUMETRIC if case["mode"] == "volumetric" else N.VOLUME_ENABLE_SIMPLE
    return p


AVERAGE = 0.35   # the adapted average luminance before the frame


def _inputs(case, seed, w, h):
    """(planes by (name, slot), the fog volume, the clean scene) a pass reads; slot 1 is the frame before."""
    kind = case["kind"]
    planes, clean, sky, g = _scene(w, h, seed, case.get("noise", "mild"))
    up = {}
    for name, t in planes.items():
        up[name, 0] = t
        if name in _BOTH_SLOTS:
            up[name, 1] = t
    if kind in ("frame", "batch", "full"):
        for name, t in _history(case["storage"], clean, sky, g).items():
            up[name, 0 if name in ("DIFF_COLOR_HISTORY", "GRADIENT_PREV_PIX") else 1] = t
        if case["storage"] in ("fp16", "bf16"):
            up["DIFF_COLOR_HISTORY_VARIANCE", 0] = up["DIFF_ACCUM_MOMENTS", 1][..., 0].square().mul(0.05).contiguous()
    if kind in ("scatter", "full"):
        fog = _fog(w, h, g)
        up["SCATTERING", 1], up["SCATTERING_HISTORY", 1] = fog["SCATTERING"], fog["SCATTERING_HISTORY"]
        volume = fog["SCATTER_VOLUME"]
    else:
        volume = None
    if kind == "post":
        hdr = (clean["D"] + clean["S"]) * torch.exp(0.3 * torch.randn(h, w, 3, generator=g, device=DEV))
        rx, ry = _regular(w, h)
        img = torch.empty_like(hdr)
        img[ry, rx] = hdr
        up["PRE_FINAL", 0] = _image(case["storage"], img)
        fog = _fog(w, h, g)
        up["SCATTERING", 0] = up["SCATTERING", 1] = fog["SCATTERING"]
    return up, volume


# ------------------------------------------------------------------------------------------
# states and passes
# ------------------------------------------------------------------------------------------
_contexts = weakref.WeakValueDictionary()


def _context(flags):
    """The program's context: one for all its streams, closed with the last of them."""
    c = _contexts.get(flags)
    if c is None:
        c = _contexts[flags] = Context(0, flags=flags)
    return c


_VIEW = {1: ("|u1", None), 2: ("|u1", None), 3: ("|u1", None), 4: ("<f2", None), 5: ("<f2", None), 6: ("<f2", None),
         7: ("<i2", torch.bfloat16), 8: ("<f4", None), 9: ("<f4", None), 10: ("<f4", None), 12: ("<i4", None), 13: ("<i4", None)}
_CHANNELS = {1: 1, 2: 2, 3: 4, 4: 1, 5: 2, 6: 4, 7: 4, 8: 1, 9: 2, 10: 4, 12: 1, 13: 1}


class _Memory:
    """Device memory of a stream for torch, which keeps this object, and so the stream, for as long as
    a tensor over it lives."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def _plane(stream, name, slot):
    """A framebuffer image as a tensor over its own memory."""
    img = stream.image(name, slot)
    typestr, dtype = _VIEW[img.format]
    ch = _CHANNELS[img.format]
    shape = (img.height, img.width) if ch == 1 else (img.height, img.width, ch)
    t = torch.as_tensor(_Memory(stream, img.data, shape, typestr), device=DEV)
    return t.view(dtype) if dtype is not None else t


def _outputs(kind, storage):
    names = []
    if kind in ("frame", "batch", "full"):
        names += ["PRE_FINAL", "HISTOGRAM_INPUT", "ACCUM_HISTORY_LENGTH", "DIFF_ACCUM_MOMENTS", "DIFF_COLOR_HISTORY"]
    if kind in ("frame", "full"):
        names += ["SPEC_ACCUM_COLOR", "INDIR_ACCUM", "DIS_GRADIENT_HISTORY", "GRADIENT_PREV_PIX"]
        names += ["DIFF_COLOR_HISTORY_VARIANCE"] if storage in ("fp16", "bf16") else []
    if kind in ("scatter", "full"):
        names += ["SCATTERING", "SCATTERING_HISTORY", "SCATTER_VOLUME"]
    if kind in ("post", "full"):
        names += ["FINAL", "BLOOM_INPUT", "BLOOM_RESULT"]
    return names


def _upload(stream, name, slot, t):
    t = t.contiguous()
    stream.upload(name, slot, (t.data_ptr(), t.numel() * t.element_size()))


class _Camera:
    """One camera stream with its history, its inputs and the calls of one frame."""

    def __init__(self, case, seed, w, h, ctx):
        kind, storage = case["kind"], case.get("storage", "fp16")
        self.stream = s = Stream(ctx, w, h, N.STORAGE_NAMES[storage])
        planes, self.volume = _inputs(case, seed, w, h)
        for (name, slot), t in planes.items():
            _upload(s, name, slot, t)
        s.set_tonemapping(None, AVERAGE)
        self.slot = 0
        self.denoiser, self.tonemapping, self.volumetric = Denoiser(s), Tonemapping(s), Volumetric(s)
        self.composition, self.bloom = ImageComposition(s), Bloom(s)
        if kind in ("frame", "batch", "full"):
            self.params = _frame_params(case, w, h)
        if kind in ("scatter", "full"):
            self.volume_params = _volume_params(case, w, h)
        if kind in ("post", "full"):
            self.final_params = N.FinalParams.defaults()
            self.final_params.flags = N.FINAL_APPLY_SCATTERING
        self.out = []
        for slot in (0, 1):
            o = {name: _plane(s, name, slot) for name in _outputs(kind, storage)}
            if kind in ("frame", "batch", "full"):
                o["average"] = torch.as_tensor(_Memory(s, s.tonemapping_device_ptr() + 1024, (1,), "<f4"), device=DEV)
            self.out.append(o)

    def next(self):
        slot, self.slot = self.slot, self.slot ^ 1
        return slot

    def frame(self):
        slot = self.next()
        self.denoiser.Denoise(slot, self.params)
        self.tonemapping.CalculateExposure(slot, self.params)
        return self.out[slot]

    def scatter(self):
        slot = self.next()
        _upload(self.stream, "SCATTER_VOLUME", slot, self.volume)
        self.volumetric.ProcessScattering(slot, self.volume_params)
        return self.out[slot]

    def post(self):
        slot = self.next()
        self.composition.Finalize(slot, self.final_params)
        self.bloom.Apply(slot)
        return self.out[slot]

    def full(self):
        slot = self.next()
        _upload(self.stream, "SCATTER_VOLUME", slot, self.volume)
        self.denoiser.Denoise(slot, self.params)
        self.volumetric.ProcessScattering(slot, self.volume_params)
        self.tonemapping.CalculateExposure(slot, self.params)
        self.composition.Finalize(slot, self.final_params)
        self.bloom.Apply(slot)
        return self.out[slot]


class _Batch:
    def __init__(self, case, seed, ctx):
        self.ctx = ctx
        self.cameras = [_Camera(case, seed * 64 + k, w, h, ctx) for k, (w, h) in enumerate(_sizes(case))]

    def batch(self):
        jobs = [(c.stream, c.next(), c.params) for c in self.cameras]
        self.ctx.submit_batch(jobs)
        return [c.out[slot] for c, (_, slot, _) in zip(self.cameras, jobs)]


def _sizes(case):
    if case["kind"] == "batch":
        return [tuple(int(v) for v in s.split("x")) for s in case["sizes"].split()]
    return [(case["width"], case["height"])]


def prepare(case, seed):
    if case["kind"] == "batch":
        # frames side by side: the context's documented setting for it
        return _Batch(case, seed, _context(N.CONTEXT_NO_L2_PERSIST)).batch
    c = _Camera(case, seed * 64, case["width"], case["height"], _context(0))
    return getattr(c, case["kind"])


def run(state):
    return state()


# ------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------
def work(case):
    px = sum(w * h for w, h in _sizes(case))
    storage, kind = case.get("storage", "fp16"), case["kind"]
    colour = {"ref": 4, "fp32": 16, "fp16": 8, "bf16": 8}[storage]
    history = {"ref": 8, "fp32": 16, "fp16": 12, "bf16": 12}[storage]   # colour and variance
    moments = 4 if storage == "ref" else 8
    length = 16 if storage == "fp32" else 8
    image = {"ref": 4, "fp32": 16, "fp16": 8, "bf16": 8}[storage]
    b = f = 0.0
    if kind in ("frame", "batch", "full"):
        gbuffer = 3 * 4 + 8 + 8 + 8 + 4 + 4 + 2 + 2 + 2 + 1 + 16     # colours, motion, view, throughput, albedo, normal, ...
        before = 2 + 4 + 16 + 4 + 8 / 9                              # depth, normal, position, gradient inputs, re-shaded
        kept = history + moments + length + 2 * colour               # read from the frame before, written for the next
        b += px * (gbuffer + before + 2 * kept + image + 2 + 2)
        f += px * (900.0 + 420.0 * case["iterations"])
    if kind in ("scatter", "full"):
        x, y, z = N.VOLUME_SIZE
        b += px * ((8 + 2 + 2 + 4 + 4 if kind == "scatter" else 0) + 4 + 2 * (8 + 2)) + 3 * 8 * x * y * z
        f += px * 250.0
    if kind in ("post", "full"):
        b += px * ((image + 8 if kind == "post" else 0) + 4 + 8 + 3 * image)
        f += px * 500.0
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------------------------------
# the same in 64 bits
# ------------------------------------------------------------------------------------------
def _shift(t, dx, dy):
    """t at (x + dx, y + dy), zero outside the image."""
    h, w = t.shape[:2]
    out = torch.zeros_like(t)
    x0, x1, y0, y1 = max(0, -dx), min(w, w - dx), max(0, -dy), min(h, h - dy)
    if x0 < x1 and y0 < y1:
        out[y0:y1, x0:x1] = t[y0 + dy:y1 + dy, x0 + dx:x1 + dx]
    return out


def _lum(c):
    return 0.2125 * c[..., 0] + 0.7154 * c[..., 1] + 0.0721 * c[..., 2]


def _unorm8(x):
    return torch.floor(x.clamp(0.0, 1.0) * 255.0 + 0.5) / 255.0


class _Grid:
    """Checkerboard geometry of a w x h image."""

    def __init__(self, w, h):
        self.w, self.h, self.sep = w, h, w // 2
        self.x = torch.arange(w, device=DEV).view(1, w).expand(h, w)
        self.y = torch.arange(h, device=DEV).view(h, 1).expand(h, w)
        half = (self.x >= self.sep).long()
        self.left, self.right = half * self.sep, (half + 1) * self.sep

    def inside(self, qx, qy):
        return (qy >= 0) & (qy < self.h) & (qx >= self.left) & (qx < self.right)

    def previous(self, mx, my):
        return (self.x + 0.5) + mx * (self.w / 2.0), (self.y + 0.5) + my * self.h

    def at(self, t, qx, qy):
        return t[qy.clamp(0, self.h - 1), qx.clamp(0, self.w - 1)]


def _antilag(g, nf):
    return torch.where(nf > 0.0001, (g.abs() / nf.clamp_min(1e-30)).clamp(0.0, 1.0), torch.zeros_like(g))


def _gradients64(up, storage, grid, p):
    w, h = grid.w, grid.h
    gw, gh = (w + 1) // 3, (h + 1) // 3
    mo = up["MOTION", 0].double()
    px, py = grid.previous(mo[..., 0], mo[..., 1])
    ix, iy = torch.floor(px).long(), torch.floor(py).long()
    ok = (ix >= 0) & (ix < w) & (iy >= 0) & (iy < h)
    lum = torch.where(ok.unsqueeze(-1), grid.at(up["GRADIENT_INPUTS", 1].double(), ix, iy), torch.zeros((), dtype=F64, device=DEV))

    def strata(t, fill):   # (gh, gw, 9, ...) with texels outside the image filled
        full = torch.full((gh * 3, gw * 3) + t.shape[2:], fill, dtype=t.dtype, device=DEV)
        hh, ww = min(h, gh * 3), min(w, gw * 3)
        full[:hh, :ww] = t[:hh, :ww]
        return full.view(gh, 3, gw, 3, *t.shape[2:]).transpose(1, 2).reshape(gh, gw, 9, *t.shape[2:])

    sl = strata(lum, 0.0)
    best = sl.amax(-1)
    k = best.argmax(-1, keepdim=True)
    prev = torch.gather(sl, 2, k.unsqueeze(-1).expand(gh, gw, 1, 2)).squeeze(2)
    pick = lambda t: torch.gather(strata(t, 0), 2, k).squeeze(2)  # noqa: E731
    pxx, pyy, cx, sky = pick(ix), pick(iy), pick(grid.x), pick(up["IS_SKY", 0].long())
    half = (cx >= grid.sep).long()
    good = (pyy >= 0) & (pyy < h) & (pxx >= half * grid.sep) & (pxx < (half + 1) * grid.sep) & (sky == 0) & (prev.amax(-1) > 0.0)
    pxx, pyy = pxx.clamp(0, w - 1), pyy.clamp(0, h - 1)
    fpl = up["GRADIENT_RESHADED", 0].double()[pyy, pxx]
    nf = torch.maximum(fpl, prev)
    bright = _lum(_colour64(storage, up["INDIR_ACCUM", 1])[pyy, pxx])
    st = ((bright - 1.0) / 9.0).clamp(0.0, 1.0)
    g = torch.stack([
        _antilag(fpl[..., 0] - prev[..., 0], nf[..., 0]) * p.gradientMultDiffuse,
        _antilag((prev[..., 0] - fpl[..., 0]).clamp_min(0.0) * (1.0 - st * st * (3.0 - 2.0 * st)), nf[..., 0]) * p.gradientMultIndirect,
        _antilag(fpl[..., 1] - prev[..., 1], nf[..., 1]) * p.gradientMultSpecular], -1)
    gx, gy = pxx // 3, pyy // 3
    inb = ((gx < gw) & (gy < gh)).unsqueeze(-1)
    old = torch.where(inb, up["DIS_GRADIENT_HISTORY", 1][gy.clamp(0, gh - 1), gx.clamp(0, gw - 1)][..., :3].double() / 255.0, torch.zeros_like(g))
    g = torch.where(good.unsqueeze(-1), _unorm8(0.5 * g + 0.5 * old), torch.zeros_like(g))
    x = torch.arange(gw, device=DEV).view(1, gw).expand(gh, gw)
    y = torch.arange(gh, device=DEV).view(gh, 1).expand(gh, gw)
    half = (x * 3 >= grid.sep).long()
    left, right, bottom = half * grid.sep // 3, (half + 1) * grid.sep // 3, h // 3
    for it in range(4):
        step, total, weight = 1 << it, torch.zeros_like(g), torch.zeros(gh, gw, dtype=F64, device=DEV)
        for yy in (-1, 0, 1):
            for xx in (-1, 0, 1):
                qx, qy = x + xx * step, y + yy * step
                wt = 0.5 ** (abs(xx) + abs(yy)) * ((qy >= 0) & (qy < bottom) & (qx >= left) & (qx < right)).double()
                total += _shift(g, xx * step, yy * step) * wt.unsqueeze(-1)
                weight += wt
        g = _unorm8(torch.where(weight.unsqueeze(-1) > 0.0, total / weight.clamp_min(1e-30).unsqueeze(-1), torch.zeros_like(g)))
    full = torch.zeros(h, w, 3, dtype=F64, device=DEV)
    gx, gy = grid.x // 3, grid.y // 3
    ok = (gx < gw) & (gy < gh)
    full[ok] = g[gy[ok], gx[ok]]
    return full


def _matrix(a):
    return torch.tensor(list(a), dtype=F64, device=DEV).view(4, 4).t()


def _mix(x, y, a):
    return x * (1.0 - a) + y * a


def _temporal64(up, storage, grid, p):
    skip = bool(p.flags & N.FLAG_SKIP_GRADIENTS)
    g = torch.zeros(grid.h, grid.w, 3, dtype=F64, device=DEV) if skip else _gradients64(up, storage, grid, p)
    a_d, a_i, a_s = g.unbind(-1)
    z, z_prev = up["DEPTH_WORLD", 0].double(), up["DEPTH_WORLD", 1].double()
    n, n_prev = _normal_decode(up["NORMAL", 0]), _normal_decode(up["NORMAL", 1])
    mo = up["MOTION", 0].double()
    rough = up["METALLIC_ROUGHNESS", 0][..., 1].double() / 255.0
    view = up["VIEW_DIRECTION", 0].double()
    unf = {k: _e5_decode(up[name, 0]) for k, name in (("d", "UNFILTERED_DIRECT"), ("s", "UNFILTERED_SPECULAR"), ("i", "UNFILTERED_INDIR"))}
    kept = torch.cat([up["DIFF_COLOR_HISTORY", 0][..., :3].double(), up["DIFF_ACCUM_MOMENTS", 1].double(),
                      up["ACCUM_HISTORY_LENGTH", 1].double(), _colour64(storage, up["SPEC_ACCUM_COLOR", 1]),
                      _colour64(storage, up["INDIR_ACCUM", 1])], -1)

    def taps(px, py, values):
        fx, fy = torch.floor(px - 0.5), torch.floor(py - 0.5)
        sx, sy = px - 0.5 - fx, py - 0.5 - fy
        fx, fy = fx.clamp(-1e6, 1e6).long(), fy.clamp(-1e6, 1e6).long()
        total, weight = 0.0, torch.zeros_like(z)
        for yy in (0, 1):
            for xx in (0, 1):
                qx, qy = fx + xx, fy + yy
                ok = grid.inside(qx, qy)
                ok &= (z - grid.at(z_prev, qx, qy) + mo[..., 2]).abs() / z.abs() < 0.1
                ok &= (n * grid.at(n_prev, qx, qy)).sum(-1) > 0.95
                wt = (sx if xx else 1.0 - sx) * (sy if yy else 1.0 - sy) * ok
                weight += wt
                if values is not None:
                    total = total + grid.at(values, qx, qy) * wt.unsqueeze(-1)
        return total, weight, fx, fy

    px, py = grid.previous(mo[..., 0], mo[..., 1])
    total, weight, fx, fy = taps(px, py, kept)
    has = weight > 0.0001
    mean = total / weight.clamp_min(1e-30).unsqueeze(-1)
    dif, mom, hl, spec, ind = mean.split([3, 2, 4, 3, 3], -1)
    # specular: on the surface, and through the virtual position behind it
    pos = up["SURFACE_POSITION", 0][..., :3].double()
    inside = (fx >= 0) & (fx < grid.w) & (fy >= 0) & (fy < grid.h)
    pos_prev = torch.where(inside.unsqueeze(-1), grid.at(up["SURFACE_POSITION", 1][..., :3].double(), fx, fy), torch.zeros_like(pos))
    delta = torch.tensor([a - b for a, b in zip(p.cameraPositionPrev[:3], p.cameraPosition[:3])], dtype=F64, device=DEV)
    v, vp = pos / pos.norm(dim=-1, keepdim=True), (pos_prev - delta) / (pos_prev - delta).norm(dim=-1, keepdim=True)
    cosa = (v * vp).sum(-1).clamp(0.0, 1.0)
    par = (1.0 - cosa * cosa).sqrt() / cosa.clamp_min(1e-6) * 60.0
    fps = 0.2 / p.timeDelta
    least = min(max(fps, 0.0), 128.0)
    most = (1.0 + hl[..., 2] * (1.0 - a_s) ** 5).clamp(least, 256.0)
    nv = -(n * view[..., :3]).sum(-1)
    nv = nv.clamp_min(0.0)

    def speed(par_):
        aa = (1.0 - nv).clamp(0.0, 1.0) ** 0.66
        b = 1.1 + rough * rough
        ps = (b + aa) / (b - aa)
        f = (1.0 - torch.exp2(-200.0 * rough * rough)) * rough.clamp(0.0, 1.0) ** (0.5 * (1.0 + par_ * ps))
        return torch.minimum((256.0 * f).clamp_min(least), most)

    on = speed(par)
    da = 0.298475 * torch.log(39.4115 - 39.0029 * rough)
    domin = ((1.0 - nv).clamp(0.0, 1.0) ** 10.8649 * (1.0 - da) + da).clamp(0.0, 1.0)
    hit_now, hit_old = view[..., 3], hl[..., 3]
    inv = 1.0 / (1.0 + on)
    spec_on, hit_on = _mix(spec, unf["s"], inv.unsqueeze(-1)), _mix(hit_old, hit_now, inv)
    virt = torch.cat([pos + view[..., :3] * (hit_on * domin).unsqueeze(-1), torch.ones_like(z).unsqueeze(-1)], -1)
    cur = virt @ (_matrix(p.projection) @ _matrix(p.view)).t()
    old = virt @ (_matrix(p.projectionPrev) @ _matrix(p.viewPrev)).t()
    m = (old[..., :2] / old[..., 3:] - cur[..., :2] / cur[..., 3:]) * 0.5
    _, weight_v, _, _ = taps(*grid.previous(torch.nan_to_num(m[..., 0]), torch.nan_to_num(m[..., 1])), None)
    av = speed(torch.zeros_like(par))
    spec_v = _mix(spec, unf["s"], (1.0 / (1.0 + av)).unsqueeze(-1))
    use_v = weight_v > 0.0001
    aa = _mix(inv, 1.0 / (1.0 + av), domin)
    s_col = torch.where(use_v.unsqueeze(-1), _mix(spec_on, spec_v, domin.unsqueeze(-1)), spec_on)
    s_len = torch.where(use_v, 1.0 / aa - 1.0, on)
    s_hit = torch.where(use_v, _mix(hit_old, hit_now, 1.0 / (1.0 + av.clamp_max(16.0))), hit_on)
    h3 = has.unsqueeze(-1)
    l_now = _lum(unf["d"])
    d_len = (hl[..., 0] * (1.0 - a_d) ** 10 + 1.0).clamp(1.0, 256.0)
    i_len = (hl[..., 1] * (1.0 - a_i) ** 10 + 1.0).clamp(1.0, 256.0)
    ad = _mix((1.0 / d_len).clamp_min(0.01), torch.ones_like(z), a_d)
    ai = _mix((1.0 / i_len).clamp_min(0.01), torch.ones_like(z), a_i)
    one = torch.ones_like(z)
    moments = torch.stack([l_now, l_now * l_now], -1)
    out = {
        "d": torch.where(h3, _mix(dif, unf["d"], ad.unsqueeze(-1)), unf["d"]),
        "m": torch.where(h3, _mix(mom, moments, ad.unsqueeze(-1)), moments),
        "s": torch.where(h3, s_col, unf["s"]), "i": torch.where(h3, _mix(ind, unf["i"], ai.unsqueeze(-1)), unf["i"]),
        "len": torch.stack([torch.where(has, d_len, one), torch.where(has, i_len, one), torch.where(has, s_len, one),
                            torch.where(has, s_hit, hit_now)], -1),
    }
    return out, z, n, rough


def _firefly64(c):
    lo, hi = torch.full_like(c, 1e6), torch.full_like(c, -1e6)
    for dy in range(-2, 3):
        for dx in range(-2, 3):
            if dx or dy:
                q = _shift(c, dx, dy)
                lo, hi = torch.minimum(lo, q), torch.maximum(hi, q)
    return torch.minimum(torch.maximum(c, lo), hi)


def _variance64(c, t, z, n, grid):
    length, mom = t["len"][..., 0], t["m"]
    temporal = (mom[..., 1] - mom[..., 0] ** 2).clamp_min(0.0) / (length - 4.0).clamp_min(1.0)
    l = _lum(c)
    s1, s2, total, weight = l + mom[..., 0], l * l + mom[..., 1], c.clone(), torch.ones_like(l)
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            if not (dx or dy):
                continue
            cq, zq = _shift(c, dx, dy), _shift(z, dx, dy)
            out = ~((grid.x + dx >= 0) & (grid.x + dx < grid.w) & (grid.y + dy >= 0) & (grid.y + dy < grid.h))
            nq = _shift(n, dx, dy)
            nq[..., 2] = torch.where(out, torch.ones_like(l), nq[..., 2])
            mz = torch.maximum(z, zq)
            w = torch.exp(-(z - zq).abs() * torch.where(mz <= 0.0, torch.zeros_like(mz), 1.0 / mz.clamp_min(1e-30)))
            w = w * (n * nq).sum(-1).clamp_min(0.0) ** 128
            lq = _lum(cq)
            s1, s2, total, weight = s1 + lq * w, s2 + lq * lq * w, total + cq * w.unsqueeze(-1), weight + w
    s1, s2, total = s1 / weight, s2 / weight, total / weight.unsqueeze(-1)
    spatial = (s2 - s1 * s1).clamp_min(0.0) * (1.0 + 2.0 * (1.0 - length / 4.0))
    far = (z < 0.0) | (z > MAX_RAY)
    keep = far | (length > 4.0)
    var = torch.where(far, torch.zeros_like(l), torch.where(length > 4.0, temporal, spatial))
    return torch.where(keep.unsqueeze(-1), c, total), var


def _atrous64(it, d, var, s, i, pref, t, z, n, rough, grad, grid):
    step = 1 << it
    far = (z < 0.0) | (z > MAX_RAY)
    if it == 0:
        pref = torch.zeros_like(var)
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                pref += _shift(var, dx, dy) * 0.25 * 0.5 ** (abs(dx) + abs(dy))
        pref = pref.clamp_min(0.0).sqrt()
    l = _lum(d)
    wl = 1.0 / (4.0 * pref + 1e-5)
    wr = (rough * 30.0 - it).clamp(0.0, 1.0)
    power = (2.0 / (rough ** 4 + 1e-4) - 2.0).clamp_min(0.01).clamp(8.0, 1024.0) * (t["len"][..., 2] / 8.0).clamp(0.0, 1.0)
    od, ov, os_, oi = d.clone(), var.clone(), s.clone(), i.clone()
    w_d = torch.ones_like(l)
    w_s, w_i = w_d.clone(), w_d.clone()
    for yy in (-1, 0, 1):
        for xx in (-1, 0, 1):
            if not (xx or yy):
                continue
            dx, dy = xx * step, yy * step
            ok = grid.inside(grid.x + dx, grid.y + dy).double()
            man = abs(xx) + abs(yy)
            dq, sq, iq = _shift(d, dx, dy), _shift(s, dx, dy), _shift(i, dx, dy)
            nn = (n * _shift(n, dx, dy)).sum(-1).clamp_min(0.0)
            wz = (z - _shift(z, dx, dy)).abs() / (grad * man).clamp_min(0.01)
            base = torch.exp(-wz * wz) * nn ** 128 * 0.5 ** man * ok
            wd = base * torch.exp(-(l - _lum(dq)).abs() * wl)
            w_rq = (1.0 - 10.0 * (rough - _shift(rough, dx, dy)).abs()).clamp_min(0.0) * wr
            ws = base * w_rq * nn ** power
            od, ov = od + dq * wd.unsqueeze(-1), ov + _shift(var, dx, dy) * wd * wd
            os_, oi = os_ + sq * ws.unsqueeze(-1), oi + iq * base.unsqueeze(-1)
            w_d, w_s, w_i = w_d + wd, w_s + ws, w_i + base
    od, ov, os_, oi = od / w_d.unsqueeze(-1), ov / (w_d * w_d), os_ / w_s.unsqueeze(-1), oi / w_i.unsqueeze(-1)
    f3 = far.unsqueeze(-1)
    if it == 0:
        d, var, s, i = torch.zeros_like(d), torch.zeros_like(var), torch.zeros_like(s), torch.zeros_like(i)
    return torch.where(f3, d, od), torch.where(far, var, ov), torch.where(f3, s, os_), torch.where(f3, i, oi), pref


def _denoise64(case, up, grid, p):
    storage = case["storage"]
    t, z, n, rough = _temporal64(up, storage, grid, p)
    d, s, i = _firefly64(t["d"]), _firefly64(t["s"]), _firefly64(t["i"])
    d, var = _variance64(d, t, z, n, grid)
    grad = up["DEPTH_GRAD", 0].double()
    pref = kept = None
    for it in range(p.atrousIterations):
        d, var, s, i, pref = _atrous64(it, d, var, s, i, pref, t, z, n, rough, grad, grid)
        if it == 0:
            kept = (d, var)
    # composition, in the regular layout
    rx, ry = _regular(grid.w, grid.h)
    albedo = _b10_decode(up["ALBEDO", 0])[ry, rx]
    tp = up["THROUGHPUT", 0].double()[..., :3]
    metal = (up["METALLIC_ROUGHNESS", 0][..., 0].double() / 255.0).unsqueeze(-1)
    st = ((rough - 0.5) * 4.0).clamp(0.0, 1.0)
    spec = _mix(s, i, (st * st * (3.0 - 2.0 * st)).unsqueeze(-1))
    la = _lum(albedo)
    q = (la - 0.02) / 0.02
    ill = ((d + i) * albedo * (1.0 - metal) + spec * _mix(torch.full_like(albedo, 0.04), albedo, metal)) * tp
    ill = ill * torch.where(la > 0.02, torch.ones_like(la), 1.0 - q * q).unsqueeze(-1)
    ill = torch.where((up["IS_SKY", 0] != 0).unsqueeze(-1), albedo * tp, ill)
    pre, hin = torch.empty_like(ill), torch.empty_like(la)
    pre[ry, rx], hin[ry, rx] = ill.clamp_min(0.0), _lum(ill).clamp_min(0.0)
    lo, hi = p.minLogLuminance, p.maxLogLuminance
    ll = ((torch.log2(hin.clamp_min(1e-30)) - lo) / (hi - lo)).clamp(0.0, 1.0)
    bins = torch.where(hin < 0.001, torch.zeros_like(ll), torch.floor(ll * 254.0 + 1.0))
    dark = float((bins == 0).sum())
    mean = float(bins.sum()) / max(grid.w * grid.h - dark, 1.0) - 1.0
    now = 2.0 ** (mean / 254.0 * (hi - lo) + lo)
    average = min(AVERAGE + (now - AVERAGE) * (1.0 - math.exp(-p.timeDelta * 1.1)), 2.0 ** hi)
    four = lambda c, a=None: _rgba(c, a)  # noqa: E731
    packed = storage == "ref"
    var_in = storage in ("ref", "fp32")
    out = {"PRE_FINAL": None if packed else four(pre), "HISTOGRAM_INPUT": hin, "ACCUM_HISTORY_LENGTH": t["len"],
           "DIFF_ACCUM_MOMENTS": t["m"], "DIFF_COLOR_HISTORY": four(kept[0], kept[1] if var_in else None),
           "SPEC_ACCUM_COLOR": None if packed else four(t["s"]), "INDIR_ACCUM": None if packed else four(t["i"]),
           "DIFF_COLOR_HISTORY_VARIANCE": kept[1], "average": torch.tensor([average], dtype=F64, device=DEV)}
    return out, pre, average


def _murmur33(x, y, z):
    k, mask = 0x5BD1E995, 0xFFFFFFFF
    lanes = []
    src = [(v * k) & mask for v in (x, y, z)]
    src = [v ^ (v >> 24) for v in src]
    src = [(v * k) & mask for v in src]
    for seed in (1190494759, 2147483647, 3559788179):
        hsh = torch.full_like(x, seed)
        for v in src:
            hsh = ((hsh * k) & mask) ^ v
        hsh = hsh ^ (hsh >> 13)
        hsh = (hsh * k) & mask
        lanes.append(hsh ^ (hsh >> 15))
    return lanes


def _lowbias32(x):
    mask = 0xFFFFFFFF
    x = x ^ (x >> 16)
    x = (x * 0x7FEB352D) & mask
    x = x ^ (x >> 15)
    x = ((x >> 16) * 0x846CA68B << 16 & mask) + ((x & 0xFFFF) * 0x846CA68B & mask) & mask
    return x ^ (x >> 16)


def _scatter64(case, up, volume, grid, p):
    w, h = grid.w, grid.h
    nx, ny, nz = N.VOLUME_SIZE
    vol = volume.double().view(nz, ny, nx, 4)
    out = torch.empty_like(vol)
    acc, e = vol[0], torch.exp(-vol[0, ..., 3])
    for k in range(nz):
        if k:
            acc = torch.cat([acc[..., :3] + e.clamp(0.0, 1.0).unsqueeze(-1) * vol[k, ..., :3], (acc[..., 3] + vol[k, ..., 3]).unsqueeze(-1)], -1)
            e = torch.exp(-acc[..., 3])
        out[k] = torch.cat([acc[..., :3], e.unsqueeze(-1)], -1)
    rx, ry = _regular(w, h)
    z, z_prev = up["DEPTH_WORLD", 0].double(), up["DEPTH_WORLD", 1].double()
    n, n_prev = _normal_decode(up["NORMAL", 0]), _normal_decode(up["NORMAL", 1])
    mo = up["MOTION", 0].double()
    px, py = grid.previous(mo[..., 0], mo[..., 1])
    fx, fy = torch.floor(px - 0.5), torch.floor(py - 0.5)
    sx, sy = px - 0.5 - fx, py - 0.5 - fy
    fx, fy = fx.long(), fy.long()
    before = torch.cat([up["SCATTERING", 1].double(), up["SCATTERING_HISTORY", 1].double().unsqueeze(-1)], -1)[ry, rx]
    total, weight = 0.0, torch.zeros_like(z)
    for yy in (0, 1):
        for xx in (0, 1):
            qx, qy = fx + xx, fy + yy
            ok = grid.inside(qx, qy) & ((z - grid.at(z_prev, qx, qy) + mo[..., 2]).abs() / z.abs() < 0.1)
            ok &= (n * grid.at(n_prev, qx, qy)).sum(-1) > 0.95
            wt = (sx if xx else 1.0 - sx) * (sy if yy else 1.0 - sy) * ok
            total, weight = total + grid.at(before, qx, qy) * wt.unsqueeze(-1), weight + wt
    has = (weight > 0.0001).unsqueeze(-1)
    total = torch.where(has, total / weight.clamp_min(1e-30).unsqueeze(-1), torch.zeros_like(total))
    length = (total[..., 4] + 1.0).clamp(1.0, p.maxHistoryLength)
    if case["mode"] == "simple":
        f = torch.exp(-z * p.volumeScattering * 0.00005)
        fog = torch.tensor(list(p.volumeAmbient), dtype=F64, device=DEV)
        now = torch.cat([fog * (1.0 - f).unsqueeze(-1), f.unsqueeze(-1)], -1)
        now = torch.where((z > MAX_RAY).unsqueeze(-1), torch.tensor([0.0, 0.0, 0.0, 1.0], dtype=F64, device=DEV), now)
    else:
        ndc = torch.stack([rx / w * 2.0 - 1.0, ry / h * 2.0 - 1.0, up["DEPTH_NDC", 0].double()[ry, rx], torch.ones_like(z)], -1)
        wp = ndc @ (_matrix(p.invView) @ _matrix(p.invProjection)).t()
        pos = wp[..., :3] / wp[..., 3:]
        a, b, c = _murmur33(rx, ry, torch.full_like(rx, p.frameId))
        rnd = _lowbias32(((c % 128) << 14) | ((b % 128) << 7) | (a % 128))
        r = [((rnd >> sh) & 255).double() / 255.0 for sh in (0, 8, 16)]
        u1, phi = r[0] * 0.99, 2.0 * math.pi * r[1] * 0.99
        k = r[2] * 2.0
        basis = [-u1.sqrt() * torch.cos(phi), -u1.sqrt() * torch.sin(phi), -(1.0 - u1).sqrt()]
        clip = torch.cat([pos, torch.ones_like(z).unsqueeze(-1)], -1) @ _matrix(p.volumeViewProj).t()
        at = [clip[..., 0] / clip[..., 3] * 0.5 + 0.5, clip[..., 1] / clip[..., 3] * 0.5 + 0.5,
              ((pos.norm(dim=-1) - p.volumeCameraNear) / (p.volumeCameraFar - p.volumeCameraNear)).clamp(0.0, 1.0)]
        idx, frac = [], []
        for v, off, size in zip(at, basis, (nx, ny, nz)):
            x = (v + k * off / size) * size - 0.5
            x0 = torch.floor(x)
            i0 = x0.clamp(-2.0, size + 1.0).long()
            idx.append((i0.clamp(0, size - 1), (i0 + 1).clamp(0, size - 1)))
            frac.append((x - x0).unsqueeze(-1))
        now = 0.0
        for cz in (0, 1):
            for cy in (0, 1):
                for cx in (0, 1):
                    wt = 1.0
                    for j, f in zip((cx, cy, cz), frac):
                        wt = wt * (f if j else 1.0 - f)
                    now = now + out[idx[2][cz], idx[1][cy], idx[0][cx]] * wt
    res = _mix(total[..., :4], now, (1.0 / length).unsqueeze(-1))
    sc, hs = torch.empty_like(res), torch.empty_like(length)
    sc[ry, rx], hs[ry, rx] = res, length
    return {"SCATTERING": sc, "SCATTERING_HISTORY": hs, "SCATTER_VOLUME": out.view(nz * ny, nx, 4)}


def _lpm64(c):
    """The 709 -> 709 luma-preserving map at its default saturation and crosstalk."""
    prim = np.array([[0.64, 0.30, 0.15], [0.33, 0.60, 0.06]])
    m = np.vstack([prim, 1.0 - prim.sum(0)])
    white = np.array([0.3127 / 0.3290, 1.0, (1.0 - 0.3127 - 0.3290) / 0.3290])
    y = m[1] * np.linalg.solve(m, white)
    y = y / y.sum()
    con, mid, top = 1.1, 256.0 * 0.18 * 2.0 ** -8, 256.0
    z0, z1, z2 = -mid ** con, top ** con * mid ** con, top ** con * mid ** con * 0.18
    z3, z4 = top ** con * 0.18, mid ** con * 0.18
    scale, bias = -((z0 + 0.18 * (z1 - z2) / (z3 - z4)) / z4), (z1 - z2) / (z3 - z4)
    y = torch.tensor(y, dtype=F64, device=DEV)
    ratio = (c / c.amax(-1, keepdim=True)) ** con
    luma = (c * y).sum(-1, keepdim=True) ** con
    luma = luma / (luma * scale + bias)
    out = (ratio * (luma / (ratio * y).sum(-1, keepdim=True)).clamp(0.0, 1.0)).clamp(0.0, 1.0)
    cap = 1.0 - out
    add = (luma - (out * y).sum(-1, keepdim=True)).clamp(0.0, 1.0)
    out = torch.nan_to_num((add / (cap * y).sum(-1, keepdim=True)) * cap + out, nan=0.0).clamp(0.0, 1.0)
    add = (luma - (out * y).sum(-1, keepdim=True)).clamp(0.0, 1.0)
    return (add / y + out).clamp(0.0, 1.0)


def _bilinear(img, u, v):
    """img at the grid of texture coordinates u (columns) x v (rows), clamp to edge."""
    h, w = img.shape[:2]

    def axis(c, size):
        x = c * size - 0.5
        x0 = torch.floor(x)
        i = x0.long()
        return i.clamp(0, size - 1), (i + 1).clamp(0, size - 1), x - x0

    x0, x1, fx = axis(u, w)
    y0, y1, fy = axis(v, h)
    rows = _mix(img[:, x0], img[:, x1], fx.view(1, -1, 1))
    return _mix(rows[y0], rows[y1], fy.view(-1, 1, 1))


def _bloom64(img, w, h):
    span = lambda k: (max(1, (w + 1) >> k), max(1, (h + 1) >> k))  # noqa: E731
    centre = lambda n, k, size: (torch.arange(n, device=DEV, dtype=F64) + 0.5) * (2.0 ** k / size)  # noqa: E731
    mips = [img]
    for k in range(8):
        dw, dh = span(k + 1)
        u, v = centre(dw, k + 1, w), centre(dh, k + 1, h)
        tx, ty = 2.0 ** k / w, 2.0 ** k / h
        tap = lambda x, y: _bilinear(mips[k], u + x * tx, v + y * ty)  # noqa: E731,B023
        grid = {(x, y): tap(x, y) for x in (-2, 0, 2) for y in (-2, 0, 2)}
        inner = (tap(-1, -1) + tap(1, -1) + tap(-1, 1) + tap(1, 1)) * 0.25
        boxes = [(inner, 0.5)]
        for x, y in ((-2, -2), (0, -2), (-2, 0), (0, 0)):
            boxes.append(((grid[x, y] + grid[x + 2, y] + grid[x, y + 2] + grid[x + 2, y + 2]) * 0.25, 0.125))
        mips.append(sum(b * (wt / (1.0 + _lum(b).unsqueeze(-1)) if k == 0 else wt) for b, wt in boxes))
    up = mips[8]
    for k in range(7, -1, -1):
        dw, dh = span(k) if k else (w, h)
        own = mips[k] if k else torch.zeros(h, w, 3, dtype=F64, device=DEV)
        sx, sy = 2.0 ** (k + 1) / w, 2.0 ** (k + 1) / h
        u, v = centre(dw, k, w) + 0.5 * sx, centre(dh, k, h) + 0.5 * sy
        tent = own
        for y, wy in ((-1, 1), (0, 2), (1, 1)):
            for x, wx in ((-1, 1), (0, 2), (1, 1)):
                tent = tent + _bilinear(up, u + x * sx, v + y * sy) * (wx * wy / 16.0)
        written = (u <= 1.0).view(1, -1, 1) & (v <= 1.0).view(-1, 1, 1)
        up = torch.where(written, tent, own)
    return up


def _post64(case, up, hdr, scattering, average, grid):
    storage = case["storage"]
    w, h = grid.w, grid.h
    emis = _b10_decode(up["SCREEN_EMIS_RT", 0])
    x, y = grid.x, grid.y
    cbx = ((x + y % 2) % 2) * grid.sep + x // 2
    split = (up["THROUGHPUT", 0][y, cbx][..., 3].double() > 0.5).unsqueeze(-1)
    left = ((cbx != 0) & (cbx != grid.sep)).double().unsqueeze(-1)
    right = ((cbx != grid.sep) & (cbx != w)).double().unsqueeze(-1)

    def resolve(c):
        cross = 0.25 * (_shift(c, -1, 0) * left + _shift(c, 1, 0) * right + _shift(c, 0, 1) + _shift(c, 0, -1))
        return torch.where(split, 0.5 * c + 0.5 * cross, c)

    hdr, emis = resolve(hdr), resolve(emis)
    hdr = hdr * scattering[..., 3:] + scattering[..., :3]
    ev = math.log2(max(0.0, average) * 8.0)
    exposure, el = 1.0 / (1.2 * 2.0 ** ev), 2.0 ** (ev + 16.0 - 3.0)
    color = _lpm64(hdr * exposure + emis * 1.5)
    bloom = (hdr + emis * el) * exposure
    st = (_lum(bloom) / 4.0).clamp(0.0, 1.0)
    bloom = bloom * (st * st * (3.0 - 2.0 * st)).unsqueeze(-1)
    result = _bloom64(bloom, w, h)
    u, v = (torch.arange(w, device=DEV, dtype=F64) + 0.5) / w, (torch.arange(h, device=DEV, dtype=F64) + 0.5) / h
    final = color + _bilinear(result, u, v)
    if storage == "ref":
        return {"FINAL": None, "BLOOM_INPUT": None, "BLOOM_RESULT": None}
    return {"FINAL": _rgba(final), "BLOOM_INPUT": _rgba(bloom), "BLOOM_RESULT": _rgba(result)}


def _exact_camera(case, seed, w, h):
    kind, storage = case["kind"], case.get("storage", "fp16")
    up, volume = _inputs(case, seed, w, h)
    grid = _Grid(w, h)
    out, pre, average = {}, None, AVERAGE
    if kind in ("frame", "batch", "full"):
        o, pre, average = _denoise64(case, up, grid, _frame_params(case, w, h))
        out.update(o)
    if kind in ("scatter", "full"):
        out.update(_scatter64(case, up, volume, grid, _volume_params(case, w, h)))
    if kind in ("post", "full"):
        hdr = _image64(storage, up["PRE_FINAL", 0]) if pre is None else pre
        fog = out["SCATTERING"] if kind == "full" else up["SCATTERING", 0].double()
        out.update(_post64(case, up, hdr, fog, average, grid))
    want = _outputs(kind, storage) + (["average"] if "average" in out else [])
    return {name: out.get(name) for name in want}


def exact(case, seed):
    if case["kind"] == "batch":
        return [_exact_camera(case, seed * 64 + k, w, h) for k, (w, h) in enumerate(_sizes(case))]
    out = _exact_camera(case, seed * 64, case["width"], case["height"])
    return out if any(v is not None for v in out.values()) else None   # packed formats alone have no such value
