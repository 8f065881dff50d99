"""The work that programs have this package do, as measurable cases: whole denoised frames, SVGF frames, the display
post, path-traced G-buffers, and the training of the parameter MLP (one frame's forward and adjoint, optimiser steps
over windows, with and without the gradient through time), each through its public Python entry point.

Sizes come from the package's own workloads (``hush_b200.scene``: 256^2 crops, 640 x 360, 1920 x 1080, 3840 x 2160,
384^2 training windows) and odd ones between them. The radiance of the synthetic scenes is scaled like the path
tracer's own output, whose samples are clamped (clampLum 16): fireflies on 0.5% of the pixels at ten times their mean.

``exact`` restates the denoiser, SVGF, the post and the trainer's frame as plain torch in float64, with the float16
texel rounding where the frame stores an image.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from hush_b200 import SVGF, Hush, Post, builtin_weights, pt
from hush_b200.dp import finish_step
from hush_b200.scene import NAMES, SceneConfig, frame_device
from hush_b200.train import TrainConfig, Trainer, window_scene, xavier_init

FULL, HALF, QUARTER = 8, 8, 8  # bytes of one rgba16float texel


# ---------------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # a crop / a thumbnail preview: the smallest frame, where launches and host time count
        dict(name="denoise-256", kind="denoise", width=256, height=256, mlp="fp32", graph=False, objects=12, moving=0),
        # the reference's demo size with its `f16` option (f16 arithmetic in the MLP), launched directly
        dict(name="denoise-360p-half", kind="denoise", width=640, height=360, mlp="half", graph=False, objects=12,
             moving=0),
        # a resized window: odd in both directions, tensor-core MLP, launched directly
        dict(name="denoise-odd-bf16", kind="denoise", width=1283, height=717, mlp="bf16", graph=False, objects=12,
             moving=3),
        # the headline: full HD, the default MLP, one graph per frame
        dict(name="denoise-1080p", kind="denoise", width=1920, height=1080, mlp="fp32", graph=True, objects=12,
             moving=3),
        # the largest frame: 4K, tensor-core MLP, one graph per frame
        dict(name="denoise-4k-bf16", kind="denoise", width=3840, height=2160, mlp="bf16", graph=True, objects=32,
             moving=8),
        # the fallback denoiser at full HD with its defaults
        dict(name="svgf-1080p", kind="svgf", width=1920, height=1080, iterations=5, taa=True, moving=3),
        # the same at an odd preview size with fewer iterations and no TAA
        dict(name="svgf-odd-3", kind="svgf", width=641, height=363, iterations=3, taa=False, moving=0),
        # the demo's split-screen output into the canvas format
        dict(name="post-1080p", kind="post", width=1920, height=1080, format="rgba8unorm", split=0.5),
        # the renderer that feeds the denoiser: 1 spp, 3 bounces, sun and sphere light, textures
        dict(name="trace-1080p", kind="trace", width=1920, height=1080, objects=32, mode=0, spp=1),
        # one frame of the training twin, forward and adjoint, as an external optimiser drives it
        dict(name="train-frame-256", kind="train_frame", size=256, mlp="fp32"),
        # one optimiser step of the training workload: 16 windows of 8 frames
        dict(name="train-step-384", kind="train_step", size=384, frames=8, windows=16, mlp="bf16", bptt=False),
        # the same with the gradient through time
        dict(name="train-bptt-384", kind="train_step", size=384, frames=8, windows=16, mlp="bf16", bptt=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["denoise", "denoise", "denoise", "svgf", "post", "trace", "train_frame", "train_step"])
    w = _log(rng, 160, 2560)
    h = max(96, min(1440, int(w * rng.uniform(0.45, 1.0))))
    if kind == "denoise":
        return dict(kind=kind, width=w, height=h, mlp=rng.choice(["fp32", "fp32", "bf16", "f16", "half"]),
                    graph=rng.random() < 0.5, objects=rng.randint(4, 32), moving=rng.randint(0, 4))
    if kind == "svgf":
        return dict(kind=kind, width=w, height=h, iterations=rng.randint(1, 5), taa=rng.random() < 0.7,
                    moving=rng.randint(0, 4))
    if kind == "post":
        return dict(kind=kind, width=w, height=h, format=rng.choice(["rgba8unorm", "bgra8unorm", "rgba32float"]),
                    split=round(rng.uniform(0.1, 0.9), 3))
    if kind == "trace":
        return dict(kind=kind, width=min(w, 1920), height=min(h, 1080), objects=rng.randint(4, 40),
                    mode=int(rng.random() < 0.3), spp=rng.randint(1, 2))
    if kind == "train_frame":
        return dict(kind=kind, size=rng.randint(97, 384), mlp=rng.choice(["fp32", "bf16", "f16"]))
    return dict(kind=kind, size=rng.randint(97, 384), frames=rng.randint(2, 8), windows=rng.randint(1, 16),
                mlp=rng.choice(["fp32", "bf16", "f16"]), bptt=rng.random() < 0.5)


def _scene(case, seed, frames):
    return SceneConfig(case["width"], case["height"], frames, n_objects=case.get("objects", 12),
                       n_moving=case.get("moving", 0), pan_min=0.0, pan_max=4.0, firefly_rate=0.005,
                       firefly_scale=10.0, seed=seed)


HISTORY = 2  # frames denoised before the measured ones


def _n_frames(case):
    return 8 if case["width"] * case["height"] <= 1920 * 1080 else 4


def _frames(case, seed, n):
    sc = _scene(case, seed, n)
    return [frame_device(sc, t) for t in range(n)]


def _svgf_inputs(frames, t):
    prev = frames[t - 1] if t else frames[0]
    return dict(frames[t], prevNormalDepth=prev["normalDepth"], prevMotion=prev["motion"])


def _post_images(case, seed):
    """Two linear HDR images of one scene: its noise-free and its 1 spp colour, as rgba16float."""
    fr = frame_device(_scene(dict(case, moving=0), seed, 1), 0, clean=True)
    left = torch.cat([fr["clean"], torch.ones_like(fr["clean"][..., :1])], -1).half().contiguous()
    right = (fr["radiance"].float() + fr["emission"].float()).half().contiguous()
    return left, right


def _sky_map(seed):
    """An equirect sky, 256 x 128: a vertical gradient with seeded clouds and a small sun."""
    rng = np.random.default_rng(seed)
    v = np.linspace(0.0, 1.0, 128)[:, None, None]
    img = np.ones((128, 256, 4), np.float32)
    img[..., :3] = (0.3 + 0.6 * v) * np.array([0.5, 0.7, 1.0]) * (0.8 + 0.4 * rng.random((128, 256, 1)))
    img[30:32, 60:62, :3] = 3000.0
    return img


def prepare(case, seed):
    kind = case["kind"]
    if kind == "denoise":
        frames = _frames(case, seed, _n_frames(case))
        den = Hush(0, {"width": case["width"], "height": case["height"], "mlp": case["mlp"], "graph": case["graph"]})
        for t in range(HISTORY):
            den.denoise(frames[t])
        return {"kind": kind, "den": den, "frames": frames, "t": HISTORY}
    if kind == "svgf":
        frames = _frames(case, seed, _n_frames(case))
        den = SVGF(0, case["width"], case["height"], {"iterations": case["iterations"], "taa": case["taa"]})
        ins = [_svgf_inputs(frames, t) for t in range(len(frames))]
        for t in range(HISTORY):
            den.encode(ins[t])
        return {"kind": kind, "den": den, "ins": ins, "t": HISTORY}
    if kind == "post":
        left, right = _post_images(case, seed)
        return {"kind": kind, "post": Post(0, case["format"]), "left": left, "right": right, "split": case["split"]}
    if kind == "trace":
        sc, env, _ = pt.demo_scene(0, seed=seed, n_objects=case["objects"])
        env = dict(env, map=pt.prepare_env_map(_sky_map(seed)))
        w, h = case["width"], case["height"]
        cam = pt.Camera(position=(0.0, 4.0, 13.0), target=(0.0, 0.8, 0.0), fov=50, aspect=w / h)
        tracer = pt.PathTracer(0, sc, w, h)
        for view in [tracer.accum, *tracer.gbuf[0].values(), *tracer.gbuf[1].values()]:
            _owned(view, tracer)
        return {"kind": kind, "tracer": tracer, "env": env, "cam": cam, "vp": None, "mode": case["mode"],
                "spp": case["spp"], "t": 0}
    if kind == "train_frame":
        n = case["size"]
        den = Hush(0, {"width": n, "height": n, "schedule": "passes"})
        tr = Trainer(den, xavier_init(seed))
        tr.set_mlp(case["mlp"])
        sc = _train_scene(n, 2, seed)
        f0, f1 = (frame_device(sc, t, clean=True) for t in range(2))
        tr.frame(f0, f0["clean"], None, LAMBDA_T, backward=False, sync=False)
        tr.end_frame()
        return {"kind": kind, "den": den, "tr": tr, "f0": f0, "f1": f1}
    if kind == "train_step":
        n = case["size"]
        cfg = TrainConfig(size=n, frames=case["frames"], batch=case["windows"], mlp=case["mlp"], bptt=case["bptt"])
        den = Hush(0, {"width": n, "height": n, "schedule": "passes"})
        tr = Trainer(den, xavier_init(seed))
        tr.set_mlp(case["mlp"])
        return {"kind": kind, "den": den, "tr": tr, "cfg": cfg, "rng": np.random.default_rng(seed)}
    raise ValueError(f"unknown kind {kind}")


LAMBDA_T = 0.5


def _train_scene(size, frames, seed):
    return window_scene(TrainConfig(size=size, frames=frames), seed).with_(firefly_scale=10.0)


def _owned(view, owner):
    """A view of an instance's own buffer, keeping the instance alive as long as the view."""
    view.owner = owner
    return view


def run(s):
    kind = s["kind"]
    if kind == "denoise":  # the next frame of the sequence
        fr = s["frames"][s["t"] % len(s["frames"])]
        s["t"] += 1
        return _owned(s["den"].denoise(fr), s["den"])
    if kind == "svgf":
        g = s["ins"][s["t"] % len(s["ins"])]
        s["t"] += 1
        return _owned(s["den"].encode(g), s["den"])
    if kind == "post":
        return s["post"].encode(s["left"], s["right"], split=s["split"])
    if kind == "trace":  # the next jittered frame
        i, tr = s["t"], s["tracer"]
        s["t"] += 1
        s["vp"] = tr.write_uniforms(camera=s["cam"], prev_view_proj=s["vp"], frame=i, mode=s["mode"],
                                    jitter=pt.JITTER[i % 16], spp=s["spp"], env=s["env"])
        if s["mode"] == 1:
            tr.clear_accum()
            tr.encode(i & 1)
            return tr.accum
        return tr.encode(i & 1)
    if kind == "train_frame":  # gradient of one frame's loss, for an optimiser outside the package
        tr = s["tr"]
        tr.zero_grad()
        tr.frame(s["f1"], s["f1"]["clean"], s["f0"]["clean"], LAMBDA_T, backward=True, sync=False)
        grad, _ = tr.accumulators()
        return {"out": _owned(tr.buffer("OUT"), tr), "par": _owned(tr.buffer("PAR"), tr),
                "dpar": _owned(tr.buffer("DPAR"), tr), "grad": grad.float()}
    tr, cfg = s["tr"], s["cfg"]  # one optimiser step
    seeds = [int(x) for x in s["rng"].integers(0, cfg.seeds, cfg.batch)]
    step = tr.windows_bptt if cfg.bptt else tr.windows
    step(window_scene(cfg), seeds, cfg.frames, cfg.lambda_t)
    grad = tr.accumulators()[0].float()
    loss, _ = finish_step(tr, None, cfg.batch * cfg.frames, cfg.lr, cfg.clip)
    return {"grad": grad, "loss": loss, "theta": _owned(tr.buffer("THETA"), tr)}


def work(case):
    """Each input read once, each output and each carried state image written (and read) once; the arithmetic is an
    estimate of the passes' operations per pixel."""
    kind = case["kind"]
    if kind in ("train_frame", "train_step"):
        px = case["size"] ** 2
        n = case.get("frames", 1) * case.get("windows", 1)
        # G-buffer and clean image in, colour / moments / key / output history in and out; forward and adjoint
        return {"bytes": px * n * (5 * FULL + 12 + 8 * FULL), "flops": px * n * 6000}
    px = case["width"] * case["height"]
    if kind == "denoise":  # five inputs, four history images and par0 in and out (the output is one of them)
        return {"bytes": px * (5 * FULL + 8 * FULL + 2 * HALF // 4), "flops": px * 1600}
    if kind == "svgf":  # seven inputs, three history images in and out (without TAA the output only leaves)
        return {"bytes": px * (7 * FULL + (6 if case["taa"] else 5) * FULL), "flops": px * (900 + 900 * case["iterations"])}
    if kind == "post":
        return {"bytes": px * (FULL + (16 if case["format"] == "rgba32float" else 4)), "flops": px * 400}
    spp = case["spp"] if case["mode"] else 1  # bounded by the traversal, not by its image traffic
    return {"bytes": px * (16 if case["mode"] else 5 * FULL), "flops": px * spp * 20000}


# ------------------------------------------------------------------------------------- float64: shared pieces
def _pow2(e):
    return torch.ldexp(torch.ones_like(e, dtype=torch.float64), e)


def _store(x):
    """A float16 texel write, rounded toward zero (values beyond the range saturate)."""
    e = torch.frexp(x.abs())[1]
    q = _pow2(torch.clamp(e - 1, min=-14) - 10)
    return torch.clamp(torch.trunc(x / q) * q, -65504.0, 65504.0)


def _qf16(x):
    """Clamped to the float16 range with an 11-bit significand (no denormal limit)."""
    x = torch.clamp(x, -65504.0, 65504.0)
    q = _pow2(torch.frexp(x.abs())[1] - 11)
    return torch.trunc(x / q) * q


def _lum(c):
    return c[..., 0] * 0.2126 + c[..., 1] * 0.7152 + c[..., 2] * 0.0722


def _oct_enc(n):
    v = n / torch.clamp(n.abs().sum(-1, keepdim=True), min=1e-20)
    s = torch.where(v[..., :2] >= 0, 1.0, -1.0)
    folded = (1.0 - v[..., [1, 0]].abs()) * s
    return torch.where(v[..., 2:3] < 0, folded, v[..., :2])


def _oct_dec(e):
    z = 1.0 - e[..., :1].abs() - e[..., 1:2].abs()
    t = torch.clamp(-z, min=0.0)
    xy = e[..., :2] + torch.where(e[..., :2] >= 0, -t, t)
    n = torch.cat([xy, z], -1)
    return n / torch.clamp(n.norm(dim=-1, keepdim=True), min=1e-20)


def _shift(a, dy, dx):
    """a[y + dy, x + dx], clamped to the edge."""
    ys = torch.arange(a.shape[0], device=a.device) + dy
    xs = torch.arange(a.shape[1], device=a.device) + dx
    return a[ys.clamp(0, a.shape[0] - 1)][:, xs.clamp(0, a.shape[1] - 1)]


def _within(a, dy, dx):
    """Whether (y + dy, x + dx) lies inside the image."""
    ys = torch.arange(a.shape[0], device=a.device) + dy
    xs = torch.arange(a.shape[1], device=a.device) + dx
    return ((ys >= 0) & (ys < a.shape[0]))[:, None] & ((xs >= 0) & (xs < a.shape[1]))[None, :]


def _pick(a, y, x):
    return a[y.clamp(0, a.shape[0] - 1), x.clamp(0, a.shape[1] - 1)]


def _grid(h, w, dev):
    return torch.meshgrid(torch.arange(h, device=dev), torch.arange(w, device=dev), indexing="ij")


def _tm(c):
    return c / (1.0 + _lum(c))[..., None]


def _itm(c):
    return c / torch.clamp(1.0 - _lum(c), min=1e-4)[..., None]


def _ycocg(c):
    r, g, b = c[..., 0], c[..., 1], c[..., 2]
    return torch.stack([r / 4 + g / 2 + b / 4, r / 2 - b / 2, -r / 4 + g / 2 - b / 4], -1)


def _rgb(c):
    y, co, cg = c[..., 0], c[..., 1], c[..., 2]
    return torch.stack([y + co - cg, y + cg, y - co - cg], -1)


def _bilinear(prev, mv, h, w):
    """The history colour at the reprojected position and whether that lies inside the image."""
    ys, xs = _grid(h, w, prev.device)
    u, v = (xs + 0.5 + mv[..., 0]) / w, (ys + 0.5 + mv[..., 1]) / h
    inside = (u >= 0) & (v >= 0) & (u <= 1) & (v <= 1)
    px, py = u * w - 0.5, v * h - 0.5
    bx, by = torch.floor(px), torch.floor(py)
    fx, fy = px - bx, py - by
    hist = 0.0
    for j in range(4):
        wt = (fx if j & 1 else 1 - fx) * (fy if j >> 1 else 1 - fy)
        hist = hist + wt[..., None] * _pick(prev, by.long() + (j >> 1), bx.long() + (j & 1))[..., :3]
    return hist, inside


def _depth_slope(z):
    """Smaller one-sided depth difference per axis, the larger of the two axes, at most the depth itself."""
    def side(dy, dx):
        q = _shift(z, dy, dx)
        return torch.where(q > 0, (q - z).abs(), torch.full_like(z, 1e9))
    gx, gy = torch.minimum(side(0, 1), side(0, -1)), torch.minimum(side(1, 0), side(-1, 0))
    return torch.minimum(torch.maximum(gx, gy), z)


SPLINE = {1: (0.25, 0.5, 0.25), 2: (1 / 16, 1 / 4, 3 / 8, 1 / 4, 1 / 16)}


def _blur3(v):
    k = SPLINE[1]
    return sum(k[dy + 1] * k[dx + 1] * _shift(v, dy, dx) for dy in (-1, 0, 1) for dx in (-1, 0, 1))


def _atrous(A, G, s, c, step, prefilter, R=1):
    """One edge-aware a-trous level of the denoiser: A colour + variance, G normal + depth (negative: sky)."""
    surf = G[..., 3] >= 0
    gv = _blur3(A[..., 3]) if prefilter else A[..., 3]
    sl = s / (torch.sqrt(torch.clamp(gv, min=1e-12)) + 1e-6)
    zg = torch.where(surf, _depth_slope(G[..., 3]), torch.ones_like(gv))
    lc, hw = _lum(A), SPLINE[R]
    wt = hw[R] * hw[R] * c * torch.ones_like(lc)
    col, var = A[..., :3] * wt[..., None], A[..., 3] * wt * wt
    for dy in range(-R, R + 1):
        for dx in range(-R, R + 1):
            if dx == 0 and dy == 0:
                continue
            g, a = _shift(G, dy * step, dx * step), _shift(A, dy * step, dx * step)
            ok = _within(G, dy * step, dx * step) & (g[..., 3] >= 0)
            wq = hw[dy + R] * hw[dx + R] * torch.clamp((g[..., :3] * G[..., :3]).sum(-1), min=0.0) ** 128 * torch.exp(
                -(g[..., 3] - G[..., 3]).abs() / (zg * (math.hypot(dx, dy) * step) + 1e-3) - sl * (_lum(a) - lc).abs())
            wq = torch.where(ok, wq, torch.zeros_like(wq))
            wt = wt + wq
            col = col + wq[..., None] * a[..., :3]
            var = var + wq * wq * a[..., 3]
    out = torch.cat([col / wt[..., None], (var / (wt * wt))[..., None]], -1)
    return torch.where(surf[..., None], out, torch.zeros_like(out))


def _as64(inputs):
    return {k: inputs[k].double() for k in NAMES}


# ------------------------------------------------------------------------------------- float64: the denoiser
def _temporal(f, st, exposure):
    """Reprojection, anti-lag clamp and blend, moments, key; the block features. st: the previous frame's stored
    images, or None without history. Returns this frame's images and the half-resolution planes."""
    nd, mv, mat = f["normalDepth"], f["motion"], f["material"]
    H, W = nd.shape[:2]
    dev = nd.device
    ok = nd[..., 3] >= 0
    z1, one = torch.zeros_like(nd[..., 0]), torch.ones_like(nd[..., 0])
    illum = torch.where(ok[..., None], f["radiance"][..., :3] / torch.clamp(mat[..., :3], min=1e-3),
                        torch.zeros_like(nd[..., :3]))
    L = _lum(illum)
    around = [(dy, dx) for dy in (-1, 0, 1) for dx in (-1, 0, 1)]
    live = {d: (_within(nd, *d) & _shift(ok, *d)).double() for d in around}
    cnt = torch.clamp(sum(live.values()), min=1.0)
    mu = sum(live[d][..., None] * _shift(illum, *d) for d in around) / cnt[..., None]
    slm = _lum(mu)
    var3 = sum(live[d][..., None] * (_shift(illum, *d) - mu) ** 2 for d in around) / cnt[..., None]
    svar = sum(live[d] * (_shift(L, *d) - slm) ** 2 for d in around) / cnt
    sd = torch.sqrt(torch.clamp(var3, min=1e-12))

    has = torch.zeros_like(ok)
    v, alpha, gamma = z1, one, one
    hc, hm = torch.zeros_like(illum), torch.zeros_like(nd)
    if st is not None:
        ys, xs = _grid(H, W, dev)
        px, py = xs + mv[..., 0], ys + mv[..., 1]
        bx, by = torch.floor(px), torch.floor(py)
        fx, fy = px - bx, py - by

        def tap(qy, qx):
            k = _pick(st["key"], qy, qx)
            good = (qx >= 0) & (qy >= 0) & (qx < W) & (qy < H) & (k[..., 2] >= 0) & (k[..., 3] == mv[..., 2])
            good &= (k[..., 2] - mv[..., 3]).abs() <= 0.05 * mv[..., 3] + 0.01
            good &= (_oct_dec(k[..., :2]) * nd[..., :3]).sum(-1) >= 0.9
            return good, _pick(st["hist"], qy, qx)[..., :3], _pick(st["mom"], qy, qx)

        sw = z1
        for i in range(4):
            good, c, m = tap(by.long() + (i >> 1), bx.long() + (i & 1))
            w = (fx if i & 1 else 1 - fx) * (fy if i >> 1 else 1 - fy)
            w = torch.where(good & (w > 0), w, z1)
            sw, hc, hm = sw + w, hc + w[..., None] * c, hm + w[..., None] * m
        near = sw >= 0.01
        s = torch.where(near, sw, one)[..., None]
        n3, hc3, hm3 = z1, torch.zeros_like(hc), torch.zeros_like(hm)
        cx, cy = torch.floor(px + 0.5).long(), torch.floor(py + 0.5).long()
        for dy, dx in around:
            good, c, m = tap(cy + dy, cx + dx)
            w = good.double()
            n3, hc3, hm3 = n3 + w, hc3 + w[..., None] * c, hm3 + w[..., None] * m
        s3 = torch.clamp(n3, min=1.0)[..., None]
        hc = torch.where(near[..., None], hc / s, hc3 / s3)
        hm = torch.where(near[..., None], hm / s, hm3 / s3)
        v = torch.where(near, sw, torch.where(n3 > 0, 0.1 * one, z1))
        has = (near | (n3 > 0)) & (hm[..., 3] > 0)
        p = st["par0"][cy.clamp(0, H - 1) >> 1, cx.clamp(0, W - 1) >> 1]
        alpha, gamma = p[..., 0], p[..., 1]
    v = torch.where(has, v, z1)
    lim = gamma[..., None] * sd
    hcl = torch.minimum(torch.maximum(hc, mu - lim), mu + lim)
    n = torch.clamp(hm[..., 3] + 1.0, max=32.0)
    a = torch.maximum(alpha, 1.0 / n)
    col = torch.where(has[..., None], hcl + (illum - hcl) * a[..., None], illum)
    m1 = torch.where(has, hm[..., 0] + (L - hm[..., 0]) * a, L)
    m2 = torch.where(has, hm[..., 1] + (L * L - hm[..., 1]) * a, L * L)
    fast = torch.where(has, hm[..., 2] + (L - hm[..., 2]) * torch.clamp(1.0 / n, min=1 / 6), L)
    length = torch.where(has, n, one)
    lh = _lum(hc)
    lag = torch.where(has, (slm - lh).abs() / (torch.sqrt(torch.clamp(svar / cnt, min=1e-12)) + 0.02 * lh + 1e-3), z1)
    tvar = torch.clamp(m2 - m1 * m1, min=0.0)
    A = torch.cat([col, (svar + (tvar - svar) * torch.clamp(length / 4, max=1.0))[..., None]], -1)
    oc = _oct_enc(nd[..., :3])
    zero4 = torch.zeros_like(nd)
    keep = ok[..., None]
    A0 = torch.where(keep, _store(A), zero4)
    mom = torch.where(keep, _store(torch.stack([m1, m2, fast, length], -1)), zero4)
    key = torch.where(keep, torch.cat([oc, nd[..., 3:4], mv[..., 2:3]], -1),
                      torch.stack([z1, z1, -one, mv[..., 2]], -1))

    # block features over 2x2 blocks
    E = exposure
    Aq, on = _qf16(A), _qf16(oc)
    q1, q2 = E * _qf16(m1), E * E * _qf16(m2)
    ns = _oct_dec(on)
    zq = _qf16(nd[..., 3])
    per = torch.stack([E * _lum(Aq), E * _qf16(L), torch.clamp(q2 - q1 * q1, min=0.0), length, _qf16(v), _qf16(lag),
                       E * _qf16(fast), q1, *ns.unbind(-1), *mat.unbind(-1), *Aq.unbind(-1),
                       _qf16(torch.hypot(mv[..., 0], mv[..., 1])), zq], -1)
    H2, W2 = (H + 1) // 2, (W + 1) // 2

    def blocks(t):
        t = torch.nn.functional.pad(t, (0,) * 2 * (t.dim() - 2) + (0, 2 * W2 - W, 0, 2 * H2 - H))
        return t.reshape(H2, 2, W2, 2, *t.shape[2:]).transpose(1, 2).reshape(H2, W2, 4, *t.shape[2:])

    okb = blocks(ok.double())
    nv = okb.sum(-1)
    okh = nv > 0
    k = 1.0 / torch.clamp(nv, min=1.0)
    pb = blocks(per)
    S = (torch.where(okb[..., None] > 0, pb, torch.zeros_like(pb)).sum(2)) * k[..., None]
    va = (okb * (pb[..., 0] - S[..., None, 0]) ** 2).sum(-1) * k
    lq = torch.nn.functional.pad(torch.where(ok, E * _qf16(L), z1), (1, 2 * W2 - W + 1, 1, 2 * H2 - H + 1))
    lw = torch.nn.functional.pad(ok.double(), (1, 2 * W2 - W + 1, 1, 2 * H2 - H + 1))
    win = [(slice(i, i + 2 * H2, 2), slice(j, j + 2 * W2, 2)) for i in range(4) for j in range(4)]
    n4 = torch.clamp(sum(lw[w] for w in win), min=1.0)
    mu4 = sum(lw[w] * lq[w] for w in win) / n4
    var4 = sum(lw[w] * (lq[w] - mu4) ** 2 for w in win) / n4
    nn = S[..., 8:11] / torch.clamp(S[..., 8:11].norm(dim=-1, keepdim=True), min=1e-6)
    big = torch.full_like(okb, 1e30)
    zb = pb[..., 20]
    zmax, zmin = torch.where(okb > 0, zb, -big).amax(-1), torch.where(okb > 0, zb, big).amin(-1)
    mind = torch.where(okb > 0, (pb[..., 8:11] * nn[..., None, :]).sum(-1), big).amin(-1)
    dz = torch.clamp((zmax - zmin) / torch.clamp(zmin, min=1e-6), 0.0, 1.0)
    dn = torch.clamp(1.0 - mind, 0.0, 2.0)
    ob = _oct_enc(nn)
    log1 = lambda x: torch.log(1.0 + x)  # noqa: E731
    fe = torch.stack([log1(S[..., 0]), log1(S[..., 1]), log1(S[..., 2]), log1(var4), S[..., 3] / 32, S[..., 4],
                      log1(S[..., 5]), log1((S[..., 6] - S[..., 7]).abs() / (S[..., 7] + 1e-3)), ob[..., 0], ob[..., 1],
                      dz, dn, *S[..., 11:15].unbind(-1), 1.0 - nv / 4, log1(S[..., 19]), log1(mu4), log1(va)], -1)
    hz = torch.zeros_like(S[..., :4])
    texel = lambda x: torch.where(okh[..., None], _store(_qf16(x)), torch.zeros_like(x))  # noqa: E731
    gn = _oct_dec(texel(ob))
    gz = torch.where(okh, _store(_qf16(S[..., 20])), -torch.ones_like(nv))
    return {"A0": A0, "mom": mom, "key": _store(key), "features": texel(fe), "ok": okh, "Ah": torch.where(
        okh[..., None], _store(_qf16(S[..., 15:19])), hz), "Gd": torch.cat([gn, gz[..., None]], -1), "count": nv}


def _mlp(fe, theta, ok):
    """The 20-16-16-12 network and its output heads; zeros on blocks without a surface."""
    w1, b1, w2, b2 = theta[:320].view(16, 20), theta[320:336], theta[336:592].view(16, 16), theta[592:608]
    w3, b3 = theta[608:800].view(12, 16), theta[800:812]
    o = torch.relu(torch.relu(fe @ w1.T + b1) @ w2.T + b2) @ w3.T + b3
    sg = torch.sigmoid
    par = torch.stack([1 / 32 + 31 / 32 * sg(o[..., 0]), 0.5 + 7.5 * sg(o[..., 1]), sg(o[..., 2]), sg(o[..., 3])]
                      + [0.25 * torch.exp(torch.clamp(o[..., i], -5, 5)) for i in range(4, 8)]
                      + [torch.exp(torch.clamp(o[..., i], -4, 4)) for i in range(8, 12)], -1)
    return torch.where(ok[..., None], par, torch.zeros_like(par))


def _coarse(t):
    """The two quarter-resolution levels: (C0, decoded guide)."""
    Ah, Gd, n = t["Ah"], t["Gd"], t["count"]
    h, w = n.shape
    qh, qw = (h + 1) // 2, (w + 1) // 2
    pad = lambda x: torch.nn.functional.pad(x, (0,) * 2 * (x.dim() - 2) + (0, 2 * qw - w, 0, 2 * qh - h))  # noqa: E731
    q = lambda x: pad(x).reshape(qh, 2, qw, 2, *x.shape[2:])  # noqa: E731
    nb = q(n)[..., None]
    N = nb.sum((1, 3))
    Ns = torch.clamp(N, min=1.0)
    S = (nb * q(torch.cat([Ah, Gd], -1))).sum((1, 3))
    nn = S[..., 4:7] / torch.clamp(S[..., 4:7].norm(dim=-1, keepdim=True), min=1e-6)
    surf = N > 0
    c = torch.where(surf, _qf16(torch.cat([S[..., :3] / Ns, S[..., 3:4] / Ns / Ns], -1)), torch.zeros_like(S[..., :4]))
    g = _qf16(torch.cat([_oct_enc(nn), S[..., 7:8] / Ns], -1))
    g = torch.where(surf, g, torch.tensor([0.0, 0.0, -1.0], dtype=g.dtype, device=g.device))
    dec = lambda g: torch.cat([_oct_dec(g[..., :2]), g[..., 2:3]], -1)  # noqa: E731
    C1 = _store(_atrous(c, dec(g), 0.25, 1.0, 1, True, R=2))
    gs = dec(_store(g))
    return _store(_atrous(C1, gs, 0.25, 1.0, 2, True, R=2)), gs


def _upsample(guide, images, n, z, scale):
    """Joint-bilinear weights of the four texels around each pixel: (sum of weights, weighted sums of the images)."""
    H, W = z.shape
    ys, xs = _grid(H, W, z.device)
    py, px = (ys + 0.5) / scale - 0.5, (xs + 0.5) / scale - 0.5
    by, bx = torch.floor(py), torch.floor(px)
    fy, fx = py - by, px - bx
    sw, out = torch.zeros_like(z), [0.0 for _ in images]
    for j in range(4):
        qy, qx = by.long() + (j >> 1), bx.long() + (j & 1)
        g = _pick(guide, qy, qx)
        ok = (qx >= 0) & (qy >= 0) & (qx < guide.shape[1]) & (qy < guide.shape[0]) & (g[..., 3] >= 0)
        w = (fx if j & 1 else 1 - fx) * (fy if j >> 1 else 1 - fy)
        w = w * torch.exp(-(g[..., 3] - z).abs() / (0.05 * z + 1e-3)) * torch.clamp(
            (g[..., :3] * n).sum(-1), min=0.0) ** 8
        w = torch.where(ok, w, torch.zeros_like(w))
        sw = sw + w
        out = [o + w[..., None] * _pick(im, qy, qx)[..., :3] for o, im in zip(out, images)]
    return sw, out


def _fine(f, t, par, B3, C0, CG, quantise):
    """Fine level and recombination: (A1, X)."""
    H, W = t["A0"].shape[:2]
    ys, xs = _grid(H, W, B3.device)
    surf = t["key"][..., 2] >= 0
    p = par[ys >> 1, xs >> 1]
    safe = torch.where(surf[..., None], p, torch.ones_like(p))
    G = torch.cat([_oct_dec(t["key"][..., :2]), t["key"][..., 2:3]], -1)
    A1 = _atrous(t["A0"], G, safe[..., 4], safe[..., 8], 1, True)
    c = quantise(A1)[..., :3]
    z = torch.where(surf, G[..., 3], torch.ones_like(G[..., 3]))
    sw, (uB, uA) = _upsample(t["Gd"], [B3, t["Ah"]], G[..., :3], z, 2.0)
    s = torch.where(sw > 1e-4, sw, torch.ones_like(sw))[..., None]
    ill = torch.where((sw > 1e-4)[..., None], uB / s + p[..., 3:4] * (c - uA / s), c)
    sw, (uC,) = _upsample(CG, [C0], G[..., :3], z, 4.0)
    s = torch.where(sw > 1e-4, sw, torch.ones_like(sw))[..., None]
    up = torch.where((sw > 1e-4)[..., None], uC / s, ill)
    ill = ill + (up - ill) * p[..., 2:3]
    emi = f["emission"][..., :3]
    return A1, torch.where(surf[..., None], ill * f["material"][..., :3] + emi, emi)


def _taa(X, prev, mv):
    cur = _tm(X)
    if prev is None:
        return _itm(cur)
    Y = _ycocg(cur)
    win = [_shift(Y, dy, dx) for dy in (-1, 0, 1) for dx in (-1, 0, 1)]
    m = sum(win) / 9
    sd = torch.sqrt(torch.clamp(sum((y - m) ** 2 for y in win) / 9, min=1e-12))
    hist, inside = _bilinear(prev, mv, *X.shape[:2])
    hr = _rgb(torch.minimum(torch.maximum(_ycocg(_tm(hist)), m - 1.25 * sd), m + 1.25 * sd))
    return _itm(torch.where(inside[..., None], hr + (cur - hr) * 0.1, cur))


def _with_alpha(c):
    return torch.cat([c, torch.ones_like(c[..., :1])], -1)


def _denoise_frame(f, st, theta):
    """One denoised frame with every image stored as float16: the next state, its "taa" being the output."""
    t = _temporal(f, st, 1.0)
    par = _store(_mlp(t["features"], theta, t["ok"]))
    one = torch.where(t["ok"][..., None], par, torch.ones_like(par))
    B = t["Ah"]
    for i, step in ((1, 1), (2, 2), (3, 4)):
        B = _store(_atrous(B, t["Gd"], one[..., 4 + i], one[..., 8 + i], step, i == 1))
    C0, CG = _coarse(t)
    A1, X = _fine(f, t, par, B, C0, CG, _qf16)
    out = _store(_taa(_store(X), None if st is None else st["taa"], f["motion"]))
    return {"hist": _store(A1), "mom": t["mom"], "key": t["key"], "par0": par[..., :4], "taa": _with_alpha(out)}


def _weights64(dev):
    return torch.from_numpy(builtin_weights().view(np.float16).astype(np.float64)).to(dev)


def _exact_denoise(case, seed):
    frames = _frames(case, seed, HISTORY + 1)
    theta, st = _weights64("cuda"), None
    for fr in frames:
        st = _denoise_frame(_as64(fr), st, theta)
    return st["taa"]


# ------------------------------------------------------------------------------------- float64: SVGF
def _svgf_frame(g, st, iterations, taa):
    nd, mv, mat = (g[k].double() for k in ("normalDepth", "motion", "material"))
    pnd, pmv = g["prevNormalDepth"].double(), g["prevMotion"].double()
    H, W = nd.shape[:2]
    ok = nd[..., 3] >= 0
    keep = ok[..., None]
    z1, one = torch.zeros_like(nd[..., 0]), torch.ones_like(nd[..., 0])
    illum = g["radiance"].double()[..., :3] / torch.clamp(mat[..., :3], min=1e-3)
    L = _lum(illum)
    col, m1, m2, length = illum, L, L * L, one
    if st is not None:
        ys, xs = _grid(H, W, nd.device)
        px, py = xs + mv[..., 0], ys + mv[..., 1]
        bx, by = torch.floor(px), torch.floor(py)
        fx, fy = px - bx, py - by

        def tap(qy, qx):
            n = _pick(pnd, qy, qx)
            good = (qx >= 0) & (qy >= 0) & (qx < W) & (qy < H) & (n[..., 3] >= 0)
            good &= _pick(pmv, qy, qx)[..., 2] == mv[..., 2]
            good &= (n[..., 3] - mv[..., 3]).abs() <= 0.05 * mv[..., 3] + 0.01
            good &= (n[..., :3] * nd[..., :3]).sum(-1) >= 0.9
            return good, torch.cat([_pick(st["hist"], qy, qx)[..., :3], _pick(st["mom"], qy, qx)[..., :3]], -1)

        sw, acc = z1, 0.0
        for i in range(4):
            good, h = tap(by.long() + (i >> 1), bx.long() + (i & 1))
            w = (fx if i & 1 else 1 - fx) * (fy if i >> 1 else 1 - fy)
            w = torch.where(good & (w > 0), w, z1)
            sw, acc = sw + w, acc + w[..., None] * h
        far = sw < 0.01
        cx, cy = torch.round(px).long(), torch.round(py).long()
        s3, a3 = sw, acc
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                good, h = tap(cy + dy, cx + dx)
                s3, a3 = s3 + good.double(), a3 + good.double()[..., None] * h
        sw, acc = torch.where(far, s3, sw), torch.where(far[..., None], a3, acc)
        has = sw >= 0.01
        h = acc / torch.where(has, sw, one)[..., None]
        n = torch.clamp(h[..., 5] + 1.0, max=64.0)
        a = torch.clamp(1.0 / n, min=0.2)
        col = torch.where(has[..., None], h[..., :3] * (1 - a)[..., None] + illum * a[..., None], illum)
        m1, m2 = torch.where(has, h[..., 3] * (1 - a) + L * a, L), torch.where(has, h[..., 4] * (1 - a) + L * L * a, L * L)
        length = torch.where(has, n, one)
    zero3 = torch.zeros_like(illum)
    tmp = torch.where(keep, _store(col), zero3)
    mom = torch.where(keep, _store(torch.stack([m1, m2, length], -1)), zero3)
    # variance: temporal with a long enough history, else from a 7 x 7 neighbourhood
    sw, acc = z1, 0.0
    for dy in range(-3, 4):
        for dx in range(-3, 4):
            q = _shift(nd, dy, dx)
            w = torch.exp(-(q[..., 3] - nd[..., 3]).abs() / (0.02 * nd[..., 3].abs() * math.hypot(dx, dy) + 1e-3))
            w = w * torch.clamp((q[..., :3] * nd[..., :3]).sum(-1), min=0.0) ** 128
            w = torch.where(_within(nd, dy, dx) & (q[..., 3] >= 0), w, z1)
            sw = sw + w
            acc = acc + w[..., None] * torch.cat([_shift(tmp, dy, dx), _shift(mom, dy, dx)[..., :2]], -1)
    acc = acc / torch.clamp(sw, min=1e-6)[..., None]
    spatial = torch.cat([acc[..., :3], (torch.clamp(acc[..., 4] - acc[..., 3] ** 2, min=0.0) * 4 /
                                        torch.clamp(mom[..., 2], min=1.0))[..., None]], -1)
    temporal = torch.cat([tmp, torch.clamp(mom[..., 1] - mom[..., 0] ** 2, min=0.0)[..., None]], -1)
    A = _store(torch.where((mom[..., 2] >= 4)[..., None], temporal, spatial))
    A = torch.where(keep, A, torch.zeros_like(A))
    z = nd[..., 3]
    zg = torch.where(ok, _depth_slope(z), one)
    hw, hist = SPLINE[2], None
    for it in range(iterations):
        step = 1 << it
        scale = 4.0 * torch.sqrt(torch.clamp(_blur3(A[..., 3]), min=0.0)) + 1e-6
        lc = _lum(A)
        wt = hw[2] * hw[2] * one
        c3, var = A[..., :3] * wt[..., None], A[..., 3] * wt * wt
        for dy in range(-2, 3):
            for dx in range(-2, 3):
                if dx == 0 and dy == 0:
                    continue
                q, a = _shift(nd, dy * step, dx * step), _shift(A, dy * step, dx * step)
                w = hw[dy + 2] * hw[dx + 2] * torch.clamp((q[..., :3] * nd[..., :3]).sum(-1), min=0.0) ** 128
                w = w * torch.exp(-(q[..., 3] - z).abs() / (zg * math.hypot(dx, dy) * step + 1e-3)
                                  - (_lum(a) - lc).abs() / scale)
                w = torch.where(_within(nd, dy * step, dx * step) & (q[..., 3] >= 0), w, z1)
                wt, c3, var = wt + w, c3 + w[..., None] * a[..., :3], var + w * w * a[..., 3]
        A = _store(torch.cat([c3 / wt[..., None], (var / (wt * wt))[..., None]], -1))
        A = torch.where(keep, A, torch.zeros_like(A))
        hist = A if it == 0 else hist
    X = A[..., :3] * mat[..., :3] + g["emission"].double()[..., :3]
    cur = _tm(X)
    res = cur
    if taa and st is not None:
        Y = _ycocg(cur)
        win = [_shift(Y, dy, dx) for dy in (-1, 0, 1) for dx in (-1, 0, 1)]
        m = sum(win) / 9
        sd = torch.sqrt(torch.clamp(sum(y * y for y in win) / 9 - m * m, min=0.0))
        old, inside = _bilinear(st["taa"], mv, H, W)
        hr = _rgb(torch.minimum(torch.maximum(_ycocg(_tm(old)), m - 1.25 * sd), m + 1.25 * sd))
        res = torch.where(inside[..., None], hr * 0.9 + cur * 0.1, cur)
    return {"hist": hist, "mom": mom, "taa": _with_alpha(_store(_itm(res)))}


def _exact_svgf(case, seed):
    frames, st = _frames(case, seed, HISTORY + 1), None
    for t in range(HISTORY + 1):
        st = _svgf_frame(_svgf_inputs(frames, t), st, case["iterations"], case["taa"])
    return st["taa"]


# ------------------------------------------------------------------------------------- float64: the post
def _sample(img, u, v):
    h, w = img.shape[:2]
    x, y = u * w - 0.5, v * h - 0.5
    x0, y0 = torch.floor(x), torch.floor(y)
    fx, fy = (x - x0)[None, :, None], (y - y0)[:, None, None]
    xa, xb = x0.long().clamp(0, w - 1), (x0.long() + 1).clamp(0, w - 1)
    ya, yb = y0.long().clamp(0, h - 1), (y0.long() + 1).clamp(0, h - 1)
    row = lambda y: img[y][:, xa] * (1 - fx) + img[y][:, xb] * fx  # noqa: E731
    return row(ya) * (1 - fy) + row(yb) * fy


def _fragments(w, h):
    ar = lambda n: (torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) / n  # noqa: E731
    return ar(w), ar(h)


def _agx(c):
    def mat(rows):
        return torch.tensor(rows, dtype=torch.float64, device="cuda").view(3, 3).T

    def mul(rows, c):  # rows: the matrix column by column
        return c @ mat(rows).T
    to2020 = (0.6274, 0.0691, 0.0164, 0.3293, 0.9195, 0.0880, 0.0433, 0.0113, 0.8956)
    to_srgb = (1.6605, -0.1246, -0.0182, -0.5876, 1.1329, -0.1006, -0.0728, -0.0083, 1.1187)
    inset = (0.856627153315983, 0.137318972929847, 0.11189821299995, 0.0951212405381588, 0.761241990602591,
             0.0767994186031903, 0.0482516061458583, 0.101439036467562, 0.811302368396859)
    outset = (1.1271005818144368, -0.1413297634984383, -0.14132976349843826, -0.11060664309660323, 1.157823702216272,
              -0.11060664309660294, -0.016493938717834573, -0.016493938717834257, 1.2519364065950405)
    c = mul(inset, mul(to2020, c))
    x = torch.clamp((torch.log2(torch.clamp(c, min=1e-10)) + 12.47393) / (4.026069 + 12.47393), 0.0, 1.0)
    c = 15.5 * x**6 - 40.14 * x**5 + 31.96 * x**4 - 6.868 * x**3 + 0.4298 * x**2 + 0.1191 * x - 0.00232
    luma = _lum(c)[..., None]
    c = luma + (torch.clamp(c, min=0.0) ** 1.22 - luma) * 1.15
    return torch.clamp(mul(to_srgb, torch.clamp(mul(outset, c), min=0.0) ** 2.2), 0.0, 1.0)


def _exact_post(case, seed):
    if case["format"] != "rgba32float":
        return None  # bytes
    left, right = _post_images(case, seed)
    H, W = left.shape[:2]
    at32 = lambda n: (torch.arange(n, device="cuda", dtype=torch.float32) + 0.5) / n  # noqa: E731
    u32 = at32(W)  # the split and line tests are defined on the 32-bit fragment position
    split = torch.tensor(case["split"], dtype=torch.float32, device="cuda")
    hdr = torch.where((u32 < split)[None, :, None], left, right).double()[..., :3]
    hdr = _store(torch.clamp(hdr, min=0.0))
    levels, src = [], hdr
    for i in range(6):
        w, h = max(1, W >> (i + 1)), max(1, H >> (i + 1))
        u, v = _fragments(w, h)
        tx, ty = 1.0 / src.shape[1], 1.0 / src.shape[0]
        s = lambda dx, dy: _sample(src, u + dx * tx, v + dy * ty)  # noqa: B023, E731
        a, b, c, d, e, f, g, k, m = (s(dx, dy) for dy in (-2, 0, 2) for dx in (-2, 0, 2))
        inner = s(-1, -1) + s(1, -1) + s(-1, 1) + s(1, 1)
        if i == 0:
            quads = [(a + b + d + e) / 4, (b + c + e + f) / 4, (d + e + g + k) / 4, (e + f + k + m) / 4, inner / 4]
            ws = [wt / (1.0 + _lum(q)) for q, wt in zip(quads, (0.125,) * 4 + (0.5,))]
            o = sum(q * wt[..., None] for q, wt in zip(quads, ws)) / sum(ws)[..., None]
        else:
            o = e / 8 + (a + c + g + m) / 32 + (b + d + f + k) / 16 + inner / 8
        src = _store(o)
        levels.append(src)

    def tent(img, u, v):
        tx, ty = 1.0 / img.shape[1], 1.0 / img.shape[0]
        return sum(_sample(img, u + dx * tx, v + dy * ty) * ((2 - abs(dx)) * (2 - abs(dy)))
                   for dx in (-1, 0, 1) for dy in (-1, 0, 1)) / 16
    for i in range(5, 0, -1):
        dst = levels[i - 1]
        levels[i - 1] = _store(dst + tent(levels[i], *_fragments(dst.shape[1], dst.shape[0])))
    u, v = _fragments(W, H)
    c = _sample(hdr, u, v) * 0.97 + tent(levels[0], u, v) * 0.03
    vig = 0.65 + 0.35 * (1.0 - ((u - 0.5)[None, :] ** 2 + ((v - 0.5) * 0.75)[:, None] ** 2) * 1.6)
    t = _agx(c * vig[..., None])
    o = torch.where(t <= 0.0031308, t * 12.92, 1.055 * t ** (1 / 2.4) - 0.055)
    line = (u32 - split).abs() * torch.tensor(float(W), device="cuda") < 1.5
    return _with_alpha(torch.where(line[None, :, None], o * 0.15 + 0.85, o))


# ------------------------------------------------------------------------------------- float64: the trainer's frame
def _exact_train_frame(case, seed):
    if case["mlp"] != "fp32":
        return None  # the caller chose 16-bit operands: no 64-bit value is what these forms return
    sc = _train_scene(case["size"], 2, seed)
    fr = [frame_device(sc, t, clean=True) for t in range(2)]
    theta = torch.from_numpy(xavier_init(seed).astype(np.float64)).cuda().requires_grad_(True)
    st = out_prev = None
    for t in range(2):
        f = _as64(fr[t])
        with torch.no_grad():
            tm = _temporal(f, st, 1.0)
            C0, CG = _coarse(tm)
        par = _mlp(tm["features"], theta, tm["ok"])
        par.retain_grad()
        one = torch.where(tm["ok"][..., None], par, torch.ones_like(par))
        B = tm["Ah"]
        for i, step in ((1, 1), (2, 2), (3, 4)):
            B = _atrous(B, tm["Gd"], one[..., 4 + i], one[..., 8 + i], step, i == 1)
        A1, X = _fine(f, tm, par, B, C0, CG, lambda x: x)
        out = _taa(X, None if st is None else st["taa"], f["motion"])
        if t == 0:
            with torch.no_grad():
                st = {"hist": _store(A1), "mom": tm["mom"], "key": tm["key"], "par0": _store(par[..., :4]),
                      "taa": _with_alpha(_store(out))}
                out_prev = out.detach()
    clean, before = fr[1]["clean"].double(), fr[0]["clean"].double()
    den = clean.abs() + 1e-2
    loss = (torch.clamp((out - clean).abs() / den, max=1.0)
            + LAMBDA_T * torch.clamp(((out - out_prev) - (clean - before)).abs() / den, max=1.0)).mean()
    loss.backward()
    return {"out": _with_alpha(out.detach()), "par": par.detach(), "dpar": par.grad, "grad": theta.grad}


def exact(case, seed):
    kind = case["kind"]
    if kind == "train_frame":
        return _exact_train_frame(case, seed)
    with torch.no_grad():
        if kind == "denoise":
            return _exact_denoise(case, seed)
        if kind == "svgf":
            return _exact_svgf(case, seed)
        if kind == "post":
            return _exact_post(case, seed)
    # a path tracer's samples follow decisions on 32-bit values: no 64-bit value exists per pixel. A training step is
    # minutes of float64 autograd.
    return None
