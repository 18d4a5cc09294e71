"""The workloads this framework's speed is judged by, through its public entry
points (the Python binding of libbm4dof_gpu.so).

A case is a dict of plain values.  "kind" says which entry point it goes
through:

  denoise  Context.runNlBayes on CUDA tensors: both steps of the denoiser
  batch    Context.run_batched: several uneven sequences in one CUDA graph
  tvl1     Context.tvl1_video: optical flow of a host video
  train    Trainer.step: one training step of the gain network

"preset" names the denoiser's parameters: video4 (4x4x4 patches, 16 similar
patches, 21x21 search window, +-4 frames: the benchmark's), image8 (8x8
patches, 16 similar patches, 21x21 window: the image benchmark's) and default
(what the command line takes when no flag is given: 39x39 windows for images;
8x8 and 7x7 patches, 7x7 windows, 8 similar patches for video).  "form" is the
variant: plain, mixed, learned, learned_mixed, vbm3d (predictive search).

Inputs are made on the GPU from the seed: a texture of cosines and constant
rectangles moved by a pan with a little zoom and rotation, opaque rectangles
moving on top, the flow of that motion with the smooth errors of an estimated
flow, and white Gaussian noise.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "bm4d-of_gb300"))

import bm4dof  # noqa: E402
import train_gains  # noqa: E402

PRESETS = {
    "video4": dict(px1=4, px2=4, pt1=4, pt2=4, wx1=21, wx2=21, np1=16, np2=16, b1=3.0),
    "image8": dict(px1=8, px2=8, pt1=1, pt2=1, wx1=21, wx2=21, np1=16, np2=16, b1=3.0),
    "default": dict(),
}


def _denoise(name, W, H, F, C, sigma, preset, form="plain", flow=True, nparts=2):
    case = dict(kind="denoise", W=W, H=H, F=F, C=C, sigma=sigma, preset=preset, form=form, flow=flow and F > 1,
                nparts=nparts)
    return dict(name=name, **case) if name else case


def listed():
    return [
        # one small grey image: the shortest call, where launches and host work count
        _denoise("image_256", 256, 256, 1, 1, 20.0, "image8"),
        # a colour photograph of odd size denoised with the command line's defaults
        _denoise("image_rgb_default", 767, 511, 1, 3, 25.0, "default"),
        # an ordinary clip with the benchmark's parameters (its second configuration)
        _denoise("video_480", 854, 480, 20, 1, 20.0, "video4"),
        # a full-HD clip: the largest call
        _denoise("video_hd", 1920, 1080, 24, 1, 20.0, "video4"),
        # a colour clip: step 2 compares and filters three channels
        _denoise("video_rgb", 640, 360, 14, 3, 20.0, "video4"),
        # a clip with the command line's defaults, odd size, on many tiles as the
        # reference makes them on a many-core host
        _denoise("video_default", 853, 481, 16, 1, 20.0, "default", nparts=8),
        # the predictive search with its own defaults, colour, high noise
        _denoise("vbm3d_default", 720, 576, 14, 3, 40.0, "default", form="vbm3d"),
        # the predictive search on the benchmark's patches
        _denoise("vbm3d_480", 854, 480, 12, 1, 20.0, "video4", form="vbm3d"),
        # the fast form: one pass with the gain network, tensor-core patch search
        _denoise("learned_mixed_480", 854, 480, 16, 1, 20.0, "video4", form="learned_mixed"),
        # many uneven sequences at once, as a server denoises them
        dict(name="batch_8", kind="batch", n=8, W=320, H=240, F=6, spread=2.0, sigma=20.0, form="plain"),
        # the optical flow the denoiser takes, from a video on the host
        dict(name="tvl1_360", kind="tvl1", W=640, H=360, F=10),
        # one step of training the gain network at its usual batch
        dict(name="train_step", kind="train", rows=8192),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    what = rng.choice(["image", "image_default", "video", "video", "video", "default", "vbm3d", "batch", "tvl1", "train"])
    sigma = float(rng.choice([5, 10, 20, 30, 40]))
    C = rng.choice([1, 1, 3])
    if what == "image":
        return _denoise(None, _log(rng, 64, 1400), _log(rng, 64, 1000), 1, C, sigma, "image8", nparts=rng.choice([2, 4, 16]))
    if what == "image_default":
        return _denoise(None, _log(rng, 96, 1000), _log(rng, 96, 800), 1, C, sigma, "default", nparts=rng.choice([2, 8]))
    if what == "batch":
        return dict(kind="batch", n=rng.randint(2, 10), W=_log(rng, 120, 480), H=_log(rng, 100, 320), F=rng.randint(4, 8),
                    spread=rng.uniform(1.0, 2.0), sigma=sigma, form="plain")
    if what == "tvl1":
        return dict(kind="tvl1", W=_log(rng, 96, 960), H=_log(rng, 80, 540), F=rng.randint(2, 12))
    if what == "train":
        return dict(kind="train", rows=_log(rng, 300, 8192))
    W, H, F = _log(rng, 64, 1000), _log(rng, 64, 600), rng.randint(4, 20)
    F = max(4, min(F, int(9e6 / (W * H * C))))
    nparts = rng.choice([2, 2, 4, 16])
    if what == "video":
        form = rng.choice(["plain", "plain", "mixed", "learned", "learned_mixed"] if C == 1 else ["plain", "plain", "mixed"])
        return _denoise(None, W, H, F, C, sigma, "video4", form=form, flow=rng.random() < 0.8, nparts=nparts)
    if what == "default":
        return _denoise(None, W, H, F, C, sigma, "default", flow=rng.random() < 0.8, nparts=nparts)
    return _denoise(None, W, H, F, C, sigma, rng.choice(["default", "video4"]), form="vbm3d", flow=rng.random() < 0.8,
                    nparts=nparts)


# ---- inputs -----------------------------------------------------------------

def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float32)


def _texture(W, H, C, g):
    """(C, H, W): 64 cosines of amplitude 1/f per channel, rescaled to 16..240,
    and 8 constant rectangles shared by the channels."""
    x = torch.arange(W, device="cuda", dtype=torch.float32)
    y = torch.arange(H, device="cuda", dtype=torch.float32)
    img = torch.zeros(C, H, W, device="cuda")
    r = _rand(g, 3, C, 64)
    f = (0.25 * r[0]).clamp(min=1.0 / max(W, H))
    th, ph = 2 * math.pi * r[1], 2 * math.pi * r[2]
    a, b = 2 * math.pi * f * torch.cos(th), 2 * math.pi * f * torch.sin(th)
    for k in range(64):
        for c in range(C):
            u, v = a[c, k] * x + ph[c, k], b[c, k] * y
            img[c] += (torch.cos(v)[:, None] * torch.cos(u)[None] - torch.sin(v)[:, None] * torch.sin(u)[None]) / f[c, k]
    lo, hi = img.amin((1, 2), True), img.amax((1, 2), True)
    img = 16 + (img - lo) * (224 / (hi - lo))
    q = _rand(g, 8, 5).cpu().numpy()
    for k in range(8):
        w, h = int(16 + q[k, 0] * min(80, W - 16)), int(16 + q[k, 1] * min(80, H - 16))
        x0, y0 = int(q[k, 2] * max(1, W - w)), int(q[k, 3] * max(1, H - h))
        img[:, y0:y0 + h, x0:x0 + w] = float(16 + 224 * q[k, 4])
    return img


def _sample(img, X, Y):
    """img (C, H, W) at (X, Y), bilinear, borders clamped."""
    H, W = img.shape[1:]
    X, Y = X.clamp(0, W - 1), Y.clamp(0, H - 1)
    x0, y0 = X.floor().long(), Y.floor().long()
    x1, y1 = (x0 + 1).clamp(max=W - 1), (y0 + 1).clamp(max=H - 1)
    fx, fy = X - x0, Y - y0
    top = img[:, y0, x0] * (1 - fx) + img[:, y0, x1] * fx
    bot = img[:, y1, x0] * (1 - fx) + img[:, y1, x1] * fx
    return top * (1 - fy) + bot * fy


def _video(W, H, F, C, seed):
    """Clean video (F, C, H, W) and forward and backward flow (F, 2, H, W)."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)
    base = _texture(W, H, C, g)
    if F == 1:
        return base[None].contiguous(), None, None
    x = torch.arange(W, device="cuda", dtype=torch.float32)[None, :].expand(H, W)
    y = torch.arange(H, device="cuda", dtype=torch.float32)[:, None].expand(H, W)
    cx, cy = (W - 1) / 2, (H - 1) / 2
    step = _rand(g, F, 4).double().cpu().numpy()
    # frame k shows the base at p = A_k (x - c) + c + s_k
    A, s = [np.eye(2)], [np.zeros(2)]
    for k in range(1, F):
        z, rot = 1 + 0.002 * (step[k, 2] - 0.5), 0.002 * (step[k, 3] - 0.5)
        A.append(A[-1] @ (z * np.array([[math.cos(rot), -math.sin(rot)], [math.sin(rot), math.cos(rot)]])))
        s.append(s[-1] + A[-1] @ (4 * step[k, :2] - 2))
    q = _rand(g, 4, 7).cpu().numpy()
    movers = []
    for k in range(4):
        w, h = int(16 + q[k, 0] * min(80, W - 16)), int(16 + q[k, 1] * min(80, H - 16))
        movers.append((int(q[k, 2] * max(1, W - w)), int(q[k, 3] * max(1, H - h)), w, h, float(16 + 224 * q[k, 4]),
                       float(4 * q[k, 5] - 2), float(4 * q[k, 6] - 2)))

    def flow(k, n):   # displacement of the background from frame k to frame n
        B = np.linalg.inv(A[n])
        M, o = B @ A[k], B @ (s[k] - s[n])
        dx, dy = x - cx, y - cy
        return torch.stack([float(M[0, 0]) * dx + float(M[0, 1]) * dy + float(o[0]) - dx,
                            float(M[1, 0]) * dx + float(M[1, 1]) * dy + float(o[1]) - dy])

    clean = torch.empty(F, C, H, W, device="cuda")
    ff, bf = torch.empty(F, 2, H, W, device="cuda"), torch.empty(F, 2, H, W, device="cuda")
    for k in range(F):
        dx, dy = x - cx, y - cy
        clean[k] = _sample(base, float(A[k][0, 0]) * dx + float(A[k][0, 1]) * dy + cx + float(s[k][0]),
                           float(A[k][1, 0]) * dx + float(A[k][1, 1]) * dy + cy + float(s[k][1]))
        ff[k] = flow(k, min(k + 1, F - 1))
        bf[k] = flow(k, max(k - 1, 0))
        # the smooth errors of an estimated flow
        for f in (ff, bf):
            e = torch.randn(1, 2, max(2, H // 24), max(2, W // 24), generator=g, device="cuda") * 0.15
            f[k] += torch.nn.functional.interpolate(e, size=(H, W), mode="bilinear", align_corners=True)[0]
        for (x0, y0, w, h, level, vx, vy) in movers:
            xa, ya = int(math.floor(x0 + k * vx + 0.5)), int(math.floor(y0 + k * vy + 0.5))
            sl = (slice(max(0, ya), max(0, min(H, ya + h))), slice(max(0, xa), max(0, min(W, xa + w))))
            clean[(k, slice(None)) + sl] = level
            for f, sg in ((ff, 1.0), (bf, -1.0)):
                f[(k, 0) + sl], f[(k, 1) + sl] = sg * vx, sg * vy
    ff[F - 1], bf[0] = ff[F - 2], bf[1]
    return clean, ff, bf


def _noisy(clean, sigma, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 104729 + 3)
    return clean + sigma * torch.randn(clean.shape, generator=g, device="cuda")


def _params(case):
    return bm4dof.cli_params((case["W"], case["H"], case["F"], case["C"]), case["sigma"], **PRESETS[case["preset"]])


def _form(case):
    f = case["form"]
    kw = {}
    if "mixed" in f:
        kw["mixed"] = True
    if "learned" in f:
        kw["learned"] = True
    if f == "vbm3d":
        kw["vbm3d"] = True
    return kw


def _batch_cases(case, seed):
    rng = np.random.default_rng(int(seed) % 1000003 + 1)
    out = []
    for i in range(case["n"]):
        k = case["spread"] ** rng.uniform(-0.5, 0.5, 3)
        out.append(dict(W=int(case["W"] * k[0]), H=int(case["H"] * k[1]), F=max(4, int(round(case["F"] * k[2]))), C=1,
                        sigma=case["sigma"], preset="video4", form=case["form"], flow=True, nparts=2))
    return out


_contexts = {}


def _context(learned):
    """The device context a program keeps for its life (one with the trained
    gain network installed)."""
    if learned not in _contexts:
        ctx = bm4dof.Context(0)
        if learned:
            ctx.set_gain_network(train_gains.load_weights())
        _contexts[learned] = ctx
    return _contexts[learned]


def prepare(case, seed):
    if case["kind"] == "denoise":
        clean, ff, bf = _video(case["W"], case["H"], case["F"], case["C"], seed)
        nz = _noisy(clean, case["sigma"], seed)
        if not case["flow"]:
            ff = bf = None
        return dict(case=case, ctx=_context("learned" in case["form"]), noisy=nz, ff=ff, bf=bf, params=_params(case),
                    basic=torch.empty_like(nz), final=torch.empty_like(nz))
    if case["kind"] == "batch":
        items = []
        # the sizes belong to the case, the pictures to the seed
        for i, c in enumerate(_batch_cases(case, case["n"] * 31 + case["W"])):
            clean, ff, bf = _video(c["W"], c["H"], c["F"], 1, int(seed) * 64 + i)
            nz = _noisy(clean, c["sigma"], int(seed) * 64 + i)
            p1, p2 = _params(c)
            items.append(dict(noisy=nz, fflow=ff, bflow=bf, basic=torch.empty_like(nz), final=torch.empty_like(nz),
                              p1=p1, p2=p2, nparts=c["nparts"]))
        # a server refills the same buffers and replays: the context is its own
        return dict(case=case, ctx=bm4dof.Context(0), items=items)
    if case["kind"] == "tvl1":
        clean, _, _ = _video(case["W"], case["H"], case["F"], 1, seed)
        video = _noisy(clean, 2.0, seed).cpu().numpy()
        return dict(case=case, ctx=_context(False), video=video)
    feat, target, blob = _training_pairs(case["rows"], seed)
    trainer = bm4dof.Trainer(batch=case["rows"], seed=1)
    trainer.set_params(blob)
    return dict(case=case, trainer=trainer, feat=feat, target=target)


def _training_pairs(rows, seed):
    """Network inputs (64 log-variance ratios and sigma/255), gains in 0..1 that
    rise with them, and a parameter blob of the usual scale."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 31 + 5)
    lv = torch.randn(rows, 64, generator=g, device="cuda") * 1.5 + torch.linspace(3.0, -0.5, 64, device="cuda")
    sig = (5 + 45 * _rand(g, rows, 1)) / 255
    feat = torch.cat([lv, sig], 1).contiguous()
    target = torch.sigmoid(1.5 * lv - 1 + 0.3 * torch.randn(rows, 64, generator=g, device="cuda")).contiguous()
    rng = np.random.default_rng(int(seed) + 11)
    parts = [rng.standard_normal(s) * (math.sqrt(2.0 / s[0]) if len(s) == 2 else 0.01)
             for s in ((65, 256), (256,), (256, 256), (256,), (256, 64), (64,))]
    return feat, target, np.concatenate([p.ravel() for p in parts]).astype(np.float32)


LR, DECAY = 1e-3, 1e-4


def run(state):
    case = state["case"]
    if case["kind"] == "denoise":
        b, f, ratios = state["ctx"].runNlBayes(state["noisy"], state["ff"], state["bf"], *state["params"],
                                               basic=state["basic"], final=state["final"], nparts=case["nparts"],
                                               **_form(case))
        return dict(basic=b, final=f, ratios=list(ratios))
    if case["kind"] == "batch":
        ratios = state["ctx"].run_batched(state["items"], **_form(case))
        out = [it["basic"] for it in state["items"]] + [it["final"] for it in state["items"]]
        return dict(videos=out, ratios=torch.tensor(ratios, dtype=torch.float64))
    if case["kind"] == "tvl1":
        ff, bf = state["ctx"].tvl1_video(state["video"])
        return dict(fflow=ff, bflow=bf)
    loss = state["trainer"].step(state["feat"], state["target"], lr=LR, weight_decay=DECAY)
    return dict(loss=loss, params=state["trainer"].params())


# ---- what a pass cannot do without --------------------------------------------

def _groups(case, p):
    return sum(len(t["xs"]) * len(t["ys"]) * len(t["fs"]) for t in
               bm4dof.plan(case["W"], case["H"], case["F"], p, case["nparts"]))


def _denoise_work(case):
    n = case["W"] * case["H"] * case["F"]
    bytes_ = 4 * n * (3 * case["C"] + (4 if case["flow"] else 0))
    flops = 0.0
    p1, p2 = _params(case)
    steps = [(p2, 2)] if "learned" in case["form"] else [(p1, 1), (p2, 2)]
    for p, s in steps:
        spc = p.sizePatch ** 2 * p.sizePatchTime
        frames = min(case["F"] - p.sizePatchTime + 1, p.sizeSearchTimeRangeFwd + p.sizeSearchTimeRangeBwd + 1)
        cand = p.sizeSearchWindow ** 2 * frames
        if case["form"] == "vbm3d":
            # the first frame's window, then one window per predicted match (they overlap)
            cand = p.sizeSearchWindow ** 2 + p.sizeSearchWindowPred ** 2 * (frames - 1)
        chans = case["C"] if s == 2 and "learned" not in case["form"] else 1
        # a subtraction, a product and a sum per compared value; a product and a sum per transform term
        flops += _groups(case, p) * (3.0 * spc * chans * cand + 2.0 * p.nSimilarPatches * spc * spc * case["C"] * (s + 1))
    return dict(bytes=bytes_, flops=flops)


def work(case):
    if case["kind"] == "denoise":
        return _denoise_work(case)
    if case["kind"] == "batch":
        w = [_denoise_work(c) for c in _batch_cases(case, case["n"] * 31 + case["W"])]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    if case["kind"] == "tvl1":
        # video in, two flows out; per pair, level (4/3 in all, without the finest) and warping some
        # 20 iterations of about 60 operations per pixel
        n = case["W"] * case["H"]
        return dict(bytes=4 * n * case["F"] * 5, flops=2.0 * (case["F"] - 1) * n / 3 * 5 * 20 * 60)
    rows, weights = case["rows"], 65 * 256 + 256 * 256 + 256 * 64
    return dict(bytes=4 * (rows * (65 + 64) + 3 * 2 * bm4dof.GAIN_PARAMS), flops=6.0 * rows * weights)


# ---- the same results in 64 bits, from plain torch -----------------------------

def _dct(n):
    k, j = np.arange(n)[:, None], np.arange(n)[None]
    return np.cos((0.5 + j) * k * math.pi / n) * np.sqrt(np.where(k == 0, 1.0, 2.0) / n)


def _bior15():
    """Length-8 bior1.5 analysis [k, p] and synthesis [p, k] as BM3D has them."""
    s, h = 1 / math.sqrt(8), math.sqrt(0.5)
    a, b, c, d, e = 0.219417649252501, 0.449283757993216, 0.569359398342846, 0.402347308162278, 0.083506045090284
    f = 0.121533978016438
    A, S = np.zeros((8, 8)), np.zeros((8, 8))
    A[0] = s
    A[1] = [a, b, b, a, -a, -b, -b, -a]
    A[2] = [c, d, -d, -c, -e, e, -e, e]
    A[3] = [-e, e, -e, e, c, d, -d, -c]
    S[:, 0] = s
    S[:, 1] = [s] * 4 + [-s] * 4
    S[:4, 2] = S[4:, 3] = [0.5, 0.5, -0.5, -0.5]
    for i in range(4):
        A[4 + i, 2 * i], A[4 + i, 2 * i + 1] = h, -h
        for pair, v in ((i, (h, -h)), ((i + 1) % 4, (f, f)), ((i - 1) % 4, (-f, -f))):
            S[2 * pair:2 * pair + 2, 4 + i] = v
    return A, S


def _bases(p):
    """Analysis rows [k, p], synthesis [p, k] and aggregation window of a
    patch, elements ordered (t, y, x)."""
    px, pt = p.sizePatch, p.sizePatchTime
    if p.transform == bm4dof.BIOR1_5:
        a, i = _bior15()
        at = np.eye(pt)
    else:
        a, at = _dct(px), _dct(pt)
        i = a.T
    ana = np.einsum("ab,cd,ef->acebdf", at, a, a).reshape(px * px * pt, -1)
    syn = np.einsum("ab,cd,ef->acebdf", at.T, i, i).reshape(px * px * pt, -1)
    win = np.ones((pt, px, px))
    if p.agg_window and px == 8:
        # BM3D's four-digit Kaiser table
        rows = [[.1924, .2989, .3846, .4325], [.2989, .4642, .5974, .6717], [.3846, .5974, .7688, .8644],
                [.4325, .6717, .8644, .9718]]
        q = np.array(rows)
        q = np.concatenate([q, q[:, ::-1]], 1)
        win = np.broadcast_to(np.concatenate([q, q[::-1]], 0), (pt, px, px))
    t = lambda v: torch.tensor(np.ascontiguousarray(v), dtype=torch.float64, device="cuda")  # noqa: E731
    return t(ana), t(syn), t(win.reshape(-1))


def _opponent(v, inverse=False):
    if v.shape[1] != 3:
        return v
    a, b = 1 / math.sqrt(3), 1 / math.sqrt(2)
    c = 2 * a * math.sqrt(2)
    M = np.array([[a, a, a], [b, 0, -b], [c / 4, -c / 2, c / 4]])
    M = torch.tensor(np.linalg.inv(M) if inverse else M, dtype=torch.float64, device="cuda")
    return torch.einsum("dc,fchw->fdhw", M, v)


def _haar(z, inverse=False):
    """Orthonormal Haar along dim 1 in place order (z[n], z[n + h])."""
    n, levels = z.shape[1], []
    h = 1
    while h < n:
        levels.append(h)
        h *= 2
    for h in (reversed(levels) if inverse else levels):
        i = torch.arange(0, n, 2 * h, device=z.device)
        u, v = z[:, i] * math.sqrt(0.5), z[:, i + h] * math.sqrt(0.5)
        z = z.clone()
        z[:, i], z[:, i + h] = u + v, u - v
    return z


def _nearest(src, ff, bf, tile, ref, p, chans, mem):
    """The nearest patches of the reference positions ref [g, 3] (x, y, t) of a
    tile: positions [g, k, 3] and squared distances [g, k]."""
    ox, oy, w, h, F = tile
    px, pt, wx = p.sizePatch, p.sizePatchTime, p.sizeSearchWindow
    fwd, bwd = p.sizeSearchTimeRangeFwd, p.sizeSearchTimeRangeBwd
    dev = src.device
    crop = src[:, :chans, oy:oy + h, ox:ox + w].contiguous()
    flat = crop.reshape(-1)
    c, dt, dy, dx = torch.meshgrid(*(torch.arange(n, device=dev) for n in (chans, pt, px, px)), indexing="ij")
    offs = (((dt * chans + c) * h + dy) * w + dx).reshape(-1)
    K = min(p.nSimilarPatches, wx * wx * min(F - pt + 1, fwd + bwd + 1))
    ar = torch.arange(wx, device=dev)
    pos, dist = [], []
    nf = min(F - pt + 1, fwd + bwd + 1)
    per = max(1, int(mem / (8 * nf * wx * wx * offs.numel())))
    for at in range(0, ref.shape[0], per):
        r = ref[at:at + per]
        x, y, t = r.unbind(1)
        shift = (t - bwd).clamp(max=0) + (t + fwd - F + pt).clamp(min=0)
        t0 = (t - bwd - shift).clamp(min=0)
        q = t0[:, None] + torch.arange(nf, device=dev)[None]      # all groups have nf frames
        cx, cy = torch.zeros_like(q), torch.zeros_like(q)
        for sgn, fl in ((1, ff), (-1, bf)):
            ux, uy = x.clone(), y.clone()
            for d in range(0, fwd + bwd + 1):
                if d:
                    qt = (t + sgn * (d - 1)).clamp(0, F - 1)
                    if fl is not None:
                        f = fl[qt, :, oy + uy, ox + ux]
                        ux, uy = ux + f[:, 0], uy + f[:, 1]
                        ux, uy = (torch.sign(v) * torch.floor(v.abs() + 0.5) for v in (ux, uy))
                        ux, uy = ux.clamp(0, w - 1).long(), uy.clamp(0, h - 1).long()
                hit = q == (t + sgn * d)[:, None]
                cx, cy = torch.where(hit, ux[:, None], cx), torch.where(hit, uy[:, None], cy)
        hw = (wx - 1) // 2
        rng = []
        for ctr, n in ((cx, w), (cy, h)):
            s = (ctr - hw).clamp(max=0) + (ctr + hw - n + px).clamp(min=0)
            lo, hi = (ctr - hw - s).clamp(min=0), torch.minimum(ctr + hw - s, torch.full_like(ctr, n - px))
            rng.append((lo[..., None] + ar, lo[..., None] + ar <= hi[..., None]))
        (X, okx), (Y, oky) = rng
        X = X[:, :, None, :].expand(-1, -1, wx, -1).reshape(r.shape[0], -1)
        Y = Y[:, :, :, None].expand(-1, -1, -1, wx).reshape(r.shape[0], -1)
        ok = (okx[:, :, None, :] & oky[:, :, :, None]).reshape(r.shape[0], -1)
        T = q[:, :, None, None].expand(-1, -1, wx, wx).reshape(r.shape[0], -1)
        start = torch.where(ok, (T * chans * h + Y) * w + X, torch.zeros_like(T))
        mine = (t * chans * h + y) * w + x
        D = (flat[start[..., None] + offs] - flat[mine[:, None] + offs][:, None]).square_().sum(-1)
        d, i = torch.where(ok, D, torch.full_like(D, math.inf)).topk(K, 1, largest=False, sorted=True)
        pos.append(torch.stack([v.gather(1, i) for v in (X, Y, T)], -1))
        dist.append(d)
    return torch.cat(pos), torch.cat(dist)


def _step(noisy, basic, ff, bf, p, first, nparts):
    """One step over all tiles (noisy and basic colour transformed, 64 bits)."""
    F, C, H, W = noisy.shape
    px, pt = p.sizePatch, p.sizePatchTime
    spc = px * px * pt
    ana, syn, win = _bases(p)
    b = next(k for k in range(2, nparts + 1) if nparts % k == 0)
    a = nparts // b
    a, b = max(a, b), min(a, b)
    tw, th = math.ceil(W / a), math.ceil(H / b)
    out = torch.empty_like(noisy)
    tau2, sigma = p.tau ** 2 * spc, p.sigma
    ratio = 0.0
    dt, dy, dx = (v.reshape(-1) for v in torch.meshgrid(*(torch.arange(n, device="cuda") for n in (pt, px, px)),
                                                       indexing="ij"))
    for k, tile in enumerate(bm4dof.plan(W, H, F, p, nparts)):
        ox, oy, w, h = tile["box"]
        ref = torch.cartesian_prod(*(torch.tensor(tile[n], device="cuda") for n in ("fs", "ys", "xs"))).flip(1)
        pos, dist = _nearest(noisy if first else basic, ff, bf, (ox, oy, w, h, F), ref, p, 1 if first else C, 2e9)
        n = torch.ones(len(ref), dtype=torch.long, device="cuda")
        m = 1
        while 2 * m <= dist.shape[1]:
            n = torch.where((n == m) & (dist[:, m] < tau2), 2 * m, n)
            m *= 2
        # a group whose nearest patch is a later reference position switches that one off
        # (the switch-off's index counts channels, its mask does not: for colour it lands in another frame)
        own = (ref[:, 2] * h + ref[:, 1]) * w + ref[:, 0]
        hit = (pos[:, 0, 2] * C * h + pos[:, 0, 1]) * w + pos[:, 0, 0]
        where = torch.searchsorted(own, hit).clamp(max=len(own) - 1)
        edges = torch.nonzero((own[where] == hit) & (hit > own)).flatten()
        on = np.ones(len(ref), bool)
        for g, v in zip(edges.tolist(), where[edges].tolist()):
            if on[g]:
                on[v] = False
        alive = torch.tensor(on, device="cuda")
        ratio += 100.0 * int(alive.sum()) / (W * H * F)
        acc = torch.zeros(F * C * h * w, dtype=torch.float64, device="cuda")
        wacc = torch.zeros(F * h * w, dtype=torch.float64, device="cuda")
        src = noisy[:, :, oy:oy + h, ox:ox + w].contiguous().reshape(-1)
        pilot = None if first else basic[:, :, oy:oy + h, ox:ox + w].contiguous().reshape(-1)
        ch = torch.arange(C, device="cuda")
        for m in torch.unique(n).tolist():
            todo = torch.nonzero((n == m) & alive).flatten()
            for part in todo.split(max(1, int(2e8 / (m * C * spc)))):
                x, y, t = pos[part, :m].unbind(-1)
                at = ((((t[..., None, None] + dt) * C + ch[:, None]) * h + y[..., None, None] + dy) * w
                      + x[..., None, None] + dx)                       # [g, m, C, spc]
                z = _haar(src[at] @ ana.T)
                if first:
                    keep = z.square() > (p.beta * sigma) ** 2
                    keep[:, 0, :, 0] = True
                    z = z * keep
                    wt = 1 / sigma ** 2 / keep.sum((1, 2, 3))
                else:
                    u = _haar(pilot[at] @ ana.T).square()
                    u = u / (u + (p.beta * sigma) ** 2)
                    z = z * u
                    wt = 1 / sigma ** 2 / u.square().sum((1, 2, 3))
                est = _haar(z, True) @ syn.T
                wp = wt[:, None, None] * win
                acc.index_add_(0, at.reshape(-1), (wp[:, :, None] * est).reshape(-1))
                lin = ((t[..., None] + dt) * h + y[..., None] + dy) * w + x[..., None] + dx
                wacc.index_add_(0, lin.reshape(-1), wp.expand(-1, m, -1).reshape(-1))
        acc, wacc = acc.reshape(F, C, h, w), wacc.reshape(F, 1, h, w)
        den = torch.where(wacc > 0, wacc, noisy[:, :, oy:oy + h, ox:ox + w])
        X, Y = (k % a) * tw, (k // a) * th
        e, f = min(W, X + tw), min(H, Y + th)
        out[:, :, Y:f, X:e] = (acc / den)[:, :, Y - oy:f - oy, X - ox:e - ox]
    return out, ratio


def _exact_denoise(case, seed):
    clean, ff, bf = _video(case["W"], case["H"], case["F"], case["C"], seed)
    noisy = _opponent(_noisy(clean, case["sigma"], seed).double())
    ff, bf = (ff.double(), bf.double()) if case["flow"] else (None, None)
    p1, p2 = _params(case)
    basic, r1 = _step(noisy, None, ff, bf, p1, True, case["nparts"])
    final, r2 = _step(noisy, basic, ff, bf, p2, False, case["nparts"])
    return dict(basic=_opponent(basic, True), final=_opponent(final, True), ratios=[r1, r2])


def _gauss(img, sigma):
    size = int(5 * sigma) + 1
    g = np.exp(-np.arange(size) ** 2 / (2 * sigma * sigma))
    g /= 2 * g.sum() - g[0]
    for dim in (1, 2):
        n = img.shape[dim]
        i = torch.arange(n, device=img.device)
        out = g[0] * img
        for j in range(1, size):
            lo, hi = (i - j).abs(), i + j
            hi = torch.where(hi >= n, 2 * n - hi - 1, hi)
            out = out + g[j] * (img.index_select(dim, lo) + img.index_select(dim, hi))
        img = out
    return img


def _cubic(v, x):
    return v[1] + 0.5 * x * (v[2] - v[0] + x * (2 * v[0] - 5 * v[1] + 4 * v[2] - v[3] + x * (3 * (v[1] - v[2]) + v[3] - v[0])))


def _bicubic(img, X, Y, border):
    """img [n, h, w] at (X, Y); outside the image 0 where border, else clamped."""
    n, h, w = img.shape
    sx, sy = torch.where(X < 0, -1, 1), torch.where(Y < 0, -1, 1)
    ix, iy = X.trunc().long(), Y.trunc().long()
    xs, ys = [ix - sx, ix, ix + sx, ix + 2 * sx], [iy - sx, iy, iy + sy, iy + 2 * sy]
    out = torch.zeros_like(X, dtype=torch.bool)
    for v, m in [(v, w) for v in xs] + [(v, h) for v in ys]:
        out |= (v < 0) | (v >= m)
    xs, ys = [v.clamp(0, w - 1) for v in xs], [v.clamp(0, h - 1) for v in ys]
    k = torch.arange(n, device=img.device)[:, None, None].expand_as(ix)
    cols = [_cubic([img[k, b, a] for b in ys], Y - ys[1]) for a in xs]
    v = _cubic(cols, X - xs[1])
    return torch.where(out, torch.zeros_like(v), v) if border else v


def _grad(f):
    fx, fy = torch.zeros_like(f), torch.zeros_like(f)
    fx[:, :, :-1], fy[:, :-1] = f[:, :, 1:] - f[:, :, :-1], f[:, 1:] - f[:, :-1]
    return fx, fy


def _div(a, b):
    d = a.clone()
    d[:, :, -1] = 0
    d[:, :, 1:] -= a[:, :, :-1]
    e = b.clone()
    e[:, -1] = 0
    e[:, 1:] -= b[:, :-1]
    return d + e


def _exact_tvl1(case, seed):
    clean, _, _ = _video(case["W"], case["H"], case["F"], 1, seed)
    v = _noisy(clean, 2.0, seed)[:, 0].double()
    I0, I1 = torch.cat([v[:-1], v[1:]]), torch.cat([v[1:], v[:-1]])
    q = bm4dof.Context.tvl1_params()
    tau, lam, theta, zf, eps = q.tau, q.lambda_, q.theta, q.zfactor, q.epsilon
    H, W = v.shape[1:]
    scales = max(1, min(q.nscales, int(1 + math.log(math.hypot(W, H) / 16) / math.log(1 / zf))))
    lo = torch.minimum(I0.amin((1, 2)), I1.amin((1, 2)))[:, None, None]
    hi = torch.maximum(I0.amax((1, 2)), I1.amax((1, 2)))[:, None, None]
    P = [[_gauss(255 * (i - lo) / (hi - lo), 0.8) for i in (I0, I1)]]
    grid = lambda h, w, fx, fy: [t.double() for t in torch.meshgrid(torch.arange(h, device="cuda") / fy,  # noqa: E731
                                                                    torch.arange(w, device="cuda") / fx, indexing="ij")]
    for s in range(1, scales):
        h, w = (int(n * zf + 0.5) for n in P[-1][0].shape[1:])
        Y, X = grid(h, w, zf, zf)
        n = I0.shape[0]
        P.append([_bicubic(_gauss(i, 0.6 * math.sqrt(1 / zf ** 2 - 1)), X.expand(n, h, w), Y.expand(n, h, w), False)
                  for i in P[-1]])
    u = [torch.zeros_like(P[-1][0]) for _ in range(2)]
    for s in range(scales - 1, -1, -1):
        A, B = P[s]
        n, h, w = A.shape
        if u[0].shape != A.shape:
            fy, fx = h / u[0].shape[1], w / u[0].shape[2]
            Y, X = grid(h, w, fx, fy)
            u = [_bicubic(c, X.expand(n, h, w), Y.expand(n, h, w), False) / zf for c in u]
        if s < min(q.fscale, scales):
            continue
        pad = torch.nn.functional.pad(B[:, None], (1, 1, 1, 1), mode="replicate")[:, 0]
        Bx, By = (pad[:, 1:-1, 2:] - pad[:, 1:-1, :-2]) / 2, (pad[:, 2:, 1:-1] - pad[:, :-2, 1:-1]) / 2
        p = [torch.zeros_like(A) for _ in range(4)]
        yy, xx = torch.meshgrid(torch.arange(h, device="cuda"), torch.arange(w, device="cuda"), indexing="ij")
        for _ in range(q.warps):
            X, Y = xx + u[0], yy + u[1]
            w0, wx, wy = (_bicubic(i, X, Y, True) for i in (B, Bx, By))
            g = wx * wx + wy * wy
            rc = w0 - wx * u[0] - wy * u[1] - A
            live = torch.ones(n, dtype=torch.bool, device="cuda")
            for it in range(300):
                rho = rc + wx * u[0] + wy * u[1]
                f = torch.where(rho < -lam * theta * g, lam * theta, torch.where(
                    rho > lam * theta * g, -lam * theta, torch.where(g < 1e-10, 0.0, -rho / g.clamp(min=1e-10))))
                new = [u[0] + f * wx + theta * _div(p[0], p[1]), u[1] + f * wy + theta * _div(p[2], p[3])]
                err = ((new[0] - u[0]) ** 2 + (new[1] - u[1]) ** 2).mean((1, 2))
                on = live[:, None, None]
                u = [torch.where(on, a, b) for a, b in zip(new, u)]
                for c in range(2):
                    gx, gy = _grad(u[c])
                    ng = 1 + tau / theta * torch.hypot(gx, gy)
                    p[2 * c] = torch.where(on, (p[2 * c] + tau / theta * gx) / ng, p[2 * c])
                    p[2 * c + 1] = torch.where(on, (p[2 * c + 1] + tau / theta * gy) / ng, p[2 * c + 1])
                live = live & (err > eps * eps)
                if it % 8 == 7 and not bool(live.any()):
                    break
    uv = torch.stack(u, 1)
    m = case["F"] - 1
    return dict(fflow=torch.cat([uv[:m], uv[m - 1:m]]), bflow=torch.cat([uv[m:m + 1], uv[m:]]))


def _exact_train(case, seed):
    feat, target, blob = _training_pairs(case["rows"], seed)
    ps = [torch.tensor(a, dtype=torch.float64, device="cuda", requires_grad=True) for a in bm4dof.split_params(blob)]
    h = torch.nn.functional.gelu(feat.double() @ ps[0] + ps[1])
    h = torch.nn.functional.gelu(h @ ps[2] + ps[3])
    loss = (torch.sigmoid(h @ ps[4] + ps[5]) - target.double()).square().mean()
    loss.backward()
    new = []
    for p in ps:   # the first AdamW step: both moments are the gradient's own
        decay = LR * DECAY * p if p.dim() == 2 else 0.0
        new.append((p - LR * p.grad / (p.grad.abs() + 1e-8) - decay).detach().reshape(-1))
    return dict(loss=float(loss.detach()), params=torch.cat(new))


def exact(case, seed):
    if case["kind"] == "tvl1":
        return _exact_tvl1(case, seed)
    if case["kind"] == "train":
        return _exact_train(case, seed)
    # The learned and predictive forms and the batch are made of the same
    # steps; in 64 bits a large clip takes minutes.
    if case["kind"] == "denoise" and case["form"] in ("plain", "mixed") and _denoise_work(case)["flops"] < 2.75e12:
        return _exact_denoise(case, seed)
    return None
