"""TV-L1 flow against a restatement in separately rounded float and double tensor
operations: one tile and many, every tile height, pairs in several launches,
and a level that does not fit on the chip.  The kernels claim the same bits."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
f32 = np.float32


def gauss(img, sigma):
    import torch
    sigma = float(sigma)
    size = int(5 * sigma) + 1
    den = 2 * sigma * sigma
    B = [1 / (sigma * math.sqrt(2.0 * 3.1415926)) * math.exp(-i * i / den) for i in range(size)]
    norm = 0.0
    for b in B:
        norm += b
    norm = norm * 2 - B[0]
    B = [b / norm for b in B]
    for dim in (2, 1):
        n = img.shape[dim]
        pos = torch.arange(n, device=img.device)
        d = img.double()
        acc = B[0] * d
        for j in range(1, size):
            lo, hi = (pos - j).abs(), pos + j
            hi = torch.where(hi >= n, 2 * n - hi - 1, hi)
            acc = acc + B[j] * (d.index_select(dim, lo) + d.index_select(dim, hi))
        img = acc.float()
    return img


def cell(v, x):
    return v[1] + 0.5 * x * (v[2] - v[0] + x * (2.0 * v[0] - 5.0 * v[1] + 4.0 * v[2] - v[3] +
                                                x * (3.0 * (v[1] - v[2]) + v[3] - v[0])))


def bicubic(img, U, V, border_out):
    import torch
    n, h, w = img.shape
    sx = torch.where(U < 0, -1, 1)
    sy = torch.where(V < 0, -1, 1)
    ui, vi = U.trunc().long(), V.trunc().long()
    X = [ui - sx, ui, ui + sx, ui + 2 * sx]
    Y = [vi - sx, vi, vi + sy, vi + 2 * sy]
    out = torch.zeros_like(U, dtype=torch.bool)
    for q, lim in [(q, w) for q in X] + [(q, h) for q in Y]:
        out |= (q < 0) | (q >= lim)
    X, Y = [q.clamp(0, w - 1) for q in X], [q.clamp(0, h - 1) for q in Y]
    fx, fy = (U - X[1].float()).double(), (V - Y[1].float()).double()
    flat = img.reshape(n, -1).double()
    at = lambda a, b: flat.gather(1, (X[a] + w * Y[b]).reshape(n, -1)).reshape(U.shape)  # noqa: E731
    r = cell([cell([at(a, b) for b in range(4)], fy) for a in range(4)], fx).float()
    return torch.where(out, torch.zeros_like(r), r) if border_out else r


def zoom(img, h, w, fx, fy):
    import torch
    # divided by a tensor: by a Python number it would be a product with the reciprocal
    q = [torch.arange(k, device=img.device).float() / torch.full((k,), float(f), device=img.device)
         for k, f in ((h, fy), (w, fx))]
    y, x = torch.meshgrid(*q, indexing="ij")
    n = img.shape[0]
    return bicubic(img, x.expand(n, h, w), y.expand(n, h, w), False)


def divergence(a, b):
    import torch
    pa, pb = torch.zeros_like(a), torch.zeros_like(b)
    pa[:, :, 1:] = a[:, :, :-1]
    pb[:, 1:] = b[:, :-1]
    a, b = a.clone(), b.clone()
    a[:, :, -1] = 0
    b[:, -1] = 0
    r = (a - pa) + (b - pb)
    for c in (0, -1):
        r[:, :, c] = ((a - pa)[:, :, c] + b[:, :, c]) - pb[:, :, c]
    return r


def gradient(u):
    import torch
    gx, gy = torch.zeros_like(u), torch.zeros_like(u)
    gx[:, :, :-1] = u[:, :, 1:] - u[:, :, :-1]
    gy[:, :-1] = u[:, 1:] - u[:, :-1]
    return gx, gy


def flow(I0, I1, scales, fscale, warps, eps, tau=0.25, lam=0.2, theta=0.3, zf=0.5):
    import torch
    tau, lam, theta, zf = f32(tau), f32(lam), f32(theta), f32(zf)
    l_t, taut, eps2 = float(lam * theta), float(tau / theta), float(f32(eps) * f32(eps))
    theta_f = float(theta)
    hi = torch.maximum(I0.amax((1, 2)), I1.amax((1, 2)))[:, None, None]
    lo = torch.minimum(I0.amin((1, 2)), I1.amin((1, 2)))[:, None, None]
    den = hi - lo
    P = []
    for I in (I0, I1):
        s = (255.0 * (I - lo).double() / den.double()).float()
        P.append(gauss(torch.where(den > 0, s, I), 0.8))
    P = [P]
    zs = f32(float(f32(0.6)) * math.sqrt(1.0 / float(zf * zf) - 1.0))
    for s in range(1, scales):
        h, w = (int(f32(f32(k) * zf) + f32(0.5)) for k in P[-1][0].shape[1:])
        P.append([zoom(gauss(i, zs), h, w, zf, zf) for i in P[-1]])
    u = [torch.zeros_like(P[-1][0]) for _ in range(2)]
    for s in range(scales - 1, -1, -1):
        A, B = P[s]
        n, h, w = A.shape
        if u[0].shape != A.shape:
            fx, fy = f32(w) / f32(u[0].shape[2]), f32(h) / f32(u[0].shape[1])
            u = [zoom(c, h, w, fx, fy) * float(f32(1.0) / zf) for c in u]
        if s < fscale:
            continue
        pad = torch.nn.functional.pad(B[:, None], (1, 1, 1, 1), mode="replicate")[:, 0]
        Bx, By = 0.5 * (pad[:, 1:-1, 2:] - pad[:, 1:-1, :-2]), 0.5 * (pad[:, 2:, 1:-1] - pad[:, :-2, 1:-1])
        p = [torch.zeros_like(A) for _ in range(4)]
        yy, xx = (q.float() for q in torch.meshgrid(torch.arange(h, device=A.device), torch.arange(w, device=A.device),
                                                    indexing="ij"))
        for _ in range(warps):
            X, Y = xx + u[0], yy + u[1]
            w0, wx, wy = (bicubic(i, X, Y, True) for i in (B, Bx, By))
            g = wx * wx + wy * wy
            rc = w0 - wx * u[0] - wy * u[1] - A
            live = torch.ones(n, dtype=torch.bool, device=A.device)
            for it in range(300):
                rho = rc + (wx * u[0] + wy * u[1])
                fi = -rho / g
                d = []
                for c in (wx, wy):
                    t = torch.where(g < float(f32(1e-10)), torch.zeros_like(g), fi * c)
                    t = torch.where(rho > l_t * g, -l_t * c, t)
                    d.append(torch.where(rho < -l_t * g, l_t * c, t))
                new = [(u[k] + d[k]) + theta_f * divergence(p[2 * k], p[2 * k + 1]) for k in range(2)]
                err = ((new[0] - u[0]).double() ** 2 + (new[1] - u[1]).double() ** 2).mean((1, 2))
                on = live[:, None, None]
                u = [torch.where(on, a, b) for a, b in zip(new, u)]
                for k in range(2):
                    gx, gy = gradient(u[k])
                    ng = 1.0 + taut * torch.sqrt(gx * gx + gy * gy)
                    p[2 * k] = torch.where(on, (p[2 * k] + taut * gx) / ng, p[2 * k])
                    p[2 * k + 1] = torch.where(on, (p[2 * k + 1] + taut * gy) / ng, p[2 * k + 1])
                live = live & (err > eps2)
                if it % 16 == 15 and not bool(live.any()):
                    break
    return torch.stack(u, 1)


def images(n, H, W, seed):
    import torch
    g = torch.Generator().manual_seed(seed)
    big = torch.rand(n, 1, H // 3 + 4, W // 3 + 4, generator=g)
    big = torch.nn.functional.interpolate(big, size=(H + 3, W + 3), mode="bicubic", align_corners=False)[:, 0] * 200
    noise = torch.randn(2, n, H, W, generator=g) * 2
    return (big[:, :H, :W] + noise[0]).contiguous(), (big[:, 1:H + 1, 2:W + 2] + noise[1]).contiguous()


@pytest.mark.parametrize("W,H,n,scales,fscale,warps", [
    (17, 9, 1, 1, 0, 2),        # less than one tile
    (32, 8, 2, 1, 0, 2),        # exactly one tile
    (33, 9, 2, 1, 0, 2),        # one pixel more
    (97, 61, 3, 2, 0, 2),
    (75, 90, 2, 3, 1, 3),       # the finest level only passed up to
    (150, 130, 10, 1, 0, 2),    # tiles of 16 rows
    (150, 130, 20, 1, 0, 2),    # of 32
    (150, 130, 45, 1, 0, 2),    # of 64
    (150, 130, 70, 1, 0, 2),    # two launches
    (1440, 900, 1, 1, 0, 1),    # run from L2
    (1440, 900, 2, 2, 0, 1),    # the fine level from L2, the coarse one on the chip
])
def test_levels_match_restatement(gpulib, gpuctx, W, H, n, scales, fscale, warps):
    import torch
    I0, I1 = images(n, H, W, W * H + n)
    p = gpuctx.tvl1_params(nscales=scales, fscale=fscale, warps=warps, epsilon=1e-6)
    want = flow(I0.cuda(), I1.cuda(), scales, fscale, warps, 1e-6)
    got = torch.from_numpy(np.ascontiguousarray(gpuctx.tvl1_pairs(I0.numpy(), I1.numpy(), p))).cuda()
    assert torch.equal(got.reshape(want.shape), want)


@pytest.mark.parametrize("value", [0.0, -3.5, 77.0])
def test_constant_images(gpulib, gpuctx, value):
    import torch
    I = torch.full((1, 40, 50), value)
    p = gpuctx.tvl1_params(nscales=2, fscale=0, warps=2, epsilon=1e-6)
    want = flow(I.cuda(), I.cuda(), 2, 0, 2, 1e-6).cpu().numpy()
    assert np.array_equal(gpuctx.tvl1_pairs(I.numpy(), I.numpy(), p).reshape(want.shape), want)
