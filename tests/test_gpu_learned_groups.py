"""Learned form's tensor-core kernels: every number of members of a group (1 to
16), both 64-element patch shapes, against a float64 restatement on the same
groups; and the network's forward kernel at the edges of its 64-row tiles."""
import numpy as np
import pytest

import gain_mlp as gm
from helpers import resolve_params, video_case

pytestmark = pytest.mark.gpu


def haar(z):
    n, h = z.shape[0], 1
    z = z.copy()
    while h < n:
        a, b = z[::2 * h].copy(), z[h::2 * h].copy()
        z[::2 * h], z[h::2 * h] = (a + b) / np.sqrt(2), (a - b) / np.sqrt(2)
        h *= 2
    return z


def unhaar(z):
    h = z.shape[0] // 2
    z = z.copy()
    while h >= 1:
        a, b = z[::2 * h].copy(), z[h::2 * h].copy()
        z[::2 * h], z[h::2 * h] = (a + b) / np.sqrt(2), (a - b) / np.sqrt(2)
        h //= 2
    return z


@pytest.mark.parametrize("px,pt,np_,tau", [(4, 4, 16, 400.), (4, 4, 16, 42.), (4, 4, 8, 400.), (4, 4, 4, 400.),
                                           (4, 4, 2, 400.), (8, 1, 16, 400.), (8, 1, 16, 42.)])
def test_apply_matches_restatement(gpulib, gpuctx, oracle, px, pt, np_, tau):
    import torch
    W, H, F, sigma = 45, 38, 6, 20.0
    clean, nz, ff, bf = video_case(W, H, F, sigma=sigma, seed=31)
    # no threshold (b1 = 0): the shrinkage is smooth, so rounding moves no coefficient across it
    p1, p2 = resolve_params(gpulib, (W, H, F, 1), sigma, px1=px, px2=px, pt1=pt, pt2=pt, wx1=9, wx2=9, np1=np_, np2=np_,
                            b1=0.0)
    for p in (p1, p2):
        p.agg_window = 0
        p.tau = tau
    d = [torch.from_numpy(a).cuda() for a in (nz, ff, bf)]
    gpuctx.set_gain_network(None, kappa=1e30)
    _, out, _ = gpuctx.runNlBayes(*d, p1, p2, nparts=1, keep_groups=True, learned=True)
    grp = gpuctx.groups(2, 0)
    assert len(grp["ref"]) > 0
    B = oracle.basis(0, px, pt)[0].astype(np.float64).reshape(64, 64)
    bs2 = (float(p2.beta) * sigma) ** 2
    acc, wacc = np.zeros((F, H, W)), np.zeros((F, H, W))
    for n, idx in zip(grp["nsimp"], grp["index"]):
        at = [np.unravel_index(int(q), (F, H, W)) for q in idx[:n]]
        G = np.array([nz[t:t + pt, 0, y:y + px, x:x + px].ravel() for t, y, x in at], np.float64)
        z = haar(G @ B.T)
        w = z * z / (z * z + bs2)
        w[0] = np.where(z[0] ** 2 > bs2, (z[0] ** 2 - bs2) / np.maximum(z[0] ** 2, 1e-30), 0)
        E = unhaar(z * w) @ B
        wgt = 1 / (sigma ** 2 * max((w * w).sum(), 1e-3))
        for (t, y, x), e in zip(at, E):
            acc[t:t + pt, y:y + px, x:x + px] += wgt * e.reshape(pt, px, px)
            wacc[t:t + pt, y:y + px, x:x + px] += wgt
    want = np.where(wacc > 0, acc / np.where(wacc > 0, wacc, 1), nz[:, 0])
    diff = np.abs(out.cpu().numpy()[:, 0] - want)
    # pixels and coefficients are rounded to BF16 (2^-9 of up to 2^8, half a grey level
    # each way, a quarter on average): their transforms keep the norm
    assert diff.max() < 3.0 and diff.mean() < 0.5, (diff.max(), diff.mean())


@pytest.mark.parametrize("n", [1, 63, 64, 65, 20000])
def test_forward_rows(gpulib, gpuctx, n):
    import torch
    rng = np.random.default_rng(n)
    tr = gpulib.Trainer(batch=n, seed=3)
    X = np.empty((n, 65), np.float32)
    X[:, :64] = rng.normal(1.0, 2.0, (n, 64))
    X[:, 64] = rng.uniform(5, 50, n) / 255.0
    got = tr.predict(torch.from_numpy(X).cuda()).cpu().numpy()
    parts = [gm.bf16_round(p) if p.ndim == 2 else p for p in gm.split(tr.params())]
    want, _ = gm.forward(gm.join(parts), gm.bf16_round(X))
    assert np.abs(got - want).max() < 1e-2   # hidden activations are BF16
