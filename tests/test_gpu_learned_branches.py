"""Learned form's tensor-core kernels on the branches that plain runs take: the
residual fallback, the hard threshold of the non-mean rows, and the network's
gains, each against a float64 restatement on the same groups."""
import numpy as np
import pytest

import gain_mlp as gm
from helpers import resolve_params, video_case
from test_gpu_learned_groups import haar, unhaar

pytestmark = pytest.mark.gpu

W, H, F, SIGMA = 45, 38, 6, 20.0


def gains_of(z, bs2):
    """Wiener gains of a pilot (0 where it was cut)."""
    return z * z / (z * z + bs2)


@pytest.fixture
def network(gpulib, gpuctx):
    """set_gain_network for one test; the session's context goes back to none."""
    yield gpuctx.set_gain_network
    gpuctx.set_gain_network(None)


def run(gpulib, gpuctx, px, pt, np_, tau, b1):
    import torch
    _, nz, ff, bf = video_case(W, H, F, sigma=SIGMA, seed=31)
    p1, p2 = resolve_params(gpulib, (W, H, F, 1), SIGMA, px1=px, px2=px, pt1=pt, pt2=pt, wx1=9, wx2=9, np1=np_, np2=np_, b1=b1)
    for p in (p1, p2):
        p.agg_window = 0
        p.tau = tau
    d = [torch.from_numpy(a).cuda() for a in (nz, ff, bf)]
    out = gpuctx.runNlBayes(*d, p1, p2, nparts=1, keep_groups=True, learned=True)[1].cpu().numpy()[:, 0]
    return nz, p2, gpuctx.groups(2, 0), gpuctx.learned_stats(), out


def restate(oracle, nz, grp, px, pt, shrink):
    """The filtered video in float64; shrink(G, Z, z) gives the gains of a group (its
    pixels, its coefficients, their Haar transform) and, per coefficient, how
    far a gain may be off because a threshold lies within the coefficients' rounding.
    Also returns, per pixel, what those can move."""
    B = oracle.basis(0, px, pt)[0].astype(np.float64).reshape(64, 64)
    acc, wacc, slack = np.zeros((F, H, W)), np.zeros((F, H, W)), np.zeros((F, H, W))
    for n, idx in zip(grp["nsimp"], grp["index"]):
        at = [np.unravel_index(int(q), (F, H, W)) for q in idx[:n]]
        G = np.array([nz[t:t + pt, 0, y:y + px, x:x + px].ravel() for t, y, x in at], np.float64)
        Z = G @ B.T
        z = haar(Z)
        w, doubt = shrink(G, Z, z)
        E = unhaar(z * w) @ B
        D = np.zeros_like(E)
        for m, k in zip(*np.nonzero(doubt)):
            one = np.zeros_like(z)
            one[m, k] = abs(z[m, k]) * doubt[m, k]
            D += np.abs(unhaar(one) @ B)
        wgt = 1 / (SIGMA ** 2 * max((w * w).sum(), 1e-3))
        for (t, y, x), e, d in zip(at, E, D):
            acc[t:t + pt, y:y + px, x:x + px] += wgt * e.reshape(pt, px, px)
            wacc[t:t + pt, y:y + px, x:x + px] += wgt
            slack[t:t + pt, y:y + px, x:x + px] += wgt * d.reshape(pt, px, px)
    some = wacc > 0
    return np.where(some, acc / np.where(some, wacc, 1), nz[:, 0]), np.where(some, slack / np.where(some, wacc, 1), 0)


SHAPES = [(4, 4, 16, 400.), (4, 4, 16, 42.), (4, 4, 4, 400.), (8, 1, 16, 400.)]


@pytest.mark.parametrize("px,pt,np_,tau", SHAPES)
def test_every_group_falls_back(gpulib, gpuctx, oracle, network, px, pt, np_, tau):
    network(None, kappa=1e-12)
    nz, p2, grp, (groups, fallbacks), out = run(gpulib, gpuctx, px, pt, np_, tau, 0.0)
    assert groups > 0 and fallbacks == groups
    bs2 = (float(p2.beta) * SIGMA) ** 2
    want, _ = restate(oracle, nz, grp, px, pt, lambda G, Z, z: (gains_of(z, bs2), np.zeros_like(z)))
    diff = np.abs(out - want)
    # pixels and coefficients are rounded to BF16 (2^-9 of up to 2^8, half a grey level
    # each way, a quarter on average): their transforms keep the norm
    assert diff.max() < 3.0 and diff.mean() < 0.5, (diff.max(), diff.mean())


@pytest.mark.parametrize("px,pt,np_,tau", SHAPES)
def test_threshold_of_the_other_rows(gpulib, gpuctx, oracle, network, px, pt, np_, tau):
    network(None, kappa=1e30)
    nz, p2, grp, (_, fallbacks), out = run(gpulib, gpuctx, px, pt, np_, tau, 3.0)
    assert fallbacks == 0
    bs2, cut = (float(p2.beta) * SIGMA) ** 2, 3.0 * SIGMA

    def shrink(G, Z, z):
        w = gains_of(np.where(np.abs(z) > cut, z, 0), bs2)
        w[0] = np.where(z[0] ** 2 > bs2, (z[0] ** 2 - bs2) / np.maximum(z[0] ** 2, 1e-30), 0)
        # a coefficient's rounding: 64 pixels and basis values of 2^-9 relative, norm 1
        doubt = np.where(np.abs(np.abs(z) - cut) < 2.5, cut ** 2 / (cut ** 2 + bs2), 0)
        doubt[0] = 0
        return w, doubt
    want, slack = restate(oracle, nz, grp, px, pt, shrink)
    diff = np.abs(out - want)
    # (a gain that goes the other way also moves its group's weight: one level more)
    assert np.all(diff < 4.0 + slack) and diff.mean() < 0.6, ((diff - slack).max(), diff.mean())


@pytest.mark.parametrize("px,pt,np_,tau", SHAPES)
def test_network_gains(gpulib, gpuctx, oracle, network, px, pt, np_, tau):
    tr = gpulib.Trainer(batch=64, seed=5)
    params = tr.params()
    network(params, kappa=1e30)
    nz, p2, grp, (_, fallbacks), out = run(gpulib, gpuctx, px, pt, np_, tau, 0.0)
    assert fallbacks == 0
    bs2 = (float(p2.beta) * SIGMA) ** 2
    rounded = gm.join([gm.bf16_round(p) if p.ndim == 2 else p for p in gm.split(params)])

    def shrink(G, Z, z):
        w = gains_of(z, bs2)
        f = np.empty((1, 65), np.float32)
        f[0, :64] = np.log(np.maximum((Z * Z).mean(0), 1e-6 * SIGMA ** 2) / SIGMA ** 2)
        f[0, 64] = SIGMA / 255.0
        w[0] = gm.forward(rounded, gm.bf16_round(f))[0][0]
        return w, np.zeros_like(z)
    want, _ = restate(oracle, nz, grp, px, pt, shrink)
    diff = np.abs(out - want)
    # a gain is within 1e-2 (hidden activations are BF16), 1.5e-3 on average; on a mean
    # of up to 255 that is 2.5 levels, 0.4 on average, beside the rounding above
    assert diff.max() < 5.5 and diff.mean() < 0.9, (diff.max(), diff.mean())
