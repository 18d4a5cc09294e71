"""Inputs on which blocks of patches do not pay: the search leaves them to the
per-group kernel, with the same outputs and little more time than that kernel
takes by itself.  (A pixel of 2e17 sends the whole source to it.)"""
import numpy as np
import pytest

from helpers import resolve_params

pytestmark = pytest.mark.gpu

P4 = dict(px1=4, px2=4, pt1=4, pt2=4, wx1=21, wx2=21, np1=16, np2=16, b1=3.0)


def compare(gpulib, gpuctx, nz, ff, bf, cli, sigma):
    """Search times, best of five runs of step 1: blocks, per-group kernel.  The
    outputs must be those of search_strip 7, which has no blocks."""
    import torch
    F, C, H, W = nz.shape
    dev = lambda a: None if a is None else torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()
    p1, p2 = resolve_params(gpulib, (W, H, F, C), sigma, **cli)
    p2.sizePatch = 0
    n, f, b = dev(nz), dev(ff), dev(bf)
    far = n.clone()
    far[F // 2, 0, H // 2, W // 2] = 2e17
    ms = []
    for src in (n, far):
        t = []
        for _ in range(6):
            out = gpuctx.runNlBayes(src, f, b, p1, p2, nparts=2)[0]
            t.append(gpuctx.timings()[0][0])
        ms.append(min(t[1:]))
        if src is n:
            got = out.clone()
    item = dict(noisy=n, fflow=f, bflow=b, basic=torch.empty_like(n), final=torch.empty_like(n), p1=p1, p2=p2)
    gpuctx.run_batched([item], tuning=dict(search_strip=7))
    assert torch.equal(got, item["basic"])
    return ms


# before the rule: 1.5 to 3.3 times the per-group kernel's time; with it a left
# block costs the look at its windows, a tenth of 7x7 windows' search
@pytest.mark.parametrize("noise,cli", [(8.0, P4), (20.0, P4), (20.0, {})], ids=["4x4x4", "rough", "defaults"])
def test_gpu_blocks_under_rough_flows(gpulib, gpuctx, noise, cli):
    W, H, F = 480, 272, 10
    rng = np.random.default_rng(17)
    y, x = np.mgrid[:H, :W]
    nz = 128 + 60 * np.sin(0.05 * x + 0.03 * y) * np.ones((F, 1, 1, 1)) + rng.normal(0, 20, (F, 1, H, W))
    ff, bf = rng.normal(0, noise, (2, F, 2, H, W))
    blocks, groups = compare(gpulib, gpuctx, nz, ff, bf, cli, 20.0)
    assert blocks <= 1.2 * groups, (blocks, groups)


# exact ties in every group: before the rule 1.4 times the per-group kernel's
# time; with it the look at the block's pixels more
def test_gpu_blocks_on_flat_frames(gpulib, gpuctx):
    nz = np.full((12, 1, 360, 640), 100.0, np.float32)
    blocks, groups = compare(gpulib, gpuctx, nz, None, None, P4, 20.0)
    assert blocks <= 1.2 * groups, (blocks, groups)


# half the frame flat: blocks are computed again where they pay
def test_gpu_blocks_on_half_flat_frames(gpulib, gpuctx):
    rng = np.random.default_rng(3)
    nz = np.full((12, 1, 360, 640), 100.0, np.float32)
    nz[..., 320:] += rng.normal(0, 20, (12, 1, 360, 320)).astype(np.float32)
    blocks, groups = compare(gpulib, gpuctx, nz, None, None, P4, 20.0)
    assert blocks <= 1.2 * groups, (blocks, groups)
