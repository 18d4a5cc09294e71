"""The ordered aggregation of 2x2 patches (aggregate.cu, bin_gather_kernel by
columns): bit for bit against the oracle for every number of patch frames and
channels at sizes around whole bins, and its time beside the filter's."""
import numpy as np
import pytest

from helpers import resolve_params, video_case

pytestmark = pytest.mark.gpu


def params(lib, size, pt, **k):
    return resolve_params(lib, size, 20.0, px1=2, px2=2, pt1=pt, pt2=pt, **dict(dict(wx1=9, wx2=9, np1=16, np2=16, b1=3.0), **k))


@pytest.mark.parametrize("W,H,F,C,pt", [(31, 33, 1, 1, 1), (33, 17, 5, 1, 2), (32, 32, 4, 1, 4), (17, 31, 6, 3, 3), (16, 33, 18, 1, 16),
                                        (33, 16, 5, 4, 4), (15, 47, 2, 3, 1)])
def test_gpu_2x2_patches(gpulib, gpuctx, oracle, W, H, F, C, pt):
    _, nz, ff, bf = video_case(W, H, F, sigma=20.0, seed=W * 64 + H, channels=C)
    po, pg = params(oracle, (W, H, F, C), pt), params(gpulib, (W, H, F, C), pt)
    ob, of, orat = oracle.runNlBayes(nz, ff, bf, *po, nparts=2)[:3]
    gb, gf, grat = gpuctx.runNlBayes(nz, ff, bf, *pg, nparts=2)
    assert np.array_equal(gb, ob, equal_nan=True) and np.array_equal(gf, of, equal_nan=True) and grat == orat


def test_gpu_2x2_patches_time(gpulib, gpuctx):
    # the aggregation took 1.4 times the filter's time with merges of per-pixel
    # lists, 2.5 times with two pixels to a lane
    W, H, F = 240, 180, 8
    _, nz, ff, bf = video_case(W, H, F, sigma=20.0, seed=5)
    p1, p2 = params(gpulib, (W, H, F, 1), 4, wx1=15, wx2=15)
    ms = []
    for _ in range(4):
        gpuctx.runNlBayes(nz, ff, bf, p1, p2, nparts=2)
        ms.append(gpuctx.timings()[0][1:3])
    filt, agg = min(m[0] for m in ms), min(m[1] for m in ms)
    assert agg < 1.6 * filt, (agg, filt)
