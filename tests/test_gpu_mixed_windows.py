"""Tensor-core pre-screen: windows from 3x3 to 31x31 on clips down to a few
patches across, where a run of 32 candidates covers many rows of the union or
part of one, most candidates or few pass the threshold, and the lists fill at
once or never.  Certified lists are the exact search's."""
import numpy as np
import pytest

from helpers import resolve_params, video_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,F,px,pt,wx,k", [
    (7, 6, 4, 4, 4, 3, 2), (9, 40, 5, 4, 4, 5, 4), (40, 9, 5, 4, 4, 21, 16), (20, 20, 6, 4, 4, 31, 16),
    (50, 34, 7, 4, 4, 9, 16), (64, 48, 6, 4, 4, 31, 32), (90, 60, 1, 8, 1, 39, 16), (19, 70, 1, 8, 1, 15, 8)])
@pytest.mark.parametrize("flat", [False, True])
def test_windows_certified(gpulib, gpuctx, W, H, F, px, pt, wx, k, flat):
    clean, nz, ff, bf = video_case(W, H, F, sigma=20.0, seed=W + H)
    if flat:   # hardly any noise on the left: nearly equal candidates
        nz[:, :, :, :W // 2] = clean[:, :, :, :W // 2] + 1e-3 * (nz - clean)[:, :, :, :W // 2]
    p = resolve_params(gpulib, (W, H, F, 1), 20.0, px1=px, px2=px, pt1=pt, pt2=pt, wx1=wx, wx2=wx, np1=k, np2=k, b1=3.0)
    got = []
    for mixed in (False, "certified"):
        out = gpuctx.runNlBayes(nz, ff, bf, *p, nparts=1, keep_groups=True, mixed=mixed)
        got.append((out[0], out[1], [gpuctx.groups(s, 0) for s in (1, 2)]))
    for a, b in zip(got[0][2], got[1][2]):
        for key in ("ref", "nsimp", "index"):
            assert np.array_equal(a[key], b[key]), key
    assert np.array_equal(got[0][0], got[1][0], equal_nan=True) and np.array_equal(got[0][1], got[1][1], equal_nan=True)
