"""Predictive search: windows of frame pt up to and past the size that a warp
takes in pairs of candidates (128), every patch shape with a kernel of its
own, distances summed once (grey) and three times (colour, step 2): neighbour
lists and outputs are the oracle's, bit for bit."""
import numpy as np
import pytest

from helpers import resolve_params, video_case
from test_gpu_vbm3d import same_groups

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [1, 3])
@pytest.mark.parametrize("px,pt,wx", [(7, 1, 3), (7, 1, 7), (7, 1, 13), (8, 1, 7), (8, 1, 11), (8, 1, 13), (4, 4, 5),
                                      (4, 4, 11), (4, 4, 13), (5, 2, 7)])
def test_windows_match_oracle(gpulib, gpuctx, oracle, C, px, pt, wx):
    W, H, F = 39, 33, 6
    clean, nz, ff, bf = video_case(W, H, F, sigma=20.0, seed=400 + wx, channels=C)
    cfg = dict(px1=px, px2=px, pt1=pt, pt2=pt, wx1=wx, wx2=wx, np1=8, np2=8, npf1=2, npf2=2, wxf1=3, wxf2=5)
    po = resolve_params(oracle, (W, H, F, C), 20.0, **cfg)
    pg = resolve_params(gpulib, (W, H, F, C), 20.0, **cfg)
    ob, of, orat, tr = oracle.runNlBayes(nz, ff, bf, *po, nparts=2, trace_cap=100000, trace_stride=32, vbm3d=True)
    gb, gf, grat = gpuctx.runNlBayes(nz, ff, bf, *pg, nparts=2, keep_groups=True, vbm3d=True)
    same_groups(gpuctx, tr, 2)
    assert np.array_equal(gb, ob) and np.array_equal(gf, of) and grat == orat


@pytest.mark.parametrize("npf,F,flow", [(1, 6, True), (2, 4, True), (2, 9, False), (3, 6, True), (4, 7, True), (8, 9, True)])
def test_first_frame_by_blocks(gpulib, gpuctx, oracle, npf, F, flow):
    # frame pt's 15x15 window: the block search for 2, 4 and 8 matches a frame,
    # the kernel's own for 1 and 3; one frame only, and flat areas whose ties the
    # block search leaves open
    W, H = 43, 37
    clean, nz, ff, bf = video_case(W, H, F, sigma=15.0, seed=500 + npf)
    nz[:, :, :, :20] = np.round(clean[:, :, :, :20] / 16) * 16
    if not flow:
        ff = bf = None
    cfg = dict(px1=4, px2=8, pt1=4, pt2=1, wx1=15, wx2=15, np1=16, np2=8, npf1=npf, npf2=npf, wxf1=5, wxf2=5)
    po = resolve_params(oracle, (W, H, F, 1), 15.0, **cfg)
    pg = resolve_params(gpulib, (W, H, F, 1), 15.0, **cfg)
    ob, of, orat, tr = oracle.runNlBayes(nz, ff, bf, *po, nparts=2, trace_cap=100000, trace_stride=32, vbm3d=True)
    gb, gf, grat = gpuctx.runNlBayes(nz, ff, bf, *pg, nparts=2, keep_groups=True, vbm3d=True)
    same_groups(gpuctx, tr, 2)
    assert np.array_equal(gb, ob, equal_nan=True) and np.array_equal(gf, of, equal_nan=True) and grat == orat
