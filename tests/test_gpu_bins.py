"""The ordered aggregation by bins of 16 x 16 pixels (aggregate.cu:
bin_list_kernel, bin_gather_kernel) at the sizes where it can go wrong, bit for
bit against the oracle: videos one pixel short of, equal to and past whole
bins, each patch shape that has its own instantiation, groups whose members
come from far apart (flows of many pixels, so that the box of groups around a
bin exceeds its bitmap), and more entries in one bin than fit its list."""
import numpy as np
import pytest

from helpers import resolve_params, video_case

pytestmark = pytest.mark.gpu

P4 = dict(px1=4, px2=4, wx1=9, wx2=9, np1=16, np2=16, b1=3.0)


def check(gpulib, gpuctx, oracle, nz, ff, bf, cli, sigma=20.0, nparts=2):
    F, C, H, W = nz.shape
    po = resolve_params(oracle, (W, H, F, C), sigma, **cli)
    pg = resolve_params(gpulib, (W, H, F, C), sigma, **cli)
    ob, of, orat = oracle.runNlBayes(nz, ff, bf, *po, nparts=nparts)
    gb, gf, grat = gpuctx.runNlBayes(nz, ff, bf, *pg, nparts=nparts)
    assert np.array_equal(gb, ob) and np.array_equal(gf, of) and grat == orat


@pytest.mark.parametrize("W,H,F,C,px,pt", [
    (31, 33, 4, 1, 4, 4), (32, 16, 5, 1, 4, 4), (33, 47, 9, 1, 4, 2), (17, 48, 4, 3, 4, 4),
    (31, 33, 3, 1, 8, 1), (48, 17, 2, 3, 7, 1), (33, 32, 2, 4, 8, 1), (32, 31, 3, 3, 4, 1),
    (33, 31, 5, 1, 5, 1), (30, 34, 6, 1, 3, 3), (34, 32, 7, 3, 2, 5), (32, 33, 5, 4, 4, 4)])
def test_gpu_bin_edges(gpulib, gpuctx, oracle, W, H, F, C, px, pt):
    _, nz, ff, bf = video_case(W, H, F, sigma=20.0, seed=W * 64 + H, channels=C)
    check(gpulib, gpuctx, oracle, nz, ff, bf, dict(P4, px1=px, px2=px, pt1=pt, pt2=pt))


@pytest.mark.parametrize("px,pt", [(4, 4), (8, 1)])
def test_gpu_members_from_far_apart(gpulib, gpuctx, oracle, px, pt):
    # every pixel's flow points somewhere else: a bin's members come from
    # groups all over the frame
    W, H, F = 150, 90, 6
    _, nz, ff, bf = video_case(W, H, F, sigma=20.0, seed=77)
    rng = np.random.default_rng(3)
    ff, bf = (rng.uniform(-120, 120, f.shape).astype(np.float32) for f in (ff, bf))
    check(gpulib, gpuctx, oracle, nz, ff, bf, dict(P4, px1=px, px2=px, pt1=pt, pt2=pt))


def test_gpu_many_slots_in_one_bin(gpulib, gpuctx, oracle):
    # one frame that repeats a 16 x 16 cell: every group picks its members
    # among exact copies, the first ones in the window's order
    rng = np.random.default_rng(9)
    cell = rng.uniform(0, 255, (16, 16)).astype(np.float32)
    nz = np.tile(cell, (5, 6))[None, None].copy()
    nz[:, :, 40:, 50:] += 0.25
    check(gpulib, gpuctx, oracle, nz, None, None, dict(px1=8, px2=8, wx1=39, wx2=39, np1=32, np2=32), nparts=1)
