"""The warp filter (filter.cu: filter_warp_kernel), bit for bit against the
oracle: every patch shape it takes, at member counts below, at and between its
lane counts (8, 16, 32), groups of different sizes side by side (a small tau
truncates some), one to four channels, order invariance, groups whose members
are all equal beside others, and more groups than one run of a warp."""
import numpy as np
import pytest

from helpers import resolve_params, video_case

pytestmark = pytest.mark.gpu

P4 = dict(px1=4, px2=4, pt1=4, pt2=4, wx1=9, wx2=9, b1=3.0)
P87 = dict(px1=8, px2=7, pt1=1, pt2=1, wx1=11, wx2=9)
P78 = dict(px1=7, px2=8, pt1=1, pt2=1, wx1=9, wx2=11)


def check(gpulib, gpuctx, oracle, nz, ff, bf, cli, sigma=20.0, tau=None):
    F, C, H, W = nz.shape
    po = resolve_params(oracle, (W, H, F, C), sigma, **cli)
    pg = resolve_params(gpulib, (W, H, F, C), sigma, **cli)
    if tau is not None:
        for p in po + pg:
            p.tau = tau
    ob, of, orat = oracle.runNlBayes(nz, ff, bf, *po, nparts=2)
    gb, gf, grat = gpuctx.runNlBayes(nz, ff, bf, *pg, nparts=2)
    assert np.array_equal(gb, ob, equal_nan=True) and np.array_equal(gf, of, equal_nan=True) and grat == orat


@pytest.mark.parametrize("cli", [P4, P87, P78], ids=["4x4x4", "8x8-7x7", "7x7-8x8"])
@pytest.mark.parametrize("np_,C,oinv", [(2, 1, False), (7, 3, False), (8, 1, True), (15, 1, False), (16, 4, False),
                                         (16, 3, True), (31, 1, False), (32, 3, False)])
def test_gpu_filter_member_counts(gpulib, gpuctx, oracle, cli, np_, C, oinv):
    _, nz, ff, bf = video_case(35, 33, 5, sigma=20.0, seed=np_ * 8 + C, channels=C)
    check(gpulib, gpuctx, oracle, nz, ff, bf, dict(cli, np1=np_, np2=np_, order_inv=oinv))


@pytest.mark.parametrize("cli", [P4, P87], ids=["4x4x4", "8x8-7x7"])
def test_gpu_filter_uneven_groups(gpulib, gpuctx, oracle, cli):
    # the nearest distances straddle tau: 1 to 16 members
    _, nz, ff, bf = video_case(60, 44, 6, sigma=20.0, seed=5)
    check(gpulib, gpuctx, oracle, nz, ff, bf, dict(cli, np1=16, np2=16), tau=21.0)


@pytest.mark.parametrize("C", [1, 3])
def test_gpu_filter_equal_groups_beside_others(gpulib, gpuctx, oracle, C):
    # constant areas beside noise: groups left as they are, with the weights of
    # the groups before them
    rng = np.random.default_rng(C)
    nz = np.full((5, C, 40, 48), 90.0, np.float32)
    nz[:, :, :, 20:] += rng.normal(0, 20, nz[:, :, :, 20:].shape).astype(np.float32)
    for cli in (P4, P87):
        check(gpulib, gpuctx, oracle, nz, None, None, dict(cli, np1=16, np2=8))
