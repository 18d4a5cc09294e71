"""The exact search by 2 x 2 blocks of reference patches (search_block.cu): the
neighbour lists and outputs of every shape it has an instantiation for, equal to
the oracle's, at grid sizes that leave single columns and rows over, with
windows cut by the borders, and on inputs that its fast comparison cannot
decide: near-equal and equal distances, values that are not finite or whose
squares overflow, and windows that lie far apart."""
import numpy as np
import pytest

from helpers import resolve_params, video_case

pytestmark = pytest.mark.gpu

P4 = dict(px1=4, px2=4, pt1=4, pt2=4, wx1=21, wx2=21, np1=16, np2=16, b1=3.0)
P8 = dict(px1=8, px2=8, pt1=1, pt2=1, wx1=21, wx2=21, np1=16, np2=16, b1=3.0)


def check(gpulib, gpuctx, oracle, nz, ff, bf, cli, sigma=20.0, nparts=2):
    F, C, H, W = nz.shape
    po = resolve_params(oracle, (W, H, F, C), sigma, **cli)
    pg = resolve_params(gpulib, (W, H, F, C), sigma, **cli)
    ob, of, orat, tr = oracle.runNlBayes(nz, ff, bf, *po, nparts=nparts, trace_cap=200000, trace_stride=32)
    gb, gf, grat = gpuctx.runNlBayes(nz, ff, bf, *pg, nparts=nparts, keep_groups=True)
    for step in (1, 2):
        for tile in range(nparts):
            sel = (tr["step"] == step) & (tr["tile"] == tile)
            gg = gpuctx.groups(step, tile)
            assert np.array_equal(gg["nsimp"], tr["nsimp"][sel])
            assert np.array_equal(gg["index"], tr["index"][sel])
    assert np.array_equal(gb, ob, equal_nan=True) and np.array_equal(gf, of, equal_nan=True) and grat == orat


@pytest.mark.parametrize("W,H,F,C,cli", [
    (37, 41, 6, 1, P4),                                   # 4x4x4, steps 3 and 2
    (38, 30, 4, 3, P4),                                   # three channels compared in step 2
    (44, 39, 13, 1, dict(P4, wx1=9, wx2=15)),             # 9-frame range, smaller windows
    (29, 26, 5, 1, dict(P4, np1=32, np2=32)),             # windows cut on every side, 32 neighbours
    (50, 45, 1, 1, P8),                                   # 8x8, step 3
    (61, 43, 7, 1, {}),                                   # defaults: 8x8 step 6, 7x7 step 4
    (53, 47, 1, 1, dict(px2=7)),                          # image defaults, 7x7 step 3
    (58, 46, 6, 1, dict(px1=8, px2=8)),                   # 8x8, steps 6 and 4
    (70, 52, 1, 3, {}),                                   # image defaults: 39x39 window, 32 neighbours
])
def test_gpu_block_search_shapes(gpulib, gpuctx, oracle, W, H, F, C, cli):
    _, nz, ff, bf = video_case(W, H, F, sigma=20.0, seed=W + H, channels=C)
    check(gpulib, gpuctx, oracle, nz, ff, bf, cli)


@pytest.mark.parametrize("levels", [2, 16, 256])
@pytest.mark.parametrize("cli,F", [(P4, 5), (P8, 1)], ids=["px4", "px8"])
def test_gpu_block_search_equal_distances(gpulib, gpuctx, oracle, levels, cli, F):
    # whole numbers of few levels: exactly equal distances in most windows
    # (std::partial_sort's heap orders them)
    rng = np.random.default_rng(levels)
    nz = rng.integers(0, levels, (F, 1, 36, 41)).astype(np.float32) * np.float32(200 // levels)
    check(gpulib, gpuctx, oracle, nz, None, None, cli, sigma=10.0)


@pytest.mark.parametrize("scale", [1e-21, 1e-3, 1e15])
def test_gpu_block_search_near_equal_distances(gpulib, gpuctx, oracle, scale):
    # a periodic frame with rounding-sized differences between its copies, at
    # scales where squares underflow or grow large
    rng = np.random.default_rng(4)
    cell = rng.uniform(1, 2, (6, 7)).astype(np.float32)
    nz = np.tile(cell, (5, 1, 6, 6)).astype(np.float32)
    nz = (nz * (1 + np.float32(2.0 ** -23) * rng.integers(-2, 3, nz.shape)) * np.float32(scale)).astype(np.float32)
    check(gpulib, gpuctx, oracle, nz, None, None, P4, sigma=float(scale))


@pytest.mark.parametrize("value", [np.inf, np.nan, 3e19, -1e18])
def test_gpu_block_search_extreme_values(gpulib, gpuctx, oracle, value):
    _, nz, ff, bf = video_case(36, 33, 5, sigma=20.0, seed=8)
    nz[2, 0, 15, 17] = value
    F, C, H, W = nz.shape
    po = resolve_params(oracle, (W, H, F, C), 20.0, **P4)
    pg = resolve_params(gpulib, (W, H, F, C), 20.0, **P4)
    po[1].sizePatch = pg[1].sizePatch = 0     # step 1: its source holds the value
    ob, _, orat, tr = oracle.runNlBayes(nz, ff, bf, *po, nparts=2, trace_cap=100000, trace_stride=16)
    gb, _, grat = gpuctx.runNlBayes(nz, ff, bf, *pg, nparts=2, keep_groups=True)
    for tile in range(2):
        gg = gpuctx.groups(1, tile, stride=16)
        assert np.array_equal(gg["index"], tr["index"][tr["tile"] == tile])
    assert np.array_equal(gb, ob, equal_nan=True) and grat == orat


def test_gpu_block_search_windows_far_apart(gpulib, gpuctx, oracle):
    # flows that jump by hundreds of pixels between neighbouring patches
    W, H, F = 330, 40, 5
    _, nz, ff, bf = video_case(W, H, F, sigma=20.0, seed=12)
    rng = np.random.default_rng(6)
    jump = rng.choice([0.0, 300.0, -300.0, 40.0], (F, 1, H // 5, W // 5)).astype(np.float32)
    jump = np.kron(jump, np.ones((1, 1, 5, 5), np.float32))
    ff[:, :1] += jump
    bf[:, :1] -= jump
    check(gpulib, gpuctx, oracle, nz, ff, bf, dict(P4, wx1=9, wx2=9))
