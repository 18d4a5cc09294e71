"""Chunk sizes of the filter and the aggregation: the arithmetic of chunk.hpp,
compiled here, and on the GPU the chunks that a memory limit and a batch's slot_mb
lead to."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from helpers import ROOT, resolve_params, video_case

P4 = dict(px1=4, px2=4, pt1=4, pt2=4, wx1=9, wx2=9, np1=16, np2=16, b1=3.0)

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include "chunk.hpp"
int main(int argc, char **argv)
{
	using namespace bm4dof;
	if (argc == 5) std::printf("%zu\n", chunk_bytes(std::atof(argv[1]), std::strtoull(argv[2], 0, 10),
	                                                std::strtoull(argv[3], 0, 10), std::atoi(argv[4]) != 0));
	else std::printf("%lld\n", chunk_groups(std::strtoull(argv[1], 0, 10), std::strtoull(argv[2], 0, 10),
	                                        std::atoi(argv[3]), std::atoi(argv[4]), std::atoll(argv[5])));
}
"""
MB, GB = 1 << 20, 1 << 30


@pytest.fixture(scope="module")
def chunk(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("chunk")
    (d / "m.cpp").write_text(SOURCE)
    subprocess.run([cxx, "-std=c++17", "-I", os.path.join(ROOT, "bm4d-of_gb300", "csrc"), str(d / "m.cpp"), "-o",
                    str(d / "m")], check=True)
    return lambda *a: int(subprocess.run([str(d / "m"), *map(str, a)], check=True, capture_output=True, text=True).stdout)


@pytest.mark.parametrize("env,usable,limit,tight,want", [
    (0, 280 * GB, 0, 0, 2 * GB), (0, 0, 0, 0, 2 * GB), (0, 16 * GB, 0, 0, GB),      # default; a full device
    (1000, 280 * GB, 0, 0, 200 * MB), (0.5, 280 * GB, 0, 0, MB // 10),              # the environment
    (100000, 280 * GB, 0, 0, 280 * GB // 16),
    (0, 280 * GB, GB, 0, 256 * MB), (0, 280 * GB, GB, 1, 32 * MB), (0, 280 * GB, 100 * GB, 0, 2 * GB)])   # a limit
def test_chunk_bytes(chunk, env, usable, limit, tight, want):
    assert chunk(env, usable, limit, tight) == want


@pytest.mark.parametrize("bytes_,per,np_,entries,G,want", [
    (GB, MB, 16, 8, 10 ** 6, 1024), (GB, MB, 16, 8, 100, 100), (1, MB, 16, 8, 100, 1),
    (300 * GB, 10880, 32, 20, 10 ** 9, (2 ** 32 - 1) // 640),      # 2x2x16 patches: 20 list entries a member
    (300 * GB, 2000, 32, 1, 10 ** 9, 2 ** 28 // 32)])
def test_chunk_groups(chunk, bytes_, per, np_, entries, G, want):
    n = chunk(bytes_, per, np_, entries, G)
    assert n == want and n * np_ * entries < 2 ** 32


@pytest.mark.gpu
def test_gpu_memory_limit_keeps_large_chunks(gpulib):
    # a quarter of the limit holds every group of a step: as few launches as without one
    W, H, F = 160, 120, 6
    _, nz, ff, bf = video_case(W, H, F, sigma=20.0, seed=3)
    p1, p2 = resolve_params(gpulib, (W, H, F, 1), 20.0, **P4)
    groups = max(len(t["xs"]) * len(t["ys"]) * len(t["fs"]) for p in (p1, p2) for t in gpulib.plan(W, H, F, p, nparts=1))
    ctx = gpulib.Context(0)
    try:
        want = ctx.runNlBayes(nz, ff, bf, p1, p2, nparts=1)
        free = ctx.timings()[1]
    finally:
        ctx.close()
    ctx = gpulib.Context(0)
    try:
        ctx.set_memory_limit(4 * groups * 16 * (64 + 1 + 8) * 4 + MB)
        got = ctx.runNlBayes(nz, ff, bf, p1, p2, nparts=1)
        assert ctx.timings()[1] == free
        # no room for that size: smaller chunks, the same results
        ctx.set_memory_limit(2 * groups * 16 * (64 + 1 + 8) * 4)
        small = ctx.runNlBayes(nz, ff, bf, p1, p2, nparts=1)
        for a, b in ((got, want), (small, want)):
            assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    finally:
        ctx.close()


@pytest.mark.gpu
def test_gpu_tight_memory_limit(gpulib):
    # the other buffers leave room for a 32nd of the limit, not for a quarter
    W, H, F = 160, 120, 6
    _, nz, ff, bf = video_case(W, H, F, sigma=20.0, seed=3)
    p1, p2 = resolve_params(gpulib, (W, H, F, 1), 20.0, **P4)
    ctx = gpulib.Context(0)
    try:
        want = ctx.runNlBayes(nz, ff, bf, p1, p2, nparts=1)
    finally:
        ctx.close()
    lo, hi = 1 * MB, 512 * MB
    while hi - lo > MB // 4:      # the smallest limit that a fresh context accepts
        mid = (lo + hi) // 2
        ctx = gpulib.Context(0)
        try:
            ctx.set_memory_limit(mid)
            b, f, _ = ctx.runNlBayes(nz, ff, bf, p1, p2, nparts=1)
            assert np.array_equal(b, want[0]) and np.array_equal(f, want[1])
            hi = mid
        except gpulib.BM4DOFError as e:
            assert e.status == "ERR_NO_MEMORY"
            lo = mid
        finally:
            ctx.close()
    print("smallest limit", hi)
    ctx = gpulib.Context(0)
    try:
        ctx.set_memory_limit(hi)
        for _ in range(2):        # the second call finds the buffers of the first
            b, f, _ = ctx.runNlBayes(nz, ff, bf, p1, p2, nparts=1)
            assert np.array_equal(b, want[0]) and np.array_equal(f, want[1])
    finally:
        ctx.close()


@pytest.mark.gpu
def test_gpu_slot_mb_is_the_chunk(gpulib, gpuctx):
    import torch
    W, H, F = 160, 120, 6
    _, nz, ff, bf = video_case(W, H, F, sigma=20.0, seed=3)
    p1, p2 = resolve_params(gpulib, (W, H, F, 1), 20.0, **P4)
    dev = [torch.from_numpy(a).cuda() for a in (nz, ff, bf)]
    item = dict(noisy=dev[0], fflow=dev[1], bflow=dev[2], basic=torch.empty_like(dev[0]), final=torch.empty_like(dev[0]),
                p1=p1, p2=p2, nparts=1)
    per = 16 * (64 + 1 + 8) * 4
    launches, chunks = [], []
    for mb in (1024, 20):
        gpuctx.run_batched([item], tuning=dict(slot_mb=mb))
        launches.append(gpuctx.timings()[1])
        chunks.append(sum(-(-sum(len(t["xs"]) * len(t["ys"]) * len(t["fs"]) for t in gpulib.plan(W, H, F, p, nparts=1)) //
                            (mb * MB // per)) for p in (p1, p2)))
    # filter 2 and aggregation 4 launches a chunk
    assert chunks[1] > chunks[0] and launches[1] - launches[0] == 6 * (chunks[1] - chunks[0]), (launches, chunks)
