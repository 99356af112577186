"""The index arithmetic of csrc/fl_index.cuh, compiled by the host's C++ compiler: the
split of the CG plan into ranges of equal weight up to the largest grid that the
entry points accept (2^30 cells: the weights' sum passes 2^32), the tiles in which the
chunks are listed, and the division by a grid extent."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fluid-simulation_gb300", "csrc")

# k_cg_plan's use of the header, its 256 threads one after the other: every thread's
# weight, the warps' sums in 32 bits, and each thread's entries through RangeSplit.
SHIM = r"""
#include "fl_index.cuh"
#include <vector>
using namespace fl;
template <class F>
static void threads(const uint8_t* flag, uint32_t nchunks, uint32_t per_chunk, uint32_t parts, uint32_t* start,
                    uint32_t* list, F each) {
    std::vector<uint32_t> w(CHUNK, 0), n(CHUNK, 0);
    uint32_t sums[CHUNK / 32] = {};
    for (uint32_t t = 0; t < (uint32_t)CHUNK; t++) {
        each(t, [&](uint32_t c) { if (c < nchunks && flag[c]) { n[t]++; w[t] += flag[c] + per_chunk; } });
        sums[t / 32] += w[t];
    }
    uint32_t e = 0;
    for (uint32_t t = 0; t < (uint32_t)CHUNK; t++) {
        uint64_t before, all;
        weights_of_warps(sums, CHUNK / 32, t / 32, before, all);
        uint32_t in_warp = 0;
        for (uint32_t u = t / 32 * 32; u < t; u++) in_warp += w[u];
        RangeSplit split(before + in_warp, all, parts);
        each(t, [&](uint32_t c) {
            if (c >= nchunks || !flag[c]) return;
            list[e++] = c;
            split.add(flag[c] + per_chunk, e, start);
        });
    }
}
extern "C" {
uint32_t max_cells() { return MAX_CELLS; }
uint32_t chunk_weight() { return CHUNK_WEIGHT; }
void split_segments(const uint8_t* flag, uint32_t nchunks, uint32_t per_chunk, uint32_t parts, uint32_t* start, uint32_t* list) {
    threads(flag, nchunks, per_chunk, parts, start, list,
            [&](uint32_t t, auto&& f) { for (uint32_t c = t; c < nchunks; c += CHUNK) f(c); });
}
void split_tiles(const uint8_t* flag, uint32_t nx, uint32_t ny, uint32_t nchunks, uint32_t per_chunk, uint32_t parts,
                 uint32_t* start, uint32_t* list) {
    const ChunkTiles tiles(nx, ny, nchunks);
    const uint32_t per = (tiles.count + CHUNK - 1) / CHUNK;
    threads(flag, nchunks, per_chunk, parts, start, list, [&](uint32_t t, auto&& f) {
        for (uint32_t k = t * per; k < (t + 1) * per && k < tiles.count; k++)
            for (uint32_t i = 0; i < TILE_Y * TILE_Z; i++) f(tiles.chunk(k, i));
    });
}
void divide(const uint32_t* n, uint32_t count, uint32_t d, uint32_t* q) {
    uint32_t mul, shift;
    division_by(d, mul, shift);
    for (uint32_t i = 0; i < count; i++) q[i] = quotient(n[i], mul, shift);
}
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("index")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I" + CSRC, str(d / "shim.cpp"), "-o", str(d / "shim.so")],
                   check=True)
    return ctypes.CDLL(str(d / "shim.so"))


def ptr(a):
    return ctypes.c_void_p(a.ctypes.data)


def check(lib, dims, flag, parts, per_chunk, tiles):
    nchunks = flag.size
    start, lst = np.full(parts + 8, 77, np.uint32), np.zeros(max(1, int((flag > 0).sum())), np.uint32)
    start[0] = 0
    if tiles:
        lib.split_tiles(ptr(flag), dims[0], dims[1], nchunks, per_chunk, parts, ptr(start), ptr(lst))
    else:
        lib.split_segments(ptr(flag), nchunks, per_chunk, parts, ptr(start), ptr(lst))
    active = np.flatnonzero(flag)
    if tiles:
        assert np.array_equal(np.sort(lst), active)  # every active chunk once
    else:
        order = np.arange(-(-nchunks // 256) * 256).reshape(-1, 256).T.ravel()
        order = order[order < nchunks]
        assert np.array_equal(lst, order[flag[order] > 0])
    # block b starts behind the first entry up to which the weight is b / parts of the whole
    upto = np.cumsum(flag[lst].astype(np.int64) + per_chunk)
    want = 1 + np.searchsorted(upto * parts, np.arange(1, parts + 1) * upto[-1])
    assert np.array_equal(start[1:parts + 1], want)
    assert start[parts] == active.size and (start[parts + 1:] == 77).all()  # nothing is written past the ranges


@pytest.mark.parametrize("dims", [(1024, 1024, 1024), (950, 953, 950), (3, 3, 119304647), (16384, 16384, 4), (16000, 16000, 4)])
@pytest.mark.parametrize("tiles", [False, True])
def test_ranges_of_full_grids(lib, dims, tiles):
    nchunks = -(-dims[0] * dims[1] * dims[2] // 256)
    assert dims[0] * dims[1] * dims[2] <= lib.max_cells()
    check(lib, dims, np.full(nchunks, 255, np.uint8), 152, lib.chunk_weight(), tiles)


@pytest.mark.parametrize("dims,parts", [((64, 64, 64), 7), ((97, 61, 83), 152), ((250, 120, 250), 152), ((10, 10, 999), 13),
                                        ((36, 36, 300), 151), ((256, 256, 256), 256)])
@pytest.mark.parametrize("tiles", [False, True])
@pytest.mark.parametrize("per_chunk", [32, 1024])
def test_ranges_of_ragged_fill(lib, dims, parts, tiles, per_chunk):
    rng = np.random.default_rng(sum(dims) + parts)
    flag = rng.integers(0, 256, -(-dims[0] * dims[1] * dims[2] // 256)).astype(np.uint8)
    flag[rng.uniform(size=flag.size) < 0.5] = 0
    check(lib, dims, flag, parts, per_chunk, tiles)


def test_quotients_are_exact(lib):
    rng = np.random.default_rng(3)
    for d in list(range(2, 300)) + [511, 512, 513, 1000, 1023, 1024, 1025, 65535, 2**20 + 7, 2**30]:
        near = rng.integers(0, 2**31 // d, 200)[:, None] * d + np.arange(-1, 2)
        n = np.concatenate([near.ravel(), rng.integers(0, 2**31, 500), [0, 1, d - 1, d, 2**31 - 1]])
        n = np.clip(n, 0, 2**31 - 1).astype(np.uint32)
        q = np.empty_like(n)
        lib.divide(ptr(n), n.size, d, ptr(q))
        assert np.array_equal(q, n // np.uint32(d)), d
