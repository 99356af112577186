// fl_index.cuh — index arithmetic that the host, the kernels and a plain C++
// compiler share: division by a grid extent, the chunk tiles and the split of
// the CG's plan.  No CUDA header is needed to compile it.
#pragma once
#include <cstddef>
#include <cstdint>

#if defined(__CUDACC__)
#define FL_HD __host__ __device__
#else
#define FL_HD
#endif

namespace fl {

constexpr uint32_t MAX_CELLS = 1u << 30;  // of a grid that the entry points accept
constexpr int CHUNK = 256;                // cells per reduction chunk (the 256-wide workgroup of cg_reduce.wgsl)
constexpr uint32_t MAX_CG_BLOCKS = 256;
// Per-chunk cost in liquid-cell units for ranges of equal weight: a warp takes a
// chunk at once, so a sparsely filled one costs it nearly as much as a full one
// (with 256, the slowest block at 256^3 got 170 chunks where the others had 150);
// solvers that list cells use 32.
constexpr uint32_t CHUNK_WEIGHT = 1024, CELL_CHUNK_WEIGHT = 32;
constexpr uint32_t MAX_CHUNK_WEIGHT = 255 + CHUNK_WEIGHT;  // chunk flags count up to 255 liquid cells

// Multiplier and shift of a division by d >= 2 of numbers below 2^31:
// n / d = (n * mul >> 32) >> shift with mul = ceil(2^(31 + L) / d), shift = L - 1,
// L = ceil(log2 d).  mul exceeds 2^(31+L) / d by less than 1 <= 2^L / d, so the
// product is above n / d by less than 1 / d for n < 2^31 and the quotient is exact
// (Granlund and Montgomery 1994).
inline void division_by(uint32_t d, uint32_t& mul, uint32_t& shift) {
    uint32_t L = 1;
    while ((1ull << L) < d) L++;
    mul = (uint32_t)(((1ull << (31 + L)) + d - 1) / d);
    shift = L - 1;
}
FL_HD inline uint32_t quotient(uint32_t n, uint32_t mul, uint32_t shift) {
    return (uint32_t)((uint64_t)n * mul >> 32) >> shift;
}

// The tiles in which a plan may list the chunks: TILE_Y neighbours along y by TILE_Z
// planes of Z chunks (whole ones: the tiles shear a little where a plane is no
// multiple of a chunk).  Every chunk is in one tile whatever Z is.
constexpr uint32_t TILE_Y = 4, TILE_Z = 4;
struct ChunkTiles {
    uint32_t nchunks, Z, ty, count;
    FL_HD ChunkTiles(uint32_t nx, uint32_t ny, uint32_t nchunks_) : nchunks(nchunks_) {
        Z = nx * ny / CHUNK ? nx * ny / CHUNK : 1u;
        ty = (Z + TILE_Y - 1) / TILE_Y;
        const uint32_t planes = (nchunks + Z - 1) / Z;
        count = ty * ((planes + TILE_Z - 1) / TILE_Z);
    }
    // Chunk i (below TILE_Y * TILE_Z) of tile t; past nchunks where there is none.
    FL_HD uint32_t chunk(uint32_t t, uint32_t i) const {
        const uint32_t y = TILE_Y * (t % ty) + i % TILE_Y, c = (TILE_Z * (t / ty) + i / TILE_Y) * Z + y;
        return y < Z ? c : nchunks;
    }
};

// Weights before a warp's and in all, from the warps' sums.  A warp's sum fits 32
// bits; the total does not: 2^30 cells are 4,194,304 chunks of up to
// MAX_CHUNK_WEIGHT, 5.4e9.
FL_HD inline void weights_of_warps(const uint32_t* sums, uint32_t warps, uint32_t warp, uint64_t& before, uint64_t& all) {
    before = all = 0;
    for (uint32_t w = 0; w < warps; w++) {
        if (w < warp) before += sums[w];
        all += sums[w];
    }
}
// (a warp of the plan's eight takes an eighth of the segments or of the tiles; tiles at
// the far sides hold fewer chunks, so an eighth of them is up to 8/5 x 8/5 of an eighth
// of the chunks, and a remainder)
static_assert((uint64_t)(MAX_CELLS / CHUNK * 3 / 8 + 32 * TILE_Y * TILE_Z) * MAX_CHUNK_WEIGHT < (1ull << 32),
              "a warp's sum of weights exceeds 32 bits");
static_assert((uint64_t)(MAX_CELLS / CHUNK) * MAX_CHUNK_WEIGHT < (1ull << 63) / MAX_CG_BLOCKS,
              "RangeSplit's products exceed 64 bits");

// Ranges of equal weight: with X and X1 the weights before and after an entry,
// blocks b with X * parts < b * W <= X1 * parts start after it.  X only grows along
// a thread's entries, so the next such block is tracked from one division.
struct RangeSplit {
    uint64_t W, XG, bW;  // total, parts x the weight so far, next * W
    uint32_t parts, next;
    FL_HD RangeSplit(uint64_t before, uint64_t total, uint32_t parts_) : W(total), XG(before * parts_), parts(parts_) {
        next = W ? (uint32_t)(XG / W) + 1u : 1u;  // at most parts + 1: before <= total
        bW = next * W;
    }
    // An entry of this weight; `end` entries are listed with it.
    FL_HD void add(uint32_t weight, uint32_t end, uint32_t* start) {
        XG += (uint64_t)weight * parts;
        for (; next <= parts && bW <= XG; next++, bW += W) start[next] = end;
    }
};

}  // namespace fl
