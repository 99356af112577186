// fl_mg.cu — multigrid-preconditioned CG, an opt-in pressure solver
// (fl_params.pressure_solver = FL_SOLVER_MGPCG).
//
// The reference solves the pressure system with plain CG (cg_*.wgsl) and
// ships a red-black Gauss-Seidel smoother (pressure.wgsl:26-61, built but not
// dispatched: gpu/fluid.rs:564-627) and a CPU Jacobi solver
// (sim/pressure.rs:68-136).  Here red-black Gauss-Seidel is the smoother of a
// multigrid V-cycle that preconditions CG.  Operator, right-hand side, warm
// start, iteration cap and stopping test (r.r <= tol^2 * r0.r0, tested after
// each update like cg_beta.wgsl:25-30) are the CG's; the iterates are not, so
// the pressure matches the CG's to the tolerance, not bit for bit.
//
// Hierarchy: level l+1 aggregates 2x2x2 cells of level l (the last aggregate
// of an odd extent has fewer).  Prolongation P is piecewise-constant
// injection, restriction is P^T (sum over the children) and the coarse
// operator is the exact Galerkin product P^T A P, which stays a 7-point
// stencil with integer weights: the weight between two aggregates is the
// number of liquid-liquid fine faces across their interface, the diagonal is
// the children's diagonals minus twice their internal couplings.  Stored as
// float4 {diag, weight to +x, +y, +z}; a cell is an unknown when diag > 0.
// V-cycle: one red-then-black sweep down, black-then-red up, symmetric
// Gauss-Seidel sweeps on the coarsest level (<= 64 cells), all from zero: a
// symmetric positive-definite preconditioner.
//
// One cooperative persistent kernel per solve, one 1024-thread block per SM.
// Level-0 cells are owned through the CG's plan of active chunks (k_cg_plan,
// split over blocks 1..G-1 when G > 1) and listed in shared memory with their
// stencil masks; level 1's unknowns are listed per block; other grid levels
// are split into one cell range per block.  The levels of at most
// MG_BLOCK0_CELLS cells run inside block 0 alone, with block barriers and
// their b, x and stencils in shared memory (the stencils in the cell-list
// space that block 0 does not need when it owns no level-0 cells).  A
// grid pass boundary is a counter barrier (bounded wait, as in k_cg); a dot
// product is a per-block float-float partial, a barrier and a fixed-order
// sum, so results repeat bit for bit.  Each smoothing pass computes what it
// needs of the other colour on the fly (the red values of the pre-smoothing
// sweep are b/D; the corrected red values of the post-smoothing sweep are
// x + e(parent)), so a level costs four passes: pre-smooth, residual +
// restriction (eight lanes per coarse cell), correction + black sweep, red
// sweep; on level 0 the CG update is fused with the pre-smoothing.
#include "fl_device.cuh"

// Vectors written during the solve (r, z, d, the coarse b and x) are read
// through plain pointers, never const __restrict__: a read-only (non-coherent)
// load could return a value cached before another block's write.  The
// stencils and masks are fixed for the whole kernel.

namespace fl {

namespace {

constexpr int MG_THREADS = 1024;
constexpr int MG_PART = 1024;             // block partial slots per exchange parity
constexpr int MG_CELLS = 20480;           // level-0 unknowns listed per block
constexpr int MG_L1 = 4096;               // level-1 unknowns listed per block
constexpr int MG_COARSE_SWEEPS = 2;       // symmetric Gauss-Seidel sweeps on the coarsest level

// Level-0 cell metadata: bits 0-9 the CG's stencil mask (bit 0 liquid, bit
// s+1 neighbour s of -x,+x,-y,+y,-z,+z liquid, bits 7-9 the non-solid count),
// bits 10-12 the parities of i, j, k, bit 13 the colour (i+j+k)&1 (0 = red).
constexpr uint32_t META_IODD = 1u << 10, META_JODD = 1u << 11, META_KODD = 1u << 12, META_BLACK = 1u << 13;

// A level that block 0 runs alone, as its passes need it (set up once per
// solve: deriving it in every pass cost more than the cells).
struct LocalLevel {
    MgLevel lv;               // vectors (and stencils) in shared memory
    uint32_t mx, mxy;         // SmallDiv's reciprocals
    uint32_t n[2], first[2];  // unknowns per colour, their places in MgShared::loc (blacks go down)
};

struct MgShared {
    uint32_t cell[MG_CELLS];
    uint16_t meta[MG_CELLS];
    uint32_t l1[MG_L1];
    float lb[MG_LOCAL_TOTAL], lx[MG_LOCAL_TOTAL];  // b and x of the levels block 0 runs alone
    uint16_t loc[MG_LOCAL_TOTAL];                  // and their unknowns, by colour
    LocalLevel local[MG_MAX_LEVELS];
    float2 red[MG_THREADS / 32];
    uint32_t wc[MG_THREADS / 32];
    float2 res;
    int ok;
    uint64_t limit;  // of a wait, in ns
    uint32_t n0[2], n1[2], list0, list1;  // unknowns listed per colour: level 0, level 1
    // solve scalars kept here rather than in registers through the loop
    float2 rs0, thr, rz;
};

__device__ __forceinline__ uint32_t make_meta(uint32_t info, uint32_t c, uint32_t nx, uint32_t ny) {
    const uint32_t i = c % nx, j = (c / nx) % ny, k = c / (nx * ny);
    return info | ((i & 1u) ? META_IODD : 0u) | ((j & 1u) ? META_JODD : 0u) | ((k & 1u) ? META_KODD : 0u) |
           (((i + j + k) & 1u) ? META_BLACK : 0u);
}

__device__ __forceinline__ float diag0(uint32_t meta) { return (float)((meta >> 7) & 7u); }

// Stencils and masks do not change during the solve: read-only cache.
__device__ __forceinline__ uint32_t ld_ci(const uint16_t* ci, uint32_t c) { return __ldg(ci + c); }

// The passes are chains of L2 loads, one cell or two per thread, so what a cell
// costs is the number of loads that wait for one another.  Every load of a cell
// is issued before the first value is used, and volatile (ld_if): the compiler
// would otherwise move each load behind the test that decides whether its value is
// needed (each neighbour then waited for the one before: 107 us per iteration
// on the 128^3 sphere-into-pool scene, against 91; 69 with the lists below).
__device__ __forceinline__ uint32_t ld_ci_if(const uint16_t* p, bool on) {
    uint32_t v;
    asm volatile("{\n.reg .pred q;\nsetp.ne.u32 q, %2, 0;\nmov.u32 %0, 0;\n@q ld.global.nc.u16 %0, [%1];\n}"
                 : "=r"(v)
                 : "l"(p), "r"((uint32_t)on));
    return v;
}
// Where a coarse level's vectors and stencils are: global memory, block 0's
// shared memory, or (a grid of one block) vectors in shared memory and
// stencils in global.
enum Mem { GRID, LOCAL, LOCAL_ONE };
template <Mem M>
__device__ __forceinline__ float ld_x(const float* p) {
    float v;
    if (M == GRID) asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    else asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"((uint32_t)__cvta_generic_to_shared(p)));
    return v;
}
template <Mem M>
__device__ __forceinline__ float4 ld_st(const float4* p) {  // fixed during the solve: read-only cache
    if (M != LOCAL) return __ldg(p);
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"((uint32_t)__cvta_generic_to_shared(p)));
    return v;
}

// The neighbours of level-0 cell c in side order (-x, +x, -y, +y, -z, +z), and
// whether each is liquid.
struct Nb0 {
    uint32_t n[6];
    bool on[6];
    __device__ __forceinline__ Nb0(uint32_t mask, uint32_t c, uint32_t nx, uint32_t nxy) {
        const uint32_t m[6] = {c - 1, c + 1, c - nx, c + nx, c - nxy, c + nxy};
#pragma unroll
        for (int s = 0; s < 6; s++) {
            on[s] = (mask >> (s + 1)) & 1u;
            n[s] = m[s];
        }
    }
    __device__ __forceinline__ void load(const float* a, float (&v)[6]) const {
#pragma unroll
        for (int s = 0; s < 6; s++) v[s] = ld_if(a + n[s], on[s]);
    }
};
// a[n] / D[n] of the liquid neighbours, summed in side order, from their values
// and stencil words.
__device__ __forceinline__ float quotient_sum(const Nb0& nb, const float (&v)[6], const uint32_t (&ci)[6]) {
    float s = 0.0f;
#pragma unroll
    for (int k = 0; k < 6; k++)
        if (nb.on[k]) s += v[k] / (float)(ci[k] >> 7);
    return s;
}

// A coarse cell's neighbours in the order +x, +y, +z, -x, -y, -z: indices (the
// cell itself where the grid ends) and weights (0: not an unknown).
template <Mem M>
struct NbC {
    uint32_t n[6];
    float w[6];
    __device__ __forceinline__ NbC(const float4* st, float4 sc, uint32_t c, uint32_t i, uint32_t j, uint32_t k,
                                   const MgLevel& lv) {
        const uint32_t nx = lv.nx, nxy = lv.nx * lv.ny;
        n[0] = sc.y != 0.0f ? c + 1 : c;
        n[1] = sc.z != 0.0f ? c + nx : c;
        n[2] = sc.w != 0.0f ? c + nxy : c;
        n[3] = i ? c - 1 : c;
        n[4] = j ? c - nx : c;
        n[5] = k ? c - nxy : c;
        const float wx = ld_st<M>(st + n[3]).y, wy = ld_st<M>(st + n[4]).z, wz = ld_st<M>(st + n[5]).w;
        w[0] = sc.y; w[1] = sc.z; w[2] = sc.w;
        w[3] = i ? wx : 0.0f;
        w[4] = j ? wy : 0.0f;
        w[5] = k ? wz : 0.0f;
    }
    __device__ __forceinline__ void load(const float* a, float (&v)[6]) const {
#pragma unroll
        for (int s = 0; s < 6; s++) v[s] = ld_x<M>(a + n[s]);
    }
    __device__ __forceinline__ float sum(const float (&v)[6]) const {
        float t = 0.0f;
#pragma unroll
        for (int s = 0; s < 6; s++) t += w[s] != 0.0f ? w[s] * v[s] : 0.0f;
        return t;
    }
};

// The coarse cell (aggregate) holding the cell at (i, j, k), or cell c.
__device__ __forceinline__ uint32_t parent_at(uint32_t i, uint32_t j, uint32_t k, const MgLevel& up) {
    return (i >> 1) + up.nx * ((j >> 1) + up.ny * (k >> 1));
}
__device__ __forceinline__ uint32_t parent_of(uint32_t c, uint32_t nx, uint32_t ny, const MgLevel& up) {
    return parent_at(c % nx, (c / nx) % ny, c / (nx * ny), up);
}

struct Ctx {
    MgShared& sh;
    const DevBufs& b;
    const MgBufs& m;
    uint32_t e0, nown;  // this block's level-0 plan entries
    uint32_t Lg;        // first level run inside block 0 alone (>= 1)
    const float* r;     // the current residual (level 0's b)
    uint32_t epoch;     // barriers so far
    uint32_t parity;    // exchange slot parity
    float4* lst;        // block 0: shared-memory copy of the stencils of levels Lg.. (nullptr: global)
};

__device__ bool mg_barrier(Ctx& x) {
    return grid_barrier(x.m.bar, ++x.epoch, x.sh.limit, &x.b.st->status, &x.sh.ok);
}

// Sum of v over all threads of all blocks, in a fixed order; false on abort.
__device__ bool mg_allreduce(Ctx& x, Df v, Df& out) {
    v = warp_sum_df(v);
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (lane == 0) x.sh.red[warp] = make_float2(v.hi, v.lo);
    __syncthreads();
    float2* part = x.m.part + (size_t)x.parity * MG_PART;
    x.parity ^= 1u;
    if (warp == 0) {  // one lane adding the 32 one after the other took 2,000 cycles
        static_assert(MG_THREADS / 32 == 32, "a lane per warp");
        const Df s = warp_sum_df(Df{x.sh.red[lane].x, x.sh.red[lane].y});
        if (lane == 0) part[blockIdx.x] = make_float2(s.hi, s.lo);
    }
    if (!mg_barrier(x)) return false;
    if (warp == 0) {
        Df s = {0.0f, 0.0f};
        for (uint32_t g0 = 0; g0 < gridDim.x; g0 += 8 * 32) {
            Df p[8];
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const uint32_t g = g0 + lane + 32u * k;
                const float2 v2 = g < gridDim.x ? part[g] : make_float2(0.0f, 0.0f);
                p[k] = {v2.x, v2.y};
            }
            s = df_add(s, df_tree(p));
        }
        s = warp_allsum_df(s);
        if (lane == 0) x.sh.res = make_float2(s.hi, s.lo);
    }
    __syncthreads();
    out = Df{x.sh.res.x, x.sh.res.y};
    return true;
}

// Position of this thread's item among the flagged items of the block (in
// thread order) and their total; uses sh.wc.
__device__ __forceinline__ uint32_t block_rank(MgShared& sh, bool flag, uint32_t& total) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t ball = __ballot_sync(0xffffffffu, flag);
    if (lane == 0) sh.wc[warp] = __popc(ball);
    __syncthreads();
    uint32_t off = 0, tot = 0;
    for (uint32_t w = 0; w < MG_THREADS / 32; w++) {
        const uint32_t v = sh.wc[w];
        off += w < warp ? v : 0u;
        tot += v;
    }
    __syncthreads();
    total = tot;
    return off + __popc(ball & ((1u << lane) - 1u));
}

// This block's share of a coarse grid level: groups of 32 cells dealt out in
// turn, so that blocks get equal numbers of unknowns wherever the liquid is
// (contiguous ranges gave the slowest block twice the median's work in a pool).
// share_size counts them (the last group may reach past the level's end),
// share_cell gives the e-th.
__device__ __forceinline__ uint32_t share_size(uint32_t C) {
    const uint32_t groups = (C + 31) / 32;
    return blockIdx.x < groups ? ((groups - blockIdx.x + gridDim.x - 1) / gridDim.x) * 32u : 0u;
}
__device__ __forceinline__ uint32_t share_cell(uint32_t e) { return ((e >> 5) * gridDim.x + blockIdx.x) * 32u + (e & 31u); }

// Lists this block's level-0 unknowns (plan order) and level-1 unknowns.
__device__ void build_lists(Ctx& x) {
    MgShared& sh = x.sh;
    const DevParams& P = *x.b.prm;
    const uint32_t C = P.C, nx = P.nx, ny = P.ny, lo = threadIdx.x & (CHUNK - 1);
    uint32_t nr = 0, nb = 0;
    for (uint32_t base = 0; base < x.nown; base += MG_THREADS / CHUNK) {
        const uint32_t e = base + threadIdx.x / CHUNK;
        uint32_t c = 0, info = 0;
        if (e < x.nown) {
            c = x.b.cg_chunk[x.e0 + e] * CHUNK + lo;
            if (c < C) info = ld_ci(x.b.cinfo, c);
        }
        const bool u = info >= (1u << 7);
        const uint32_t meta = u ? make_meta(info, c, nx, ny) : 0u;
        const bool black = (meta & META_BLACK) != 0u;
        uint32_t totr, totb;
        const uint32_t pr = nr + block_rank(sh, u && !black, totr), pb = nb + block_rank(sh, u && black, totb);
        nr += totr;
        nb += totb;
        if (u && nr + nb <= (uint32_t)MG_CELLS) {  // reds from the front, blacks from the back
            const uint32_t at = black ? MG_CELLS - 1 - pb : pr;
            sh.cell[at] = c;
            sh.meta[at] = (uint16_t)meta;
        }
    }
    const MgLevel& l1 = x.m.lv[1];
    uint32_t n1r = 0, n1b = 0;
    const uint32_t n1 = share_size(l1.C);
    for (uint32_t base = 0; base < n1; base += MG_THREADS) {
        const uint32_t e = base + threadIdx.x, I = share_cell(e);
        const bool u = e < n1 && I < l1.C && ld_st<GRID>(l1.st + I).x > 0.0f;
        const bool black = u && ((I % l1.nx + (I / l1.nx) % l1.ny + I / (l1.nx * l1.ny)) & 1u) != 0u;
        uint32_t totr, totb;
        const uint32_t pr = n1r + block_rank(sh, u && !black, totr), pb = n1b + block_rank(sh, u && black, totb);
        n1r += totr;
        n1b += totb;
        if (u && n1r + n1b <= (uint32_t)MG_L1) sh.l1[black ? MG_L1 - 1 - pb : pr] = I;
    }
    if (threadIdx.x == 0) {
        sh.n0[0] = nr;
        sh.n0[1] = nb;
        sh.list0 = nr + nb <= (uint32_t)MG_CELLS;
        sh.n1[0] = n1r;
        sh.n1[1] = n1b;
        sh.list1 = n1r + n1b <= (uint32_t)MG_L1;
    }
    __syncthreads();
}

// f(c, meta) for every level-0 unknown of this block of a colour (0 red, 1
// black).  The colours are listed apart: a pass that treats them differently
// keeps all lanes at work.
template <class F>
__device__ __forceinline__ void for_own(const Ctx& x, uint32_t colour, F f) {
    const MgShared& sh = x.sh;
    if (sh.list0) {
        const uint32_t n = sh.n0[colour];
        for (uint32_t e = threadIdx.x; e < n; e += MG_THREADS) {
            const uint32_t at = colour ? MG_CELLS - 1 - e : e;
            f(sh.cell[at], (uint32_t)sh.meta[at]);
        }
        return;
    }
    const DevParams& P = *x.b.prm;
    const uint32_t C = P.C, lo = threadIdx.x & (CHUNK - 1);
    for (uint32_t e = threadIdx.x / CHUNK; e < x.nown; e += MG_THREADS / CHUNK) {
        const uint32_t c = x.b.cg_chunk[x.e0 + e] * CHUNK + lo;
        if (c >= C) continue;
        const uint32_t info = ld_ci(x.b.cinfo, c);
        if (info < (1u << 7)) continue;
        const uint32_t meta = make_meta(info, c, P.nx, P.ny);
        if (((meta & META_BLACK) != 0u) == (colour != 0u)) f(c, meta);
    }
}

// f(c, i, j, k, st) for every unknown of coarse level l of a colour: level 1 and
// the local levels (block 0 alone, shared memory) from lists, other grid levels
// over this block's share.
// (i, j, k) of cell c of a level of at most MG_BLOCK0_CELLS cells by
// multiply-high with rounded-up reciprocals ceil(2^32 / d): exact because
// c * d stays below 2^32 (integer division by a runtime divisor is a long
// instruction sequence, and the levels block 0 runs alone are issue-bound).
// A divisor of 1 is stored as 0.
struct SmallDiv {
    uint32_t nx, nxy, mx, mxy;
    __device__ __forceinline__ static uint32_t recip(uint32_t d) { return d > 1u ? 0xffffffffu / d + 1u : 0u; }
    __device__ __forceinline__ explicit SmallDiv(const LocalLevel& l)
        : nx(l.lv.nx), nxy(l.lv.nx * l.lv.ny), mx(l.mx), mxy(l.mxy) {}
    __device__ __forceinline__ void ijk(uint32_t c, uint32_t& i, uint32_t& j, uint32_t& k) const {
        k = mxy ? __umulhi(c, mxy) : c;
        const uint32_t rem = c - k * nxy;
        j = mx ? __umulhi(rem, mx) : rem;
        i = rem - j * nx;
    }
};
static_assert((uint64_t)MG_BLOCK0_CELLS * MG_BLOCK0_CELLS < (1ull << 32), "SmallDiv needs c * divisor < 2^32");

// colour: 0 red, 1 black.
template <Mem M, class F>
__device__ __forceinline__ void for_level(const Ctx& x, uint32_t l, const MgLevel& lv, uint32_t colour, F f) {
    if (M != GRID) {
        const LocalLevel& ll = x.sh.local[l];
        const SmallDiv dv(ll);
        const uint32_t n = ll.n[colour], at0 = ll.first[colour];
        for (uint32_t e = threadIdx.x; e < n; e += MG_THREADS) {
            const uint32_t c = x.sh.loc[colour ? at0 - e : at0 + e];
            uint32_t i, j, k;
            dv.ijk(c, i, j, k);
            f(c, i, j, k, ld_st<M>(lv.st + c));
        }
        return;
    }
    auto ijk = [&](uint32_t c, uint32_t& i, uint32_t& j, uint32_t& k) {
        i = c % lv.nx;
        j = (c / lv.nx) % lv.ny;
        k = c / (lv.nx * lv.ny);
    };
    if (l == 1 && x.sh.list1) {
        const uint32_t n = x.sh.n1[colour];
        for (uint32_t e = threadIdx.x; e < n; e += MG_THREADS) {
            const uint32_t c = x.sh.l1[colour ? MG_L1 - 1 - e : e];
            uint32_t i, j, k;
            ijk(c, i, j, k);
            f(c, i, j, k, ld_st<M>(lv.st + c));
        }
        return;
    }
    const uint32_t n = share_size(lv.C);
    for (uint32_t e = threadIdx.x; e < n; e += MG_THREADS) {
        const uint32_t c = share_cell(e);
        if (c >= lv.C) continue;
        const float4 sc = ld_st<GRID>(lv.st + c);
        uint32_t i, j, k;
        ijk(c, i, j, k);
        if (sc.x > 0.0f && ((i + j + k) & 1u) == colour) f(c, i, j, k, sc);
    }
}

// ---- level 0 passes (b = r, x = z) ----

// pre-smoothing from zero: red z = r/D; black z = (r + sum r_nb/D_nb)/D
__device__ void pre0(const Ctx& x) {
    const DevParams& P = *x.b.prm;
    const uint32_t nx = P.nx, nxy = nx * P.ny;
    const float* r = x.r;
    const uint16_t* ci = x.b.cinfo;
    float* z = x.m.lv[0].x;
    for_own(x, 1, [&](uint32_t c, uint32_t meta) {
        const Nb0 nb(meta, c, nx, nxy);
        float rn[6];
        uint32_t cn[6];
        nb.load(r, rn);
#pragma unroll
        for (int s = 0; s < 6; s++) cn[s] = ld_ci_if(ci + nb.n[s], nb.on[s]);
        const float rc = ld_if(r + c, true);
        z[c] = (rc + quotient_sum(nb, rn, cn)) / diag0(meta);
    });
    for_own(x, 0, [&](uint32_t c, uint32_t meta) { z[c] = r[c] / diag0(meta); });
}

// p += alpha d.  Nothing waits for p: it is advanced while block 0 runs the coarse
// levels and the other blocks have nothing else to do (a pool at 128^3, 22
// iterations: 1,555 -> 1,540 us).
__device__ void advance_p(const Ctx& x, float alpha, const float* d) {
    float* p = x.b.p;
    for (uint32_t colour = 0; colour < 2; colour++)
        for_own(x, colour, [&](uint32_t c, uint32_t) {
            const float pc = ld_if(p + c, true), dc = ld_if(d + c, true);
            p[c] = pc + alpha * dc;
        });
}

// The CG update of r fused with pre0: r_next = r - alpha q, and the
// pre-smoothing of r_next (a black cell's red neighbours' r_next computed on
// the fly from their r and q, which this pass does not change).  Returns this
// thread's share of r_next . r_next.
__device__ Df update_pre0(const Ctx& x, float alpha, float* r_next) {
    const DevParams& P = *x.b.prm;
    const uint32_t nx = P.nx, nxy = nx * P.ny;
    const float* r = x.r;
    const float* q = x.b.q;
    const uint16_t* ci = x.b.cinfo;
    float* z = x.m.lv[0].x;
    Df acc = {0.0f, 0.0f};
    for_own(x, 1, [&](uint32_t c, uint32_t meta) {
        const Nb0 nb(meta, c, nx, nxy);
        float rn[6], qn[6];
        uint32_t cn[6];
        nb.load(r, rn);
        nb.load(q, qn);
#pragma unroll
        for (int s = 0; s < 6; s++) cn[s] = ld_ci_if(ci + nb.n[s], nb.on[s]);
        const float rc = ld_if(r + c, true), qc = ld_if(q + c, true);
#pragma unroll
        for (int s = 0; s < 6; s++) rn[s] -= alpha * qn[s];
        const float rnew = rc - alpha * qc;
        r_next[c] = rnew;
        z[c] = (rnew + quotient_sum(nb, rn, cn)) / diag0(meta);
        acc = df_add(acc, df_prod(rnew, rnew));
    });
    for_own(x, 0, [&](uint32_t c, uint32_t meta) {
        const float rc = ld_if(r + c, true), qc = ld_if(q + c, true);
        const float rnew = rc - alpha * qc;
        r_next[c] = rnew;
        z[c] = rnew / diag0(meta);
        acc = df_add(acc, df_prod(rnew, rnew));
    });
    return acc;
}

// Unknowns of level l (grid pass: this block's share; local: all), eight
// consecutive lanes per cell: f(I, ii, jj, kk, child d = lane & 7) returns the
// child's term, the eight terms are summed in a fixed shuffle order and
// g(I, sum) runs on the first lane.  A cell's children are visited together.
template <Mem M, class F, class G>
__device__ __forceinline__ void for_level8(const Ctx& x, uint32_t l, const MgLevel& lv, F f, G g) {
    constexpr bool local = M != GRID;
    const uint32_t d = threadIdx.x & 7u, slot = threadIdx.x >> 3;
    constexpr uint32_t per = MG_THREADS / 8;
    const LocalLevel& ll = x.sh.local[l];
    const SmallDiv dv(ll);  // used for local levels only (at most MG_BLOCK0_CELLS cells)
    auto one = [&](bool valid, uint32_t I) {
        float t = 0.0f;
        if (valid) {
            uint32_t ii, jj, kk;
            if (local) {
                dv.ijk(I, ii, jj, kk);
            } else {
                ii = I % lv.nx;
                jj = (I / lv.nx) % lv.ny;
                kk = I / (lv.nx * lv.ny);
            }
            t = f(I, ii, jj, kk, d);
        }
        t += __shfl_xor_sync(0xffffffffu, t, 1);
        t += __shfl_xor_sync(0xffffffffu, t, 2);
        t += __shfl_xor_sync(0xffffffffu, t, 4);
        if (valid && d == 0) g(I, t);
    };
    if (local || (l == 1 && x.sh.list1)) {  // the lists: reds, then blacks
        const uint32_t nr = local ? ll.n[0] : x.sh.n1[0], n = nr + (local ? ll.n[1] : x.sh.n1[1]);
        const uint32_t r0 = local ? ll.first[0] : 0u, b0 = local ? ll.first[1] : MG_L1 - 1u;
        for (uint32_t e0 = 0; e0 < n; e0 += per) {
            const uint32_t e = e0 + slot, at = e < nr ? r0 + e : b0 - (e - nr);
            one(e < n, e < n ? (local ? (uint32_t)x.sh.loc[at] : x.sh.l1[at]) : 0u);
        }
        return;
    }
    const uint32_t n = share_size(lv.C);
    for (uint32_t e0 = 0; e0 < n; e0 += per) {
        const uint32_t e = e0 + slot, I = share_cell(e);
        const bool in = e < n && I < lv.C;
        one(in && ld_st<GRID>(lv.st + (in ? I : 0u)).x > 0.0f, I);
    }
}

// b1 = P^T (r - A z)
__device__ void restrict0(const Ctx& x) {
    const DevParams& P = *x.b.prm;
    const uint32_t nx = P.nx, ny = P.ny, nz = P.nz, nxy = nx * ny, last = P.C - 1;
    const float* r = x.r;
    const uint16_t* ci = x.b.cinfo;
    const float* z = x.m.lv[0].x;
    const MgLevel& up = x.m.lv[1];
    for_level8<GRID>(
        x, 1, up,
        [&](uint32_t, uint32_t ii, uint32_t jj, uint32_t kk, uint32_t d) {
            const uint32_t i = 2 * ii + (d & 1), j = 2 * jj + ((d >> 1) & 1), k = 2 * kk + (d >> 2);
            if (i >= nx || j >= ny || k >= nz) return 0.0f;
            const uint32_t c = i + nx * (j + ny * k);
            // the neighbours' z with the cell's own stencil word (some cell
            // where the grid ends), kept where the word names them
            const uint32_t info = ld_ci_if(ci + c, true);
            const uint32_t n[6] = {c - 1, c + 1, c - nx, c + nx, c - nxy, c + nxy};
            float zn[6];
#pragma unroll
            for (int s = 0; s < 6; s++) zn[s] = ld_if(z + (n[s] < last ? n[s] : last), true);
            const float rc = ld_if(r + c, true), zc = ld_if(z + c, true);
            if (info < (1u << 7)) return 0.0f;
            float sum = 0.0f;
#pragma unroll
            for (int s = 0; s < 6; s++) sum += (info >> (s + 1)) & 1u ? zn[s] : 0.0f;
            return rc - (diag0(info) * zc - sum);
        },
        [&](uint32_t I, float s) { up.b[I] = s; });
}

// correction + black sweep: z_black = (r + sum (z_red + e(parent))) / D
__device__ void post0_black(const Ctx& x) {
    const DevParams& P = *x.b.prm;
    const uint32_t nx = P.nx, ny = P.ny, nxy = nx * ny;
    const float* r = x.r;
    float* z = x.m.lv[0].x;
    const MgLevel& up = x.m.lv[1];
    const float* e = up.x;
    const uint32_t unx = up.nx, unxy = up.nx * up.ny;
    for_own(x, 1, [&](uint32_t c, uint32_t meta) {
        const Nb0 nb(meta, c, nx, nxy);
        const uint32_t pc = parent_of(c, nx, ny, up);
        const bool io = meta & META_IODD, jo = meta & META_JODD, ko = meta & META_KODD;
        // parents of the neighbours: the own parent, or the next one when the
        // step leaves the 2x2x2 aggregate
        const uint32_t pn[6] = {io ? pc : pc - 1, io ? pc + 1 : pc, jo ? pc : pc - unx, jo ? pc + unx : pc,
                                ko ? pc : pc - unxy, ko ? pc + unxy : pc};
        float zn[6], en[6];
        nb.load(z, zn);
#pragma unroll
        for (int s = 0; s < 6; s++) en[s] = ld_if(e + pn[s], nb.on[s]);
        const float rc = ld_if(r + c, true);
        float sum = 0.0f;
#pragma unroll
        for (int s = 0; s < 6; s++)
            if (nb.on[s]) sum += zn[s] + en[s];
        z[c] = (rc + sum) / diag0(meta);
    });
}

// red sweep; returns this thread's share of r.z
__device__ Df post0_red(const Ctx& x) {
    const DevParams& P = *x.b.prm;
    const uint32_t nx = P.nx, nxy = nx * P.ny;
    const float* r = x.r;
    float* z = x.m.lv[0].x;
    Df acc = {0.0f, 0.0f};
    for_own(x, 0, [&](uint32_t c, uint32_t meta) {
        const Nb0 nb(meta, c, nx, nxy);
        float zn[6];
        nb.load(z, zn);
        const float rc = ld_if(r + c, true);
        float sum = 0.0f;
#pragma unroll
        for (int s = 0; s < 6; s++) sum += zn[s];  // 0 where there is none
        const float zc = (rc + sum) / diag0(meta);
        z[c] = zc;
        acc = df_add(acc, df_prod(rc, zc));
    });
    for_own(x, 1, [&](uint32_t c, uint32_t) {
        const float rc = ld_if(r + c, true), zc = ld_if(z + c, true);
        acc = df_add(acc, df_prod(rc, zc));
    });
    return acc;
}

// ---- coarse level passes (grid levels, or block 0's local levels) ----

// Pre-smoothing from zero: red x = b/D, black x = (b + sum w b_nb/D_nb)/D.  Block
// 0 alone puts a block barrier between the colours and reads the reds' quotients.
template <Mem M>
__device__ void pre_l(const Ctx& x, uint32_t l, const MgLevel& lv) {
    const float4* st = lv.st;
    auto red = [&](uint32_t c, uint32_t, uint32_t, uint32_t, float4 sc) { lv.x[c] = lv.b[c] / sc.x; };
    constexpr bool local = M != GRID;
    if (local) {
        for_level<M>(x, l, lv, 0, red);
        __syncthreads();
    }
    for_level<M>(x, l, lv, 1, [&](uint32_t c, uint32_t i, uint32_t j, uint32_t k, float4 sc) {
        const NbC<M> nb(st, sc, c, i, j, k, lv);
        float bn[6], dn[6];
        nb.load(local ? lv.x : lv.b, bn);
#pragma unroll
        for (int s = 0; s < 6; s++) dn[s] = local ? 1.0f : ld_st<M>(st + nb.n[s]).x;
        const float bc = ld_x<M>(lv.b + c);
        float sum = 0.0f;
#pragma unroll
        for (int s = 0; s < 6; s++)
            if (nb.w[s] != 0.0f) sum += nb.w[s] * (local ? bn[s] : bn[s] / dn[s]);
        lv.x[c] = (bc + sum) / sc.x;
    });
    if (!local) for_level<M>(x, l, lv, 0, red);
}

template <Mem M>
__device__ void restrict_l(const Ctx& x, uint32_t l, const MgLevel& lv, const MgLevel& up) {
    const float4* st = lv.st;
    for_level8<M>(
        x, l + 1, up,
        [&](uint32_t, uint32_t ii, uint32_t jj, uint32_t kk, uint32_t d) {
            const uint32_t i = 2 * ii + (d & 1), j = 2 * jj + ((d >> 1) & 1), k = 2 * kk + (d >> 2);
            if (i >= lv.nx || j >= lv.ny || k >= lv.nz) return 0.0f;
            const uint32_t c = i + lv.nx * (j + lv.ny * k);
            const float4 sc = ld_st<M>(st + c);
            const float bc = ld_x<M>(lv.b + c), xc = ld_x<M>(lv.x + c);
            if (!(sc.x > 0.0f)) return 0.0f;
            const NbC<M> nb(st, sc, c, i, j, k, lv);
            float xn[6];
            nb.load(lv.x, xn);
            return bc - (sc.x * xc - nb.sum(xn));
        },
        [&](uint32_t I, float s) { up.b[I] = s; });
}

template <Mem M>
__device__ void post_black_l(const Ctx& x, uint32_t l, const MgLevel& lv, const MgLevel& up) {
    const float4* st = lv.st;
    for_level<M>(x, l, lv, 1, [&](uint32_t c, uint32_t i, uint32_t j, uint32_t k, float4 sc) {
        const NbC<M> nb(st, sc, c, i, j, k, lv);
        const uint32_t pc = parent_at(i, j, k, up), unx = up.nx, unxy = up.nx * up.ny;
        // the neighbours' parents (the own one where there is no neighbour)
        const uint32_t pn[6] = {nb.n[0] != c && (i & 1u) ? pc + 1 : pc,       nb.n[1] != c && (j & 1u) ? pc + unx : pc,
                                nb.n[2] != c && (k & 1u) ? pc + unxy : pc,    nb.n[3] != c && !(i & 1u) ? pc - 1 : pc,
                                nb.n[4] != c && !(j & 1u) ? pc - unx : pc,    nb.n[5] != c && !(k & 1u) ? pc - unxy : pc};
        float xn[6], en[6];
        nb.load(lv.x, xn);
#pragma unroll
        for (int s = 0; s < 6; s++) en[s] = ld_x<M>(up.x + pn[s]);
        const float bc = ld_x<M>(lv.b + c);
#pragma unroll
        for (int s = 0; s < 6; s++) xn[s] += en[s];
        lv.x[c] = (bc + nb.sum(xn)) / sc.x;
    });
}

template <Mem M>
__device__ void post_red_l(const Ctx& x, uint32_t l, const MgLevel& lv) {
    const float4* st = lv.st;
    for_level<M>(x, l, lv, 0, [&](uint32_t c, uint32_t i, uint32_t j, uint32_t k, float4 sc) {
        const NbC<M> nb(st, sc, c, i, j, k, lv);
        float xn[6];
        nb.load(lv.x, xn);
        const float bc = ld_x<M>(lv.b + c);
        lv.x[c] = (bc + nb.sum(xn)) / sc.x;
    });
}

// Levels Lg .. L-1 by block 0 alone (block barriers instead of grid
// barriers): V-cycle with symmetric Gauss-Seidel sweeps from zero on the
// coarsest level.
template <Mem M>
__device__ void local_cycle(const Ctx& x) {
    const uint32_t L = x.m.L, Lg = x.Lg;
    {
        const MgLevel g = x.m.lv[Lg], s = x.sh.local[Lg].lv;
        for (uint32_t c = threadIdx.x; c < g.C; c += MG_THREADS) s.b[c] = g.b[c];
        __syncthreads();
    }
    for (uint32_t l = Lg; l + 1 < L; l++) {
        const MgLevel lv = x.sh.local[l].lv, up = x.sh.local[l + 1].lv;
        pre_l<M>(x, l, lv);
        __syncthreads();
        restrict_l<M>(x, l, lv, up);
        __syncthreads();
    }
    {
        const MgLevel lv = x.sh.local[L - 1].lv;
        const uint32_t t = threadIdx.x, nx = lv.nx, ny = lv.ny, nxy = nx * ny;
        uint32_t i = 0, j = 0, k = 0, col = 0;
        float4 sc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (t < lv.C) {
            i = t % nx; j = (t / nx) % ny; k = t / nxy;
            col = (i + j + k) & 1u;
            sc = ld_st<M>(lv.st + t);
            lv.x[t] = 0.0f;
        }
        const uint32_t at = t < lv.C ? t : 0u;
        const NbC<M> nb(lv.st, sc, at, i, j, k, lv);
        const float bt = lv.b[at];
        __syncthreads();
        for (int h = 0; h < 4 * MG_COARSE_SWEEPS; h++) {
            // forward sweeps red, black; backward sweeps black, red
            const uint32_t want = h < 2 * MG_COARSE_SWEEPS ? (uint32_t)(h & 1) : (uint32_t)((h & 1) ^ 1);
            if (t < lv.C && sc.x > 0.0f && col == want) {
                float xn[6];
                nb.load(lv.x, xn);
                lv.x[t] = (bt + nb.sum(xn)) / sc.x;
            }
            __syncthreads();
        }
    }
    for (uint32_t l = L - 1; l-- > Lg;) {
        const MgLevel lv = x.sh.local[l].lv, up = x.sh.local[l + 1].lv;
        post_black_l<M>(x, l, lv, up);
        __syncthreads();
        post_red_l<M>(x, l, lv);
        __syncthreads();
    }
    {
        const MgLevel g = x.m.lv[Lg], s = x.sh.local[Lg].lv;
        for (uint32_t c = threadIdx.x; c < g.C; c += MG_THREADS) g.x[c] = s.x[c];
    }
}

// z = M^-1 r, then the r.z all-reduce (whose barrier ends the cycle).  With
// presmoothed, pre0 and its barrier have already run (update_pre0), and p has
// yet to advance by alpha d.
__device__ bool vcycle(Ctx& x, Df& rz, bool presmoothed, float alpha = 0.0f, const float* d = nullptr) {
    const MgBufs& m = x.m;
    const uint32_t Lg = x.Lg;
    if (!presmoothed) {
        pre0(x);
        if (!mg_barrier(x)) return false;
    }
    restrict0(x);
    if (!mg_barrier(x)) return false;
    for (uint32_t l = 1; l < Lg; l++) {
        pre_l<GRID>(x, l, m.lv[l]);
        if (!mg_barrier(x)) return false;
        restrict_l<GRID>(x, l, m.lv[l], m.lv[l + 1]);
        if (!mg_barrier(x)) return false;
    }
    if (presmoothed) advance_p(x, alpha, d);  // block 0 of several owns no cells
    if (blockIdx.x == 0) {
        if (x.lst) local_cycle<LOCAL>(x);
        else local_cycle<LOCAL_ONE>(x);
    }
    if (!mg_barrier(x)) return false;
    for (uint32_t l = Lg; l-- > 1;) {
        post_black_l<GRID>(x, l, m.lv[l], m.lv[l + 1]);
        if (!mg_barrier(x)) return false;
        post_red_l<GRID>(x, l, m.lv[l]);
        if (!mg_barrier(x)) return false;
    }
    post0_black(x);
    if (!mg_barrier(x)) return false;
    return mg_allreduce(x, post0_red(x), rz);
}

__global__ void __launch_bounds__(MG_THREADS, 1) k_mgpcg(DevBufs b, MgBufs m) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    MgShared& sh = *reinterpret_cast<MgShared*>(smem_raw);
    const DevParams& P = *b.prm;
    const uint32_t tid = threadIdx.x;
    const uint32_t* start = b.cg_off + CHUNK + 3;
    uint32_t Lg = 1;
    while (Lg + 1 < m.L && m.lv[Lg].C > MG_BLOCK0_CELLS) Lg++;
    // With more than one block, block 0 owns no level-0 cells (launch_mgpcg
    // splits the plan over blocks 1..G-1): it runs the coarse levels alone
    // while the others wait, and its cell list space holds their stencils, so
    // its sweeps read shared memory instead of chains of L2 loads.
    const bool b0_local = gridDim.x > 1;
    uint32_t e0 = 0, nown = 0;
    if (!b0_local || blockIdx.x > 0) {
        const uint32_t pb = b0_local ? blockIdx.x - 1 : 0u;
        e0 = start[pb];
        nown = start[pb + 1] - start[pb];
    }
    Ctx x{sh, b, m, e0, nown, Lg, b.r, 0u, 0u, nullptr};
    if (tid == 0) sh.limit = wait_limit_ns(&P);
    build_lists(x);
    if (blockIdx.x == 0) {  // the unknowns of the levels it runs alone
        uint32_t off = 0;
        for (uint32_t l = Lg; l < m.L; l++) {
            const MgLevel& lv = m.lv[l];
            uint32_t nr = 0, nb = 0;
            for (uint32_t base = 0; base < lv.C; base += MG_THREADS) {
                const uint32_t c = base + tid;
                const bool u = c < lv.C && ld_st<GRID>(lv.st + c).x > 0.0f;
                const bool black = u && ((c % lv.nx + (c / lv.nx) % lv.ny + c / (lv.nx * lv.ny)) & 1u) != 0u;
                uint32_t totr, totb;
                const uint32_t pr = nr + block_rank(sh, u && !black, totr), pb = nb + block_rank(sh, u && black, totb);
                if (u) sh.loc[black ? off + lv.C - 1 - pb : off + pr] = (uint16_t)c;
                nr += totr;
                nb += totb;
            }
            if (tid == 0) {
                LocalLevel& ll = sh.local[l];
                ll.lv = lv;
                ll.lv.b = sh.lb + off;
                ll.lv.x = sh.lx + off;
                if (b0_local) ll.lv.st = reinterpret_cast<float4*>(sh.cell) + off;
                ll.mx = SmallDiv::recip(lv.nx);
                ll.mxy = SmallDiv::recip(lv.nx * lv.ny);
                ll.n[0] = nr;
                ll.n[1] = nb;
                ll.first[0] = off;
                ll.first[1] = off + lv.C - 1;
            }
            off += lv.C;
        }
        __syncthreads();
    }
    if (b0_local && blockIdx.x == 0) {
        static_assert(sizeof(sh.cell) >= MG_LOCAL_TOTAL * sizeof(float4), "local stencils exceed the cell list");
        float4* lst = reinterpret_cast<float4*>(sh.cell);
        uint32_t off = 0;
        for (uint32_t l = Lg; l < m.L; l++) {
            for (uint32_t c = tid; c < m.lv[l].C; c += MG_THREADS) lst[off + c] = ld_st<GRID>(m.lv[l].st + c);
            off += m.lv[l].C;
        }
        x.lst = lst;
        __syncthreads();
    }
    const uint32_t nx = P.nx, nxy = P.nx * P.ny;
    const uint32_t iters = P.iters;
    const bool stop_on = P.tol_sq > 0.0f;
    float* q = b.q;
    const float* z = m.lv[0].x;
    DevStats* st = b.st;

    // r0.r0 (grid_prep left r = rhs - A p0)
    Df acc = {0.0f, 0.0f};
    for (uint32_t colour = 0; colour < 2; colour++)
        for_own(x, colour, [&](uint32_t c, uint32_t) {
            const float rc = x.r[c];
            acc = df_add(acc, df_prod(rc, rc));
        });
    Df rs;
    if (!mg_allreduce(x, acc, rs)) return;
    if (tid == 0) {
        const double thr = P.thr_abs ? P.thr_abs_d : (double)P.tol_sq_d * df_to_double(rs);
        const float hi = (float)thr;
        sh.rs0 = make_float2(rs.hi, rs.lo);
        sh.thr = make_float2(hi, (float)(thr - (double)hi));
    }
    {
        Df rz;
        if (!vcycle(x, rz, false)) return;  // its barriers also publish rs0 and thr
        if (tid == 0) sh.rz = make_float2(rz.hi, rz.lo);
    }
    float beta = 0.0f;
    uint32_t k = 0;
    for (uint32_t it = 0; it < iters; it++) {
        float* d_cur = (it & 1u) ? b.dB : b.dA;
        const float* d_prev = (it & 1u) ? b.dA : b.dB;
        const bool first = it == 0;
        // direction d = z + beta d_prev and q = A d (neighbours' d on the fly)
        acc = Df{0.0f, 0.0f};
        for (uint32_t colour = 0; colour < 2; colour++)
            for_own(x, colour, [&](uint32_t c, uint32_t meta) {
                const Nb0 nb(meta, c, nx, nxy);
                float zn[6], dn[6];
                nb.load(z, zn);
#pragma unroll
                for (int s = 0; s < 6; s++) dn[s] = ld_if(d_prev + nb.n[s], nb.on[s] && !first);
                const float zc = ld_if(z + c, true), dp = ld_if(d_prev + c, !first);
                auto dir = [&](float zv, float dv) { return first ? zv : zv + beta * dv; };
                float sum = 0.0f;
#pragma unroll
                for (int s = 0; s < 6; s++) sum += dir(zn[s], dn[s]);  // 0 where there is none
                const float dc = dir(zc, dp), qc = diag0(meta) * dc - sum;
                d_cur[c] = dc;
                q[c] = qc;
                acc = df_add(acc, df_prod(dc, qc));
            });
        Df dq;
        if (!mg_allreduce(x, acc, dq)) return;
        // cg_alpha.wgsl:16-22: alpha = 0 when |d.q| <= 1e-30
        const float alpha = fabsf(dq.hi) > 1e-30f ? df_div(Df{sh.rz.x, sh.rz.y}, dq) : 0.0f;
        // residuals alternate between r and r2: neighbours' old values are
        // read while the new ones are written
        float* r_next = x.r == b.r ? m.r2 : b.r;
        if (!mg_allreduce(x, update_pre0(x, alpha, r_next), rs)) return;
        x.r = r_next;
        k = it + 1;
        if (it + 1 == iters || (stop_on && df_le(rs, Df{sh.thr.x, sh.thr.y}))) {
            advance_p(x, alpha, d_cur);
            break;
        }
        Df rz_new;
        if (!vcycle(x, rz_new, true, alpha, d_cur)) return;
        const Df rz = {sh.rz.x, sh.rz.y};
        beta = rz.hi > 1e-30f ? df_div(rz_new, rz) : 0.0f;  // cg_beta.wgsl:16-23
        __syncthreads();
        if (tid == 0) sh.rz = make_float2(rz_new.hi, rz_new.lo);
    }
    if (blockIdx.x == 0 && tid == 0) {
        st->cg_iters = k;
        st->rs_init = df_to_double(Df{sh.rs0.x, sh.rs0.y});
        st->rs_final = df_to_double(rs);
    }
}

// Level 1 from the grid's stencil masks.
__global__ void __launch_bounds__(256) k_mg_agg0(DevBufs b, MgBufs m) {
    after_previous();
    const DevParams& P = *b.prm;
    const uint32_t nx = P.nx, ny = P.ny, nz = P.nz;
    const MgLevel& up = m.lv[1];
    for (uint32_t I = blockIdx.x * blockDim.x + threadIdx.x; I < up.C; I += gridDim.x * blockDim.x) {
        const uint32_t ii = I % up.nx, jj = (I / up.nx) % up.ny, kk = I / (up.nx * up.ny);
        float D = 0.0f, wx = 0.0f, wy = 0.0f, wz = 0.0f;
        for (uint32_t d = 0; d < 8; d++) {
            const uint32_t dx = d & 1, dy = (d >> 1) & 1, dz = d >> 2;
            const uint32_t i = 2 * ii + dx, j = 2 * jj + dy, k = 2 * kk + dz;
            if (i >= nx || j >= ny || k >= nz) continue;
            const uint32_t info = b.cinfo[i + nx * (j + ny * k)];
            if (info < (1u << 7)) continue;
            D += diag0(info);
            if (info & (1u << 2)) { if (dx == 0) D -= 2.0f; else wx += 1.0f; }
            if (info & (1u << 4)) { if (dy == 0) D -= 2.0f; else wy += 1.0f; }
            if (info & (1u << 6)) { if (dz == 0) D -= 2.0f; else wz += 1.0f; }
        }
        up.st[I] = make_float4(D, wx, wy, wz);
    }
}

// Level l+1 from level l (l >= 1).
__global__ void __launch_bounds__(256) k_mg_agg(MgBufs m, uint32_t l) {
    after_previous();
    const MgLevel& lv = m.lv[l];
    const MgLevel& up = m.lv[l + 1];
    for (uint32_t I = blockIdx.x * blockDim.x + threadIdx.x; I < up.C; I += gridDim.x * blockDim.x) {
        const uint32_t ii = I % up.nx, jj = (I / up.nx) % up.ny, kk = I / (up.nx * up.ny);
        float D = 0.0f, wx = 0.0f, wy = 0.0f, wz = 0.0f;
        for (uint32_t d = 0; d < 8; d++) {
            const uint32_t dx = d & 1, dy = (d >> 1) & 1, dz = d >> 2;
            const uint32_t i = 2 * ii + dx, j = 2 * jj + dy, k = 2 * kk + dz;
            if (i >= lv.nx || j >= lv.ny || k >= lv.nz) continue;
            const float4 s = lv.st[i + lv.nx * (j + lv.ny * k)];
            if (!(s.x > 0.0f)) continue;
            D += s.x;
            if (dx == 0) D -= 2.0f * s.y; else wx += s.y;
            if (dy == 0) D -= 2.0f * s.z; else wy += s.z;
            if (dz == 0) D -= 2.0f * s.w; else wz += s.w;
        }
        up.st[I] = make_float4(D, wx, wy, wz);
    }
}

}  // namespace

int mg_max_blocks_per_sm() {
    int n = 0;
    if (cudaFuncSetAttribute(k_mgpcg, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(MgShared)) !=
        cudaSuccess)
        return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_mgpcg, MG_THREADS, sizeof(MgShared)) != cudaSuccess)
        return 0;
    return n;
}

// The caller has run k_grid_prep (r, p, cinfo, chunk_flag) and zeroed
// nothing: the plan, the barrier counter and the coarse operators are
// prepared here.  L.cg_blocks blocks (<= MG_PART), at most one per SM.
cudaError_t launch_mgpcg(const DevBufs& b, const MgBufs& m, const LaunchCfg& L, cudaStream_t s) {
    if (L.cg_blocks < 1 || L.cg_blocks > MG_PART || m.L < 2) return cudaErrorInvalidValue;
    // level-0 cells go to blocks 1..G-1 (block 0 runs the coarse levels)
    cudaError_t e = launch_cg_plan(b, L.cg_blocks > 1 ? (uint32_t)L.cg_blocks - 1 : 1u, s);
    if (e != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(m.bar, 0, BAR_BYTES, s)) != cudaSuccess) return e;
    const int gb = L.num_sms * 8;
    launch_after(k_mg_agg0, dim3(gb), 256, s, b, m);
    for (uint32_t l = 1; l + 1 < m.L; l++) launch_after(k_mg_agg, dim3(gb), 256, s, m, l);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(L.cg_blocks);
    cfg.blockDim = dim3(MG_THREADS);
    cfg.dynamicSmemBytes = sizeof(MgShared);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_mgpcg, b, m);
}

}  // namespace fl
