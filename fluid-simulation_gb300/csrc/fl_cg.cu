// fl_cg.cu — persistent matrix-free CG for the MAC pressure Poisson system.
//
// One cooperative launch runs the whole solve that the reference issues as
// 9 dispatches per iteration (fluid.rs:1689-1701): cg_spmv, cg_reduce(d,q),
// cg_alpha, cg_update, cg_reduce(r,r), cg_beta, cg_dir.  Per iteration:
//
//   phase 1   d_new = r + beta*d_old (cg_dir.wgsl:30) fused with q = A d_new
//             (cg_spmv.wgsl:46-68); neighbours' d_new are recomputed from r and
//             d_old (same f32 ops, same bits), so no grid-wide step separates
//             the direction update from the stencil.  d ping-pongs between two
//             buffers.  One d.q partial per 256-cell chunk.
//   exchange  alpha = rs_old/dq (cg_alpha.wgsl)
//   phase 2   p += alpha d, r -= alpha q (cg_update.wgsl); r.r partials
//   exchange  beta and the convergence test (cg_beta.wgsl); the loop exits.
//
// A warp takes whole 256-cell chunks (the 256-wide workgroups of
// cg_reduce.wgsl).  Lane l holds the quads (four consecutive cells) l and
// l + 32 of the chunk, so the first level of the chunk's reduction tree is in
// the lane, the next five are shuffles and the last two are shuffles between
// the lanes that hold a quad's components: the same pairing as the 256-thread
// tree, with no shared memory and no block barrier inside a phase.  The x
// neighbours come from the neighbouring lanes by shuffle; the y and z rows
// load as float4.  Cells that are not liquid hold zero in d and r, so nothing
// branches per lane.  Two forms, chosen by each block from its chunk count:
//
//   register form   one chunk per warp (up to CG_WARPS chunks): d, r and the
//                   stencil words stay in registers for the whole solve, p, q
//                   and a copy of the neighbours' d in shared memory; only the
//                   neighbours' r is loaded.
//   general form    chunks in turn, {d, r, q, p} of as many half chunks as the
//                   pool holds in shared memory, the rest in global memory.
//
// What bounds it: up to one chunk per warp, the latency of the two exchanges
// (4,000-6,000 cycles each: publication, L2 round trip, skew, trees) and of one L2
// load, then instruction issue (about 300 instructions per warp and phase 1);
// beyond, reads of the L2 (about 20 B per clock and SM) and the same latencies.  Solves of
// 40 / 179 / 200 / 200 iterations on 32^3 / 64^3 / 128^3 (2.0 M particles) /
// 256^3 (18.3 M): 161 / 830 / 1,255 / 5,000 us (ncu, one launch) against 224 / 1,123 / 1,558 /
// 7,197 for the earlier kernel (1,024 threads over listed cells or quads, chunk
// trees from shared memory, every block reading every chunk partial).
//
// Two things to keep: a warp index that the compiler knows to be uniform (the
// shuffle trees took 1,600 cycles instead of 560 without), and no spilled
// registers in the loops (the acquire of exchange B empties the L1, so each
// reload is an L2 round trip: phase 1 took 5,500 cycles instead of 3,000).
//
// Exchange = grid barrier and reduction in one step.  Partials are published
// as 64-bit words {tag, value}; readers poll until every word carries the
// exchange's tag.  No counter, no broadcast: seeing the tags is the barrier,
// and all blocks evaluate the same reduction in the same order.  Tags are
// unique per solve (a per-area epoch advanced by k_cg_plan), so words left by
// earlier solves never match.  Exchange B publishes with release semantics and
// polls with acquire loads: a block's release covers all of its vector writes
// of the update phase and the phase before, which is what the next direction +
// SpMV phase's neighbour loads need.  Exchange A carries only its partials
// (relaxed).
//
// Only 256-cell chunks holding a liquid cell are visited (the rest are zero in
// every vector).  Segment li = active chunks li, li + 256, ... in ascending
// order: the nonzero terms that thread li of cg_reduce_final.wgsl adds in
// sequence (the skipped terms are +0, and acc + 0 == acc for an accumulator
// that starts at +0).  k_cg_plan gives the blocks their chunks once per solve:
//
//   heads and tails  a block owns the first chunks of its segments and
//                    publishes their partial sums; chunks beyond T of a segment
//                    go to other blocks and are published one by one.  Every
//                    block adds the tails to the heads itself: one hop.
//   split segments   (more chunks than that is good for) ranges of equal weight;
//                    all chunk partials are published, a block adds those of its
//                    segments and publishes the sums: two hops.
//
// Every block then evaluates the 256-wide tree of cg_reduce_final.wgsl over the
// segment sums, so in FL_CG_F32 the scalars are the reference's f32 arithmetic
// exactly.  The extended-precision forms publish one float-float or double
// partial per block instead.
#include <cstddef>

#include "fl_device.cuh"

namespace fl {

constexpr int CG_THREADS = 512;
constexpr int CG_WARPS = CG_THREADS / 32;
constexpr uint32_t KCH = 512;            // chunks a block keeps a table of
constexpr uint32_t RAW_MAX = 1024;       // tail partials read by every block
constexpr uint32_t TAG_SPAN_MAX = 1u << 30;
// What the pool leaves of the 228 KB serves as L1 for the neighbours' rows: 140 KB
// against 200 KB and 100 KB on the full-depth 128^3 dam (FL_CG_F64): 2,073, 2,094
// and 2,206 us per solve; 256^3 within 1 %.
constexpr uint32_t POOL_BYTES = 140 * 1024;
constexpr uint32_t HALF_BYTES = 32 * 4 * 16;  // a resident half chunk: float4 d, r, q, p of 32 quads

enum { SLOT_A, SLOT_B, SEG_A, SEG_B, WORD_A, WORD_B };  // exchange areas

struct CgShared {
    // Per half chunk (32 quads, one per lane).  Register form: float4 p and the
    // neighbours' d.  Otherwise: operands of the resident halves, then the
    // stencil words of all (4 B per quad).
    alignas(16) unsigned char pool[POOL_BYTES];
    union {
        alignas(16) float stage[2 * CHUNK];  // partials of two split segments
        float raw[RAW_MAX];                // tail partials
        struct {
            double dpart[CG_THREADS];      // FL_CG_F64_IEEE: thread partials
            float words[2 * MAX_CG_BLOCKS];  // extended forms: the blocks' partials
        };
    };
    uint4 tab[KCH];            // the block's chunks: id, active quads (two masks), first half's index
    float part[KCH];           // chunk partials of one phase
    uint32_t off[CHUNK + 1];   // plan entries of the segments' heads
    uint32_t toff[CHUNK + 1];  // and of their tails
    uint32_t segslot[CHUNK];   // exchange words of the segments, ~0 for an empty one
    float seg[CHUNK];          // segment sums (cg_reduce_final.wgsl thread accumulators)
    float red[2 * CG_THREADS / 32];   // extended forms: warp partials
    float scal[2];             // alpha or beta, and whether the solve is done; broadcast by warp 0
    unsigned long long* area[6];  // exchange areas (see k_cg)
    // Block-uniform values read where they are used: the cell loops are at the
    // 128-register limit of a 512-thread block, and a spilled register costs an
    // L2 round trip after every exchange (the acquire empties the L1).
    uint32_t iters, nh, s0, m, mres, HL, HR, nheads, ah, nact, segline;
    uint64_t limit;            // of every wait, in ns
    float one;                 // 1.0f (see addp2)
    float thr_f;               // f32 stopping threshold on r.r
    float thr_dh, thr_dl;      // FL_CG_F64 stopping threshold on r.r (float-float)
    double rs_d, thr_d;        // FL_CG_F64_IEEE: r.r of the last exchange, stopping threshold
    float rs_hi, rs_lo;        // r.r of the last exchange (rs_old); FL_CG_F32 uses rs_hi
};
static_assert(CG_WARPS * 2 * 6 * 32 * 16 <= POOL_BYTES, "register form: six quads per lane and half in the pool");
static_assert(CG_THREADS == 2 * CHUNK, "split segments: half a block per segment");
static_assert(sizeof(CgShared) <= 227 * 1024, "CG shared memory exceeds the 227 KB per-block limit");

// ---------------------------------------------------------------------------
// Tagged words

__device__ __forceinline__ void st_release_u64(unsigned long long* p, unsigned long long v) {
    asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// The polling loads carry no "memory" clobber, so the compiler may compute
// all of a batch's addresses (shared-memory lookups) before issuing the
// loads; what follows a poll is ordered by data dependence or a barrier.
__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ void st_relaxed_u64(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}
// `rel`: release store, for the exchange after which other blocks read this
// block's vector writes; the other exchange carries only its partials.
__device__ __forceinline__ void publish(unsigned long long* p, uint32_t tag, float v, bool rel) {
    const unsigned long long w = ((unsigned long long)tag << 32) | (unsigned long long)__float_as_uint(v);
    if (rel) st_release_u64(p, w);
    else st_relaxed_u64(p, w);
}
// Polls of an exchange after which the reader loads other blocks' vector
// writes are acquire loads (measured faster than relaxed polls followed by an
// acquire fence in every thread); the other exchange polls relaxed.
__device__ __forceinline__ unsigned long long ld_tag(const unsigned long long* p, bool acq) {
    return acq ? ld_acquire_u64(p) : ld_relaxed_u64(p);
}

// Polls *p until it carries `tag` and returns the word.  Bounded: after `limit`
// ns, or once another block recorded an error, it records FL_TIMEOUT and returns
// a word without the tag.  The clock is read on the first re-poll and then
// every 64 polls (so a limit below one poll's latency expires at the first
// miss); the status word, a global load, every 64 polls only.
__device__ __noinline__ unsigned long long wait_tag(const unsigned long long* p, uint32_t tag, DevStats* st, bool acq,
                                                    const uint64_t* limit) {
    const uint64_t t0 = global_ns();
    for (uint32_t spins = 1;; spins++) {
        const unsigned long long w = ld_tag(p, acq);
        if ((uint32_t)(w >> 32) == tag) return w;
        const bool slow = (spins & 63u) == 0u;
        if (slow && *(volatile uint32_t*)&st->status != 0u) return 0ull;
        if ((slow || spins == 1u) && global_ns() - t0 > *limit) {
            atomicCAS(&st->status, 0u, 5u /* FL_TIMEOUT */);
            return 0ull;
        }
    }
}

// ---------------------------------------------------------------------------
// Reductions

// A block-uniform value read from shared memory at its use (not kept in a register).
template <class T>
__device__ __forceinline__ T vld(const T& x) {
    return *(const volatile T*)&x;
}

// A quad of f32 values as two register pairs, for the packed f32x2
// instructions: each half rounds like the scalar operation, and a phase, which
// is bound by instruction issue, takes half as many.
struct __align__(16) Quad {
    unsigned long long a, b;
};
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(x), "f"(y));
    return v;
}
__device__ __forceinline__ float lo2(unsigned long long v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi2(unsigned long long v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ unsigned long long mul2(unsigned long long x, unsigned long long y) {
    unsigned long long v;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(x), "l"(y));
    return v;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long x, unsigned long long y) {
    unsigned long long v;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(x), "l"(y));
    return v;
}
// prod * one + y with `one` a pair of ones that the assembler cannot see
// through.  An add.rn.f32x2 of a mul.rn.f32x2's result comes out as one fused
// multiply-add (one rounding instead of two), so every product is added with
// this.
__device__ __forceinline__ unsigned long long addp2(unsigned long long prod, unsigned long long one, unsigned long long y) {
    unsigned long long v;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(prod), "l"(one), "l"(y));
    return v;
}
__device__ __forceinline__ Quad qmul(Quad x, Quad y) { return {mul2(x.a, y.a), mul2(x.b, y.b)}; }
__device__ __forceinline__ Quad qadd(Quad x, Quad y) { return {add2(x.a, y.a), add2(x.b, y.b)}; }
__device__ __forceinline__ Quad qaddp(Quad prod, Quad one, Quad y) { return {addp2(prod.a, one.a, y.a), addp2(prod.b, one.a, y.b)}; }
// y - x, by way of -x * one: the same single rounding
__device__ __forceinline__ Quad qsubp(Quad x, Quad one, Quad y) {
    return {addp2(x.a, one.b, y.a), addp2(x.b, one.b, y.b)};
}
__device__ __forceinline__ Quad qall(float x) { return {pack2(x, x), pack2(x, x)}; }
__device__ __forceinline__ Quad quad(float x, float y, float z, float w) { return {pack2(x, y), pack2(z, w)}; }
__device__ __forceinline__ Quad ld_quad(const float* a) { return *reinterpret_cast<const Quad*>(a); }
__device__ __forceinline__ void st_quad(float* a, Quad v) { *reinterpret_cast<Quad*>(a) = v; }

// cg_reduce.wgsl:38-49 over s[0..255], evaluated by one warp: lane l forms the
// level-128 sums of indices l, l+32, l+64, l+96, the level-64 sums of l and
// l+32, the level-32 sum of l, then the shuffle steps 16..1.  Operand
// order and pairing equal the 256-thread tree's.  Valid in lane 0.
__device__ __forceinline__ float tree256(const float* s, uint32_t lane) {
    const float a0 = __fadd_rn(s[lane], s[lane + 128]);
    const float a1 = __fadd_rn(s[lane + 32], s[lane + 160]);
    const float a2 = __fadd_rn(s[lane + 64], s[lane + 192]);
    const float a3 = __fadd_rn(s[lane + 96], s[lane + 224]);
    float v = __fadd_rn(__fadd_rn(a0, a2), __fadd_rn(a1, a3));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}

// The same tree over a chunk whose products sit in the warp's registers: a
// and b are the products of the lane's quads l and l + 32 (tree slots 4l..4l+3
// and 128 + 4l..).  Level 128 adds them; at levels 64 and 32 a lane keeps half
// of its components and hands the partner lane the other half, so that from
// then on it carries one component (2*bit4 + bit3 of the lane) of the quads
// that share its low three bits; levels 16..4 add quads, levels 2 and 1
// components.  f32 addition commutes, so every lane ends with the same bits.
template <bool VEC>
__device__ __forceinline__ float tree256_quads(Quad a, Quad b, Quad one, uint32_t lane) {
    const Quad t = qaddp(a, one, b);
    const float x = lo2(t.a), y = hi2(t.a), z = lo2(t.b), w = hi2(t.b);
    if (!VEC) {  // components 32 apart: levels 64 and 32 in the lane, then the shuffle steps
        float v = __fadd_rn(__fadd_rn(x, z), __fadd_rn(y, w));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
        return v;
    }
    const bool h4 = (lane & 16u) != 0u, h3 = (lane & 8u) != 0u;
    const float u0 = __fadd_rn(h4 ? z : x, __shfl_xor_sync(0xffffffffu, h4 ? x : z, 16));
    const float u1 = __fadd_rn(h4 ? w : y, __shfl_xor_sync(0xffffffffu, h4 ? y : w, 16));
    float v = __fadd_rn(h3 ? u1 : u0, __shfl_xor_sync(0xffffffffu, h3 ? u0 : u1, 8));
    v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 4));
    v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 2));
    v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 1));
    v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 16));
    return __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 8));
}

// Two chunks' trees in one, from their level-128 sums (the products' halves added):
// once a lane holds one component (VEC) or one slot, partner lanes swap, so that half of
// the lanes carry each chunk through the remaining shuffles: 11 instead of 16 (6 instead
// of 10), and one latency for both.  Lane 0 ends with the first chunk's sum, lane
// PAIR_LANE with the second's; the pairs that are added are those of the tree above.
template <bool VEC>
constexpr uint32_t PAIR_LANE = VEC ? 4u : 16u;
template <bool VEC>
__device__ __forceinline__ float tree256_pair(Quad s, Quad t, uint32_t lane) {
    const bool h4 = (lane & 16u) != 0u, h3 = (lane & 8u) != 0u, h2 = (lane & 4u) != 0u;
    auto first = [&](Quad q) {
        const float x = lo2(q.a), y = hi2(q.a), z = lo2(q.b), w = hi2(q.b);
        if (!VEC) return __fadd_rn(__fadd_rn(x, z), __fadd_rn(y, w));
        const float u0 = __fadd_rn(h4 ? z : x, __shfl_xor_sync(0xffffffffu, h4 ? x : z, 16));
        const float u1 = __fadd_rn(h4 ? w : y, __shfl_xor_sync(0xffffffffu, h4 ? y : w, 16));
        return __fadd_rn(h3 ? u1 : u0, __shfl_xor_sync(0xffffffffu, h3 ? u0 : u1, 8));
    };
    const float a = first(s), b = first(t);
    if (!VEC) {
        float v = __fadd_rn(h4 ? b : a, __shfl_xor_sync(0xffffffffu, h4 ? a : b, 16));
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
        return v;
    }
    float v = __fadd_rn(h2 ? b : a, __shfl_xor_sync(0xffffffffu, h2 ? a : b, 4));
    v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 2));
    v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 1));
    v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 16));
    return __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, 8));
}

// Per-thread inner-product accumulator of the extended-precision forms:
// float-float (FL_CG_F64: exact products by two-product, sums by two-sum on
// the FP32 pipe) or IEEE double (FL_CG_F64_IEEE: f32 x f32 products are
// exact in double; sums, trees and combines in double).
template <int PREC>
struct AccT {
    using type = Df;
};
template <>
struct AccT<FL_CG_F64_IEEE> {
    using type = double;
};
__device__ __forceinline__ void acc_add(Df& a, float x, float y) { a = df_acc(a, x, y); }
// f32 x f32 is exact in double, so one fma = the exact product added with one rounding
__device__ __forceinline__ void acc_add(double& a, float x, float y) { a = __fma_rn((double)x, (double)y, a); }
__device__ __forceinline__ double warp_sum_d(double v) {  // result in lane 0
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
// a double's bits in two f32 slots (shared-memory staging and tagged words)
__device__ __forceinline__ float d_lo(double v) { return __int_as_float(__double2loint(v)); }
__device__ __forceinline__ float d_hi(double v) { return __int_as_float(__double2hiint(v)); }
__device__ __forceinline__ double d_of(float lo, float hi) { return __hiloint2double(__float_as_int(hi), __float_as_int(lo)); }

// ---------------------------------------------------------------------------
// Plan

// Plan header (cg_off): the offsets of the segments' heads [CHUNK + 1], tag
// base, form, first plan entry of every block [G + 1], blocks that own chunks,
// blocks that own heads, exchange word of every segment [CHUNK], offsets of the
// tails [CHUNK + 1].
enum { PLAN_F32, PLAN_EXTENDED, PLAN_RANGES };
constexpr uint32_t H_TAG = CHUNK + 1, H_FORM = CHUNK + 2, H_START = CHUNK + 3;

// Words of one owner block among the segment sums of the split form: whole
// 128-byte lines (with the sums of sixteen blocks in a line, the exchange took
// 1,000-2,000 cycles more), at most 16 G + 256 words in all.
__device__ __forceinline__ uint32_t seg_line(uint32_t nact) { return ((CHUNK + nact - 1) / nact + 15u) & ~15u; }

// One block of 256 threads.  Lists the active chunks, gives each block a
// contiguous range of the list, and reserves this solve's tag range.  When the
// 32-bit epoch would wrap, the exchange words are cleared first, so no stale
// word can carry a tag of a later solve.
//
// Heads and tails: a block takes at most T chunks, a multiple of its warps (or
// half of them where that leaves no tails: a small solve with more SMs at work).
// A segment's first T chunks are its head; heads are packed in order, whole;
// what is left of the segments goes to blocks of its own, T chunks each.  The
// smallest T of 32 (one per lane) is taken that needs no more than G blocks and
// leaves at most RAW_MAX tail chunks.  At 128^3 every warp then has one chunk:
// segments of 17 chunks kept whole gave some warps two (1,546 against 1,385 us).
//
// Split segments, when that needs more than one more round of CG_WARPS chunks:
// ranges of equal weight (liquid cells + CHUNK_WEIGHT per chunk) of the list in
// segment order; with at least 9 chunks per block on average no range is empty.
//
// PLAN_EXTENDED (no segment sums) and PLAN_RANGES (solvers that use just the
// ranges, of equal weight) are free to give a block any chunks: they list them in
// tiles of TILE_Y neighbours along y by TILE_Z planes, so that the chunks that a
// block's warps work on at a time share their neighbours' rows in the L1 (reads of
// the L2 are what bounds phase 1).  Against the segment order, whose neighbours
// are 256 chunks apart: FL_CG_F64 1,976 -> 1,890 us on the full-depth 128^3 dam,
// 4,126 -> 3,990 at 256^3, multigrid 1,584 -> 1,555; tiles of 2 x 8 and 8 x 2 give
// the same within 1 %.  Blocks of one chunk per warp (or half of that) where there
// are enough blocks.  For split segments the order was tried at 256^3 alone (5,183 ->
// 5,238 us: a block's partials then belong to many segments), where a plane is 256
// chunks and a segment's neighbours are z neighbours anyway; on other planes, where
// they share nothing, it has not been measured.
__global__ void __launch_bounds__(CHUNK) k_cg_plan(DevBufs b, uint32_t G, int form) {
    after_previous();
    const bool ranges_only = form == PLAN_RANGES;
    const uint32_t per_chunk = ranges_only ? CELL_CHUNK_WEIGHT : CHUNK_WEIGHT;
    __shared__ uint32_t s_wc[CHUNK / 32], s_ww[CHUNK / 32], s_wa[CHUNK / 32], s_wh[CHUNK / 32];
    __shared__ __align__(16) uint32_t s_cnt[CHUNK];
    __shared__ uint32_t s_blk[CHUNK / 2][32];  // blocks of the heads of segments 2i and 2i + 1 under lane l's T
    __shared__ uint16_t s_first[MAX_CG_BLOCKS];
    __shared__ uint32_t s_sel, s_T, s_nblk;
    __shared__ int s_wrap;
    const DevParams& P = *b.prm;
    const uint32_t nchunks = P.nchunks;
    const uint32_t li = threadIdx.x, lane = li & 31, warp = li >> 5;
    uint32_t* hdr = b.cg_off;
    uint32_t* start = hdr + H_START;
    uint32_t* segslot = start + G + 3;
    uint32_t* toffs = segslot + CHUNK;
    const uint32_t epoch = (uint32_t)b.cg_x[0], max_iters = P.iters;  // for the tags, below
    // fn(chunk, liquid cells) for the active chunks of segment li, in order; sixteen
    // loads at a time (one after the other: 19 us more per plan at 256^3).
    auto segment = [&](auto&& fn) {
        for (uint32_t c0 = li; c0 < nchunks; c0 += 16 * CHUNK) {
            uint8_t f[16];
#pragma unroll
            for (uint32_t i = 0; i < 16; i++) f[i] = c0 + i * CHUNK < nchunks ? b.chunk_flag[c0 + i * CHUNK] : (uint8_t)0;
#pragma unroll
            for (uint32_t i = 0; i < 16; i++)
                if (f[i]) fn(c0 + i * CHUNK, (uint32_t)f[i]);
        }
    };
    uint32_t cnt = 0, wsum = 0;
    segment([&](uint32_t, uint32_t f) {
        cnt++;
        wsum += f + per_chunk;
    });
    const uint32_t has = __ballot_sync(0xffffffffu, cnt != 0u);
    auto scan = [&](uint32_t v) {  // inclusive, within the warp
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= (uint32_t)o) v += t;
        }
        return v;
    };
    const uint32_t x = scan(cnt), y = scan(wsum);
    s_cnt[li] = cnt;
    if (lane == 31) {
        s_wc[warp] = x;
        s_ww[warp] = y;
        s_wa[warp] = (uint32_t)__popc(has);
    }
    __syncthreads();
    uint32_t base = 0, A = 0, act = (uint32_t)__popc(has & ((1u << lane) - 1u));
    for (uint32_t w = 0; w < CHUNK / 32; w++) {
        if (w < warp) {
            base += s_wc[w];
            act += s_wa[w];
        }
        A += s_wc[w];
    }
    uint64_t wbase, W;
    weights_of_warps(s_ww, CHUNK / 32, warp, wbase, W);
    if (form == PLAN_F32 && warp == 0) {
        const uint32_t T = lane ? CG_WARPS * lane : CG_WARPS / 2;
        // A chain of an add, a compare and a select per segment: the counts are loaded
        // sixteen at a time and the blocks stored in pairs (with a load, a branch and
        // a store in every step it took 9 us, at any size).
        uint32_t blk = 0xffffffffu, cur = T, tails = 0;
#pragma unroll 1
        for (uint32_t i0 = 0; i0 < (uint32_t)CHUNK; i0 += 16) {
            uint32_t c[16];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint4 v = reinterpret_cast<const uint4*>(s_cnt + i0)[i];
                c[4 * i] = v.x; c[4 * i + 1] = v.y; c[4 * i + 2] = v.z; c[4 * i + 3] = v.w;
            }
            uint32_t pair = 0;
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const uint32_t h = c[i] < T ? c[i] : T, sum = cur + h;
                const bool next = h != 0u && sum > T;
                tails += c[i] - h;
                cur = next ? h : sum;
                blk += next ? 1u : 0u;
                if (i & 1) s_blk[(i0 + i) / 2][lane] = pair | blk << 16;
                else pair = blk & 0xffffu;
            }
        }
        const uint32_t nb = blk + 1u + (tails + T - 1) / T;
        const uint32_t fits = __ballot_sync(0xffffffffu, nb <= G && tails <= (lane ? RAW_MAX : 0u) && T <= KCH);
        const uint32_t sel = fits ? (uint32_t)__ffs(fits) - 1u : 31u;
        if (lane == sel) {
            s_sel = sel;
            s_T = fits ? T : 0u;
            s_nblk = blk + 1u;
        }
    }
    __syncthreads();
    // chunks per block: T of heads and tails, Tq of ranges that give each warp one
    uint32_t Gs = G, T = 0, Tq = 0;
    if (form == PLAN_EXTENDED) {
        Tq = A <= G * (CG_WARPS / 2) ? CG_WARPS / 2 : A <= G * CG_WARPS ? CG_WARPS : 0u;
    } else if (form == PLAN_F32) {
        const uint32_t per = (A + G - 1) / G;
        const uint32_t rounds = (s_T + CG_WARPS - 1) / CG_WARPS;
        if (s_T && rounds <= (per + CG_WARPS - 1) / CG_WARPS + 1) T = s_T;
    }
    if (form != PLAN_RANGES) Gs = A / 9u < 1u ? 1u : (A / 9u < G ? A / 9u : G);
    if (Tq) Gs = A ? (A + Tq - 1) / Tq : 1u;
    // head and tail of segment li, their places in the list
    const uint32_t nh = T && cnt > T ? T : cnt;
    const uint32_t xh = scan(nh);
    if (lane == 31) s_wh[warp] = xh;
    __syncthreads();
    uint32_t hoff = xh - nh, Ah = 0;
    for (uint32_t w = 0; w < CHUNK / 32; w++) {
        if (w < warp) hoff += s_wh[w];
        Ah += s_wh[w];
    }
    const uint32_t toff = base + x - cnt - hoff;
    hdr[li] = hoff;
    if (li == CHUNK - 1) hdr[CHUNK] = hoff + nh;
    const uint32_t nheads = T ? s_nblk : Gs, ntails = T ? (A - Ah + T - 1) / T : 0u;
    const uint32_t nact = A == 0 ? 1u : nheads + ntails;
    if (form == PLAN_F32) {  // in segment order
        uint32_t k = 0;
        if (T) {
            segment([&](uint32_t c, uint32_t) {
                b.cg_chunk[k < nh ? hoff + k : Ah + toff + (k - nh)] = c;
                k++;
            });
        } else {
            RangeSplit split(wbase + (y - wsum), W, Gs);
            segment([&](uint32_t c, uint32_t f) {
                b.cg_chunk[hoff + k] = c;
                k++;
                split.add(f + per_chunk, hoff + k, start);
            });
        }
    } else {  // in tile order
        const ChunkTiles tiles(P.nx, P.ny, nchunks);
        const uint32_t per = (tiles.count + CHUNK - 1) / CHUNK;  // of a thread
        const uint32_t t0 = li * per < tiles.count ? li * per : tiles.count, t1 = t0 + per < tiles.count ? t0 + per : tiles.count;
        auto flags = [&](uint32_t t, uint8_t (&f)[16]) {
#pragma unroll
            for (uint32_t i = 0; i < 16; i++) {
                const uint32_t c = tiles.chunk(t, i);
                f[i] = c < nchunks ? b.chunk_flag[c] : (uint8_t)0;
            }
        };
        uint32_t n = 0, w = 0;
        for (uint32_t t = t0; t < t1; t++) {
            uint8_t f[16];
            flags(t, f);
#pragma unroll
            for (int i = 0; i < 16; i++)
                if (f[i]) {
                    n++;
                    w += f[i] + per_chunk;
                }
        }
        const uint32_t xn = scan(n), xw = scan(w);
        __syncthreads();
        if (lane == 31) {
            s_wc[warp] = xn;
            s_ww[warp] = xw;
        }
        __syncthreads();
        uint32_t e = xn - n;
        for (uint32_t v = 0; v < warp; v++) e += s_wc[v];
        uint64_t wb, all;
        weights_of_warps(s_ww, CHUNK / 32, warp, wb, all);
        RangeSplit split(wb + (xw - w), all, Gs);
        for (uint32_t t = t0; t < t1; t++) {
            uint8_t f[16];
            flags(t, f);
#pragma unroll
            for (uint32_t i = 0; i < 16; i++) {
                if (!f[i]) continue;
                b.cg_chunk[e++] = tiles.chunk(t, i);
                if (!Tq) split.add(f[i] + per_chunk, e, start);
            }
        }
        if (Tq)
            for (uint32_t bb = li; bb <= Gs; bb += CHUNK) start[bb] = bb * Tq < A ? bb * Tq : A;
    }
    // split segments: block li % nact adds segment li
    uint32_t slot = seg_line(nact) * (li % nact) + li / nact;
    if (T && A) {  // each block's words start on a 128-byte line
        auto block_of = [&](uint32_t i) { return s_blk[i / 2][s_sel] >> (16u * (i & 1u)) & 0xffffu; };
        const uint32_t blk = block_of(li);
        if (cnt && (li == 0 || block_of(li - 1) != blk)) {
            s_first[blk] = (uint16_t)act;
            start[blk] = hoff;
        }
        __syncthreads();
        if (cnt) {
            const uint32_t first = s_first[blk];
            slot = 16u * blk + (first & ~15u) + (act - first);
        }
        for (uint32_t t = li; t < ntails; t += CHUNK) start[nheads + t] = Ah + t * T;
    }
    if (li == 0 && (!T || A == 0)) start[0] = 0;
    for (uint32_t bb = nact + li; bb <= G; bb += CHUNK)
        if (T || bb > Gs || A == 0) start[bb] = A;
    if (!ranges_only) {
        segslot[li] = slot;
        toffs[li] = toff;
        if (li == CHUNK - 1) toffs[CHUNK] = A - Ah;
    }
    if (li == 0) {
        hdr[H_FORM] = T ? 1u : 0u;
        if (!ranges_only) {
            start[G + 1] = nact;
            start[G + 2] = nheads;
        }
        const uint32_t span = 2u * (max_iters < TAG_SPAN_MAX ? max_iters : TAG_SPAN_MAX) + 4u;
        uint32_t e0 = epoch;
        int wrap = 0;
        if (e0 > 0xffffffffu - span) {
            wrap = 1;
            e0 = 0;
        }
        b.cg_x[0] = (unsigned long long)(e0 + span);
        hdr[H_TAG] = e0;
        s_wrap = wrap;
    }
    __syncthreads();
    if (s_wrap) {
        const size_t n = cg_x_words(nchunks, G);
        for (size_t i = 1 + li; i < n; i += CHUNK) b.cg_x[i] = 0ull;
    }
}

// ---------------------------------------------------------------------------
// The solve

// VEC: rows are a multiple of four cells and the vectors 16-byte aligned, so a
// quad and its +-y and +-z rows load as float4.  Otherwise a lane's four cells
// of a half are 32 apart, so that its scalar loads are coalesced whatever the
// rows' alignment (consecutive cells made each load touch four times the lines:
// 121 x 112 x 110, 60 iterations, a whole fl_solve_pressure call: 1,520 us
// against 1,289).  Either way component k of a
// lane's quad is the cell at CSTEP * k from its first.
template <int PREC, bool VEC>
__global__ void __launch_bounds__(CG_THREADS, 1) k_cg(DevBufs b) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    CgShared& sh = *reinterpret_cast<CgShared*>(smem_raw);
    // Settings in registers: the L1 is invalidated at every exchange.
    const DevParams& P = *b.prm;
    const uint32_t C = P.C, iters = P.iters < TAG_SPAN_MAX ? P.iters : TAG_SPAN_MAX, nchunks = P.nchunks;
    const uint32_t nx = P.nx, nxy = P.nx * P.ny;  // grids hold at most 2^30 cells
    constexpr uint32_t CSTEP = VEC ? 1u : 32u, LSTEP = VEC ? 4u : 1u;  // between a lane's cells, between lanes
    constexpr bool f64 = PREC != FL_CG_F32;       // no chunk trees: per-thread accumulators
    constexpr bool ieee = PREC == FL_CG_F64_IEEE;
    using Acc = typename AccT<PREC>::type;
    // Stopping test enabled: evaluated once (a double compare in the loop
    // would run on the FP64 pipe in every warp of every iteration).
    const bool stop_on = f64 ? P.tol_sq_d > 0.0 : P.tol_sq > 0.0f;
    DevStats* st = b.st;
    const uint32_t G = gridDim.x, tid = threadIdx.x, lane = tid & 31u;
    const uint32_t warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // known to be uniform
    const uint32_t* hdr = b.cg_off;
    const uint32_t* start = hdr + H_START;
    const uint32_t nact = start[G + 1];
    if (blockIdx.x >= nact) return;  // only blocks that own chunks take part
    float* r = b.r;
    float* p = b.p;
    float* q = b.q;
    const uint16_t* __restrict__ cinfo = b.cinfo;
    const uint32_t s0 = start[blockIdx.x], m = start[blockIdx.x + 1] - s0;  // plan entries [s0, s0 + m)
    const uint32_t* __restrict__ plan = b.cg_chunk + s0;
    const bool whole = hdr[H_FORM] != 0u;  // heads and tails
    const uint32_t tag_base = hdr[H_TAG];
    {
        const uint32_t* segslot = start + G + 3;
        const uint32_t* toffs = segslot + CHUNK;
        for (uint32_t i = tid; i <= (uint32_t)CHUNK; i += CG_THREADS) {
            sh.off[i] = hdr[i];
            sh.toff[i] = toffs[i];
        }
    }
    if (tid < (uint32_t)CHUNK) sh.segslot[tid] = hdr[tid] != hdr[tid + 1] ? start[G + 3 + tid] : 0xffffffffu;
    // Every exchange area starts on a 128-byte line (the pool is 256-byte
    // aligned): a block's line must not share a physical line with a
    // neighbour's (measured 8-11 % of the solve at 128^3 when it did).
    if (tid == 0) {
        const size_t nslot = ((size_t)nchunks + 15) & ~(size_t)15, nseg = 16 * (size_t)G + CHUNK;
        unsigned long long* a = b.cg_x + 16;
        sh.area[SLOT_A] = a;                  // d.q chunk partials: split segments in plan order, or the tails'
        sh.area[SLOT_B] = a += nslot;         // r.r chunk partials
        sh.area[SEG_A] = a += nslot;          // segment sums
        sh.area[SEG_B] = a += nseg;
        sh.area[WORD_A] = a += nseg;          // extended forms: two words of block bb at 16*bb
        sh.area[WORD_B] = a += 16 * (size_t)G;
        sh.iters = iters;
        sh.s0 = s0;
        sh.m = m;
        sh.nheads = start[G + 2];
        sh.ah = hdr[CHUNK];  // plan entries of the heads
        sh.nact = nact;
        sh.segline = seg_line(nact);
        sh.one = 1.0f;
        sh.limit = wait_limit_ns(b.prm);
    }

    // ---- the block's chunks: active quads, stencil words, resident operands
    // Stencil word of the quad at c: bits 0-3 liquid cells, 4-15 the cells'
    // counts of non-solid neighbours.
    auto load_info = [&](uint32_t c) -> uint32_t {
        uint32_t w[4], e = 0;
        if (VEC && c < C) {  // C is a multiple of 4
            const uint2 v = *reinterpret_cast<const uint2*>(cinfo + c);
            w[0] = v.x; w[1] = v.x >> 16; w[2] = v.y; w[3] = v.y >> 16;
        } else {
#pragma unroll
            for (uint32_t k = 0; k < 4; k++) w[k] = c + CSTEP * k < C ? (uint32_t)cinfo[c + CSTEP * k] : 0u;
        }
#pragma unroll
        for (int k = 0; k < 4; k++) e |= (w[k] & 1u) << k | ((w[k] >> 7) & 7u) << (4 + 3 * k);
        return e;
    };
    const uint32_t mc = m < KCH ? m : KCH;
    for (uint32_t j = warp; j < mc; j += CG_WARPS) {
        const uint32_t id = plan[j], c = id * CHUNK + LSTEP * lane;
        const uint32_t lo = __ballot_sync(0xffffffffu, (load_info(c) & 15u) != 0u);
        const uint32_t hi = __ballot_sync(0xffffffffu, (load_info(c + CHUNK / 2) & 15u) != 0u);
        if (lane == 0) sh.tab[j] = make_uint4(id, lo, hi, (lo != 0u) + (hi != 0u));
    }
    __syncthreads();
    if (warp == 0) {
        uint32_t run = 0;
        for (uint32_t j0 = 0; j0 < mc; j0 += 32) {
            const uint32_t n = j0 + lane < mc ? sh.tab[j0 + lane].w : 0u;
            uint32_t x = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= (uint32_t)o) x += t;
            }
            if (j0 + lane < mc) sh.tab[j0 + lane].w = run + x - n;
            run += __shfl_sync(0xffffffffu, x, 31);
        }
        if (lane == 0) sh.nh = run;
    }
    __syncthreads();
    // Register form: one chunk per warp, whose d, r and q stay in registers.
    const bool regs = m <= (uint32_t)CG_WARPS;
    // Halves [0, HR) have their operands in the pool, [0, HL) their stencil words.
    uint32_t HR, HL;
    {
        const uint32_t nh = sh.nh;
        HR = regs ? 0u : nh * (HALF_BYTES + 128u) <= POOL_BYTES ? nh : (nh * 128u < POOL_BYTES ? (POOL_BYTES - nh * 128u) / HALF_BYTES : 0u);
        HL = nh < (POOL_BYTES - HR * HALF_BYTES) / 128u ? nh : (POOL_BYTES - HR * HALF_BYTES) / 128u;
    }
    if (tid == 0) {
        sh.HL = HL;
        sh.HR = HR;
    }
    // The resident arrays: operand k (0 d, 1 r, 2 q, 3 p) of quad i; after them
    // the stencil words of all halves.
    auto op = [&](uint32_t k, uint32_t i) -> Quad& { return reinterpret_cast<Quad*>(sh.pool)[32u * k * HR + i]; };
    auto lst = [&](uint32_t i) -> uint32_t& { return reinterpret_cast<uint32_t*>(sh.pool)[(HALF_BYTES / 4u) * HR + i]; };
    __syncthreads();
    // +1 and -1, which the assembler cannot see through (see addp2)
    const Quad one = {pack2(vld(sh.one), vld(sh.one)), pack2(-vld(sh.one), -vld(sh.one))};
    const uint32_t safe = (nxy + nx) & ~3u;
    const Quad z4 = {0ull, 0ull};
    // A quad of a vector: whole when VEC (cells that are not liquid hold
    // zero), else its liquid cells (p may be a caller's array of any alignment).
    auto ld_q = [&](const float* a, uint32_t c, uint32_t e) -> Quad {
        if (VEC) return (e & 15u) ? ld_quad(a + c) : z4;
        return quad((e & 1u) ? a[c] : 0.0f, (e & 2u) ? a[c + CSTEP] : 0.0f, (e & 4u) ? a[c + 2 * CSTEP] : 0.0f,
                    (e & 8u) ? a[c + 3 * CSTEP] : 0.0f);
    };
    auto st_q = [&](float* a, uint32_t c, uint32_t e, Quad v) {
        if (VEC) {
            if (e & 15u) st_quad(a + c, v);
        } else {
            if (e & 1u) a[c] = lo2(v.a);
            if (e & 2u) a[c + CSTEP] = hi2(v.a);
            if (e & 4u) a[c + 2 * CSTEP] = lo2(v.b);
            if (e & 8u) a[c + 3 * CSTEP] = hi2(v.b);
        }
    };
    // The chunk's halves in the arrays: index of half h's quad of this lane.
    auto slot_of = [&](uint4 t, int h) { return (t.w + (h && t.y ? 1u : 0u)) * 32u + lane; };
    auto ends = [&](uint4 t) { return t.w + (t.y != 0u) + (t.z != 0u); };  // first half past the chunk's
    for (uint32_t j = warp; j < mc && !regs; j += CG_WARPS) {
        const uint4 t = sh.tab[j];
        const uint32_t end = ends(t);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if ((h ? t.z : t.y) == 0u) continue;
            const uint32_t c = t.x * CHUNK + h * (CHUNK / 2) + LSTEP * lane, i = slot_of(t, h);
            const uint32_t e = load_info(c);
            if (end <= HL) lst(i) = e;
            if (end <= HR) {
                op(0, i) = ld_q(b.dA, c, e);
                op(1, i) = ld_q(r, c, e);
                op(2, i) = z4;
                op(3, i) = ld_q(p, c, e);
            }
        }
    }
    {  // chunks [0, mres) have their operands here
        uint32_t lo = 0, hi = mc;  // first chunk that ends past HR (ends grow with j)
        while (lo < hi) {
            const uint32_t mid = (lo + hi) / 2;
            if (ends(sh.tab[mid]) <= HR) lo = mid + 1;
            else hi = mid;
        }
        if (tid == 0) sh.mres = lo;  // visible after the barrier before the loop
    }

    // The lane's two quads of chunk j: first cells (of some interior quad for an
    // inactive one, whose results are masked), stencil words, indices of the
    // resident operands, and whether the warp has an active quad in the half.
    struct Quads {
        uint32_t c[2], i[2], e[2];
        bool any[2];
    };
    auto quads_of = [&](uint32_t j) -> Quads {
        Quads k;
        const bool in = j < KCH;
        const uint4 t = in ? sh.tab[j] : make_uint4(b.cg_chunk[vld(sh.s0) + j], 1u, 1u, 0u);
        const bool listed = in && ends(t) <= vld(sh.HL);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint32_t c = t.x * CHUNK + h * (CHUNK / 2) + LSTEP * lane;
            uint32_t e = 0;
            k.i[h] = slot_of(t, h);
            if (h ? t.z : t.y) e = listed ? lst(k.i[h]) : load_info(c);
            k.any[h] = __any_sync(0xffffffffu, (e & 15u) != 0u);
            k.c[h] = (e & 15u) ? c : safe;
            k.e[h] = e;
        }
        return k;
    };
    // Counts of non-solid neighbours as floats, and the quad with its cells that
    // are not liquid cleared.
    auto counts = [&](uint32_t e) -> Quad {
        return quad((float)((e >> 4) & 7u), (float)((e >> 7) & 7u), (float)((e >> 10) & 7u), (float)((e >> 13) & 7u));
    };
    auto liquid = [&](Quad v, uint32_t e) -> Quad {
        auto m2 = [&](float x, int k) { return (e >> k) & 1u ? x : 0.0f; };
        return quad(m2(lo2(v.a), 0), m2(hi2(v.a), 1), m2(lo2(v.b), 2), m2(hi2(v.b), 3));
    };

    // ---- exchanges
    // The scalars that follow an exchange, from its sum v: post 1 alpha
    // (cg_alpha.wgsl:17-22, sc = rs_old / v), post 2 beta and the stopping test
    // (cg_beta.wgsl:16-30, sc = v / rs_old, dn).  Evaluated once, by lane 0 of
    // warp 0, and broadcast through sh.scal.
    auto post_f32 = [&](int post, float v) {
        const float rs_old = sh.rs_hi;
        float sc = 0.0f;
        bool dn = false;
        if (post == 1) sc = fabsf(v) > 1e-30f ? __fdiv_rn(rs_old, v) : 0.0f;
        if (post != 1) sh.rs_hi = v;  // the initial r.r, or rs_new
        if (post == 2) {
            sc = rs_old > 1e-30f ? __fdiv_rn(v, rs_old) : 0.0f;
            dn = v <= sh.thr_f;
        }
        sh.scal[0] = sc;
        sh.scal[1] = dn ? 1.0f : 0.0f;
    };
    auto wait_word = [&](const unsigned long long* w, uint32_t tag, bool acq, bool& ok) -> float {
        unsigned long long v = ld_tag(w, acq);
        if ((uint32_t)(v >> 32) != tag && ok) {
            v = wait_tag(w, tag, st, acq, &sh.limit);
            ok = (uint32_t)(v >> 32) == tag;
        }
        return __uint_as_float((uint32_t)v);
    };
    // The end of a phase: chunk partials sh.part[0..n) of chunks j0.. are
    // published (split segments).  A release fence comes first where the
    // readers go on to load this block's vectors; the barrier before it orders
    // the other warps' stores.
    auto publish_parts = [&](uint32_t j0, uint32_t n, unsigned long long* slots, uint32_t tag, bool rel) {
        __syncthreads();
        if (warp * 32u < n) {
            if (rel) asm volatile("fence.acq_rel.gpu;" ::: "memory");
            for (uint32_t t = tid; t < n; t += CG_THREADS) publish(slots + vld(sh.s0) + j0 + t, tag, sh.part[t], false);
        }
    };
    // FL_CG_F32: the segment sums of cg_reduce_final.wgsl, then its 256-wide
    // tree and the post scalars by warp 0.  Returns false on abort.
    auto reduce_f32 = [&](unsigned long long* slots, unsigned long long* segw, uint32_t tag, bool acq, int post,
                          float& sc, bool& dn) -> bool {
        bool ok = true;
        if (whole) {
            __syncthreads();  // sh.part is complete, the phase's stores are issued
            const uint32_t ntail = vld(sh.toff[CHUNK]);
            if (tid < (uint32_t)CHUNK) {
                const uint32_t segslot = sh.segslot[tid];
                const uint32_t lo = sh.off[tid], hi = sh.off[tid + 1], s0 = vld(sh.s0);
                const bool mine = segslot != 0xffffffffu && lo >= s0 && lo < s0 + vld(sh.m);
                float s = 0.0f;
                if (mine) {
                    if (acq) asm volatile("fence.acq_rel.gpu;" ::: "memory");
                    // 8 loads first (past the head's end: +0), then the sequential
                    // adds.  s starts at +0 and a sum of floats is -0 only when both
                    // terms are, so s is never -0 and adding +0 leaves it unchanged.
                    for (uint32_t e = lo; e < hi; e += 8) {
                        float v[8];
#pragma unroll
                        for (int k2 = 0; k2 < 8; k2++) v[k2] = e + k2 < hi ? sh.part[e - s0 + k2] : 0.0f;
#pragma unroll
                        for (int k2 = 0; k2 < 8; k2++) s = __fadd_rn(s, v[k2]);
                    }
                    publish(segw + segslot, tag, s, false);
                }
                __syncwarp();  // every word of the warp is out before it waits
                if (!mine && segslot != 0xffffffffu) s = wait_word(segw + segslot, tag, acq, ok);
                sh.seg[tid] = s;
            } else if (ntail) {
                const uint32_t t = tid - CHUNK;
                if (blockIdx.x >= vld(sh.nheads) && warp * 32u < (uint32_t)CHUNK + vld(sh.m)) {
                    if (acq) asm volatile("fence.acq_rel.gpu;" ::: "memory");
                    for (uint32_t j = t; j < vld(sh.m); j += CHUNK)
                        publish(slots + (vld(sh.s0) - vld(sh.ah)) + j, tag, sh.part[j], false);
                }
                __syncwarp();
                unsigned long long w[RAW_MAX / CHUNK];
#pragma unroll
                for (uint32_t k2 = 0; k2 < RAW_MAX / CHUNK; k2++)
                    w[k2] = t + k2 * CHUNK < ntail ? ld_tag(slots + t + k2 * CHUNK, acq) : 0ull;
#pragma unroll
                for (uint32_t k2 = 0; k2 < RAW_MAX / CHUNK; k2++) {
                    const uint32_t i = t + k2 * CHUNK;
                    if (i >= ntail) continue;
                    if ((uint32_t)(w[k2] >> 32) != tag && ok) {
                        w[k2] = wait_tag(slots + i, tag, st, acq, &sh.limit);
                        ok = (uint32_t)(w[k2] >> 32) == tag;
                    }
                    sh.raw[i] = __uint_as_float((uint32_t)w[k2]);
                }
            }
            if (ntail) {  // the tails follow their heads, in order
                __syncthreads();
                if (tid < (uint32_t)CHUNK) {
                    const uint32_t lo = sh.toff[tid], hi = sh.toff[tid + 1];
                    if (lo != hi) {
                        float s = sh.seg[tid];
                        for (uint32_t e = lo; e < hi; e += 8) {
                            float v[8];
#pragma unroll
                            for (int k2 = 0; k2 < 8; k2++) v[k2] = e + k2 < hi ? sh.raw[e + k2] : 0.0f;
#pragma unroll
                            for (int k2 = 0; k2 < 8; k2++) s = __fadd_rn(s, v[k2]);
                        }
                        sh.seg[tid] = s;
                    }
                }
            }
        } else {
            // Block bb adds segments bb, bb + nact, ...: two at a time, a half of the
            // block each, so that a thread waits for one word.  (One warp per segment
            // with eight words per lane waited for up to eight round trips, one after
            // the other: 12,000 cycles per exchange at 256^3 instead of 6,300.)
            const uint32_t half = tid / CHUNK;
            for (uint32_t l0 = blockIdx.x; l0 < (uint32_t)CHUNK; l0 += 2u * vld(sh.nact)) {
                const uint32_t l1 = l0 + vld(sh.nact), li = half ? l1 : l0;
                const uint32_t lo = li < (uint32_t)CHUNK ? sh.off[li] : 0u, hi = li < (uint32_t)CHUNK ? sh.off[li + 1] : 0u;
                const uint32_t n0 = sh.off[l0 + 1] - sh.off[l0], n1 = l1 < (uint32_t)CHUNK ? sh.off[l1 + 1] - sh.off[l1] : 0u;
                float s = 0.0f;
                for (uint32_t e0 = 0; e0 < (n0 > n1 ? n0 : n1); e0 += CHUNK) {
                    const uint32_t e = lo + e0 + (tid & (CHUNK - 1u));
                    sh.stage[tid] = e < hi ? wait_word(slots + e, tag, acq, ok) : 0.0f;
                    __syncthreads();
                    if ((tid & (CHUNK - 1u)) == 0u && lo + e0 < hi) {
                        // cg_reduce_final.wgsl:29-36: in plan order, from +0 (past the end: +0);
                        // the next eight are loaded ahead: the chain is the adds alone
                        const float4* const b4 = reinterpret_cast<const float4*>(sh.stage + tid);
                        const uint32_t n = hi - lo - e0 < (uint32_t)CHUNK ? hi - lo - e0 : CHUNK;
                        float4 u = b4[0], v = b4[1];
                        for (uint32_t j = 0; j < n; j += 8) {
                            const uint32_t jn = j + 8 < (uint32_t)CHUNK ? j / 4 + 2 : 0u;
                            const float4 un = b4[jn], vn = b4[jn + 1];
                            s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, u.x), u.y), u.z), u.w);
                            s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, v.x), v.y), v.z), v.w);
                            u = un;
                            v = vn;
                        }
                    }
                    // a segment whose partials did not all arrive is not published
                    if (__syncthreads_or(!ok)) return false;
                }
                if ((tid & (CHUNK - 1u)) == 0u && lo != hi)
                    publish(segw + vld(sh.segline) * blockIdx.x + li / vld(sh.nact), tag, s, acq);
            }
            __syncwarp();
            const uint32_t segslot = sh.segslot[tid & (CHUNK - 1u)];
            if (tid < (uint32_t)CHUNK) sh.seg[tid] = segslot != 0xffffffffu ? wait_word(segw + segslot, tag, acq, ok) : 0.0f;
        }
        __syncwarp();
        if (__syncthreads_or(!ok)) return false;
        __syncwarp();
        if (warp == 0) {
            const float v = tree256(sh.seg, lane);
            if (lane == 0) post_f32(post, v);
        }
        __syncthreads();
        sc = sh.scal[0];
        dn = sh.scal[1] != 0.0f;
        return true;
    };
    // Extended forms: the blocks' partials (two words of block bb at 16*bb),
    // summed by warp 0 in a fixed order (lanes stride over blocks, then a
    // shuffle tree); lane 0 evaluates the post scalars.
    auto reduce_df = [&](const unsigned long long* words, uint32_t tag, bool acq, int post, float& sc,
                         bool& dn) -> bool {
        bool ok = true;
        for (uint32_t v = tid; v < 2u * nact; v += CG_THREADS)
            sh.words[v] = wait_word(words + (v >> 1) * 16u + (v & 1u), tag, acq, ok);
        if (__syncthreads_or(!ok)) return false;
        if (ieee && warp == 0) {  // the blocks' doubles, in the same fixed order
            double v = 0.0;
            for (uint32_t bb = lane; bb < nact; bb += 32) v += d_of(sh.words[2 * bb], sh.words[2 * bb + 1]);
            v = warp_sum_d(v);
            if (lane == 0) {
                const double rs_old = sh.rs_d;
                float scv = 0.0f;
                bool d2 = false;
                if (post == 1) scv = fabs(v) > 1e-30 ? (float)(rs_old / v) : 0.0f;
                if (post == 2) {
                    scv = rs_old > 1e-30 ? (float)(v / rs_old) : 0.0f;
                    d2 = v <= sh.thr_d;
                    sh.rs_d = v;
                }
                sh.scal[0] = scv;
                sh.scal[1] = d2 ? 1.0f : 0.0f;
            }
        } else if (warp == 0) {
            // a lane's up to MAX_CG_BLOCKS / 32 blocks, loaded first and added in pairs (one
            // after the other, a load and a chain of eleven adds each, the solve took 980
            // instead of 938 us at 64^3)
            Df v[MAX_CG_BLOCKS / 32];
#pragma unroll
            for (uint32_t i = 0; i < MAX_CG_BLOCKS / 32; i++) {
                const uint32_t bb = lane + 32u * i;
                v[i] = bb < nact ? Df{sh.words[2 * bb], sh.words[2 * bb + 1]} : Df{0.0f, 0.0f};
            }
            const Df acc = warp_sum_df(df_tree(v));
            if (lane == 0) {
                const Df rs_old = {sh.rs_hi, sh.rs_lo};
                float scv = 0.0f;
                bool d2 = false;
                if (post == 1) scv = fabsf(acc.hi) > 1e-30f ? df_div(rs_old, acc) : 0.0f;
                if (post == 2) {
                    scv = rs_old.hi > 1e-30f ? df_div(acc, rs_old) : 0.0f;
                    d2 = df_le(acc, Df{sh.thr_dh, sh.thr_dl});
                    sh.rs_hi = acc.hi;
                    sh.rs_lo = acc.lo;
                }
                sh.scal[0] = scv;
                sh.scal[1] = d2 ? 1.0f : 0.0f;
            }
        }
        __syncthreads();
        sc = sh.scal[0];
        dn = sh.scal[1] != 0.0f;
        return true;
    };
    // Block partial published as two tagged words on the block's line: the
    // float-float {hi, lo}, or a double's low and high 32 bits (lanes 0 and 1
    // store in one instruction, so a reader finds both).
    auto publish_df = [&](Acc acc, unsigned long long* words, uint32_t tag, bool rel) {
        if constexpr (ieee) {
            // The FP64 pipe (about 2 lane-operations per clock per SM) is the
            // bound: warp 0 sums the thread partials (lane l: partials l,
            // l + 32, ... in sequence, then a 5-level tree) instead of a tree
            // in every warp.
            sh.dpart[tid] = acc;
            __syncthreads();
            if (warp == 0) {
                double s = 0.0;
                for (uint32_t t2 = lane; t2 < (uint32_t)CG_THREADS; t2 += 32) s += sh.dpart[t2];
                const double v = warp_sum_d(s);
                const float lo = __shfl_sync(0xffffffffu, d_lo(v), 0), hi = __shfl_sync(0xffffffffu, d_hi(v), 0);
                if (lane < 2) publish(words + 16 * blockIdx.x + lane, tag, lane ? hi : lo, rel);
            }
        } else {
            acc = warp_sum_df(acc);
            if (lane == 0) {
                sh.red[2 * warp] = acc.hi;
                sh.red[2 * warp + 1] = acc.lo;
            }
            __syncthreads();
            if (warp == 0) {
                Df v = {0.0f, 0.0f};
                if (lane < CG_WARPS) v = {sh.red[2 * lane], sh.red[2 * lane + 1]};
                v = warp_sum_df<CG_WARPS>(v);
                const float lo = __shfl_sync(0xffffffffu, v.lo, 0);
                if (lane < 2) publish(words + 16 * blockIdx.x + lane, tag, lane ? lo : v.hi, rel);
            }
        }
    };

    // ---- initial residual norm (cg_init.wgsl + cg_reduce of r.r), from the
    // per-chunk partials of all chunks (zero where a chunk holds no liquid)
    float rs_init_f = 0.0f;
    Df rs_init_d = {0.0f, 0.0f};
    if (ieee) {  // the chunks' float-float partials (exact in double), summed in double
        double acc = 0.0;
        for (uint32_t c = tid; c < nchunks; c += CG_THREADS) {
            const float2 v = b.chunk_rr_df[c];
            acc += (double)v.x + (double)v.y;
        }
        sh.dpart[tid] = acc;
        __syncthreads();
        if (warp == 0) {
            double s = 0.0;
            for (uint32_t t2 = lane; t2 < (uint32_t)CG_THREADS; t2 += 32) s += sh.dpart[t2];
            s = warp_sum_d(s);
            if (lane == 0) {
                sh.rs_d = s;
                sh.thr_d = !stop_on ? -1.0 : P.thr_abs ? P.thr_abs_d : P.tol_sq_d * s;  // r.r is never below 0
                if (blockIdx.x == 0) st->rs_init = s;
            }
        }
    } else if (f64) {
        Df acc = {0.0f, 0.0f};
        for (uint32_t c = tid; c < nchunks; c += CG_THREADS) {
            const float2 v = b.chunk_rr_df[c];
            acc = df_add(acc, Df{v.x, v.y});
        }
        acc = warp_sum_df(acc);
        if (lane == 0) {
            sh.red[2 * warp] = acc.hi;
            sh.red[2 * warp + 1] = acc.lo;
        }
        __syncthreads();
        if (warp == 0) {
            Df v = {0.0f, 0.0f};
            if (lane < CG_WARPS) v = {sh.red[2 * lane], sh.red[2 * lane + 1]};
            rs_init_d = warp_sum_df(v);
            // stopping threshold tol^2 * rs_init (or the absolute one), once per solve
            if (lane == 0) {
                sh.rs_hi = rs_init_d.hi;
                sh.rs_lo = rs_init_d.lo;
                const double thr = !stop_on ? -1.0 : P.thr_abs ? P.thr_abs_d : P.tol_sq_d * df_to_double(rs_init_d);
                sh.thr_dh = (float)thr;
                sh.thr_dl = (float)(thr - (double)sh.thr_dh);
                if (blockIdx.x == 0) st->rs_init = df_to_double(rs_init_d);
            }
        }
    } else {
        // thread li of cg_reduce_final.wgsl: partials li, li + 256, ... in order
        if (tid < (uint32_t)CHUNK) {
            float s = 0.0f;
            for (uint32_t c = tid; c < nchunks; c += 16 * CHUNK) {
                float v[16];
#pragma unroll
                for (int k2 = 0; k2 < 16; k2++) v[k2] = c + k2 * CHUNK < nchunks ? b.part_rr[c + k2 * CHUNK] : 0.0f;
#pragma unroll
                for (int k2 = 0; k2 < 16; k2++) s = __fadd_rn(s, v[k2]);
            }
            sh.seg[tid] = s;
        }
        __syncthreads();
        if (warp == 0) {
            rs_init_f = tree256(sh.seg, lane);
            // f32 threshold: tol^2 * rs_init (cg_beta.wgsl:25-30) or the absolute one
            if (lane == 0) {
                sh.rs_hi = rs_init_f;
                sh.thr_f = !stop_on ? -1.0f : P.thr_abs ? P.thr_abs_f : __fmul_rn(P.tol_sq, rs_init_f);
                if (blockIdx.x == 0) st->rs_init = (double)rs_init_f;
            }
        }
    }
    __syncthreads();

    // Shared by both loops: the rows of a quad's neighbours, the sum over its x
    // neighbours (within the quad, the lanes beside, left0 / right31 at the ends
    // of the warp), and the products of a half in the extended forms.
    auto row = [&](const float* a, uint32_t c, uint32_t e) -> Quad {
        if (VEC) return ld_quad(a + c);
        const float* const at = a + (int)c;  // below the array while a later component is inside
        return quad((e & 1u) ? at[0] : 0.0f, (e & 2u) ? at[CSTEP] : 0.0f, (e & 4u) ? at[2 * CSTEP] : 0.0f,
                    (e & 8u) ? at[3 * CSTEP] : 0.0f);
    };
    auto xsum = [&](Quad dq, float left0, float right31) -> Quad {
        const float d0 = lo2(dq.a), d1 = hi2(dq.a), d2 = lo2(dq.b), d3 = hi2(dq.b);
        if (VEC) {
            const float ls = __shfl_up_sync(0xffffffffu, d3, 1), rs = __shfl_down_sync(0xffffffffu, d0, 1);
            const float left = lane == 0 ? left0 : ls, right = lane == 31 ? right31 : rs;
            return quad(__fadd_rn(__fadd_rn(0.0f, left), d1), __fadd_rn(__fadd_rn(0.0f, d0), d2),
                        __fadd_rn(__fadd_rn(0.0f, d1), d3), __fadd_rn(__fadd_rn(0.0f, d2), right));
        }
        const float v[4] = {d0, d1, d2, d3};
        float u[4], d[4], s[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            u[k] = __shfl_sync(0xffffffffu, v[k], (lane + 31u) & 31u);
            d[k] = __shfl_sync(0xffffffffu, v[k], (lane + 1u) & 31u);
        }
#pragma unroll
        for (int k = 0; k < 4; k++)
            s[k] = __fadd_rn(__fadd_rn(0.0f, lane ? u[k] : k ? u[k ? k - 1 : 0] : left0),
                             lane != 31 ? d[k] : k < 3 ? d[k < 3 ? k + 1 : 3] : right31);
        return quad(s[0], s[1], s[2], s[3]);
    };
    // The cell before the chunk (lane 0) or after it (lane 31), if a liquid
    // cell's neighbour.
    auto edge = [&](uint32_t c0, uint32_t e0, uint32_t c1, uint32_t e1) -> uint32_t {
        return lane == 0 && (e0 & 1u) ? c0 - 1u : lane == 31 && (e1 & 8u) ? c1 + 3u * CSTEP + 1u : 0u;
    };
    // x . y of a quad; every lane of the warp calls it.
    auto acc_quad = [&](Acc& a, Quad x, Quad y) {
        const float xs[4] = {lo2(x.a), hi2(x.a), lo2(x.b), hi2(x.b)}, ys[4] = {lo2(y.a), hi2(y.a), lo2(y.b), hi2(y.b)};
        // The FP64 pipe bounds the phases of FL_CG_F64_IEEE, and it takes 16 clocks for a warp
        // whatever number of lanes holds a liquid cell.  With its two conversions per term
        // on that pipe a chunk half full took as long as a full one (128^3 with liquid below
        // x = 0.5: 2,586 us per solve, with the listed cells before 2,482; 191 x 151 x 170:
        // 2,243 and 1,668); converted by integer operations 2,015 and 1,717 (256^3: 5,308
        // against 7,335).  Subnormal, infinite or NaN terms take the instruction.
        if constexpr (ieee) {
            bool plain = true;
#pragma unroll
            for (int k = 0; k < 4; k++) plain = plain && is_plain(xs[k]) && is_plain(ys[k]);
            if (__all_sync(0xffffffffu, plain)) {
#pragma unroll
                for (int k = 0; k < 4; k++) a = __fma_rn(plain_double(xs[k]), plain_double(ys[k]), a);
                return;
            }
        }
#pragma unroll
        for (int k = 0; k < 4; k++) acc_add(a, xs[k], ys[k]);
    };
    // The exchange after a phase: post 1 alpha, post 2 beta and the stopping test.
    // `meanwhile` (extended forms) is done while the words travel.
    auto exchange = [&](Acc (&acc)[2], uint32_t tag, int post, float& sc, bool& dn, auto&& meanwhile) -> bool {
        if constexpr (f64) {
            if constexpr (ieee) acc[0] += acc[1];
            else acc[0] = df_add(acc[0], acc[1]);
            unsigned long long* const w = vld(sh.area[post == 1 ? WORD_A : WORD_B]);
            publish_df(acc[0], w, tag, post == 2);
            __syncwarp();
            meanwhile();
            return reduce_df(w, tag, post == 2, post, sc, dn);
        } else {
            return reduce_f32(vld(sh.area[post == 1 ? SLOT_A : SLOT_B]), vld(sh.area[post == 1 ? SEG_A : SEG_B]), tag,
                              post == 2, post, sc, dn);
        }
    };
    const auto nothing = [] {};

    float beta = 0.0f;  // the first direction is r + 0 * r
    uint32_t it = 0, tag = tag_base;
    if (regs) {
        // One chunk per warp.  A lane keeps its two quads' d, r and stencil words
        // in registers; p, q and the d of the y and z neighbours in shared
        // memory (the latter are advanced here as their owners advance them, so
        // only the neighbours' r is loaded, both halves' rows in flight).
        const bool mine = warp < m;
        uint32_t c[2], e[2];
        Quad dq[2], r4[2];
        Quad* const pool = reinterpret_cast<Quad*>(sh.pool) + (warp * 2u * 6u) * 32u + lane;  // [half][p, 4 rows, q][lane]
        {
            const uint32_t id = mine ? plan[warp] : 0u;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const uint32_t c0 = id * CHUNK + h * (CHUNK / 2) + LSTEP * lane;
                e[h] = mine ? load_info(c0) : 0u;
                c[h] = (e[h] & 15u) ? c0 : safe;
                dq[h] = z4;  // beta is 0 in the first direction
                r4[h] = ld_q(r, c[h], e[h]);
                pool[(h * 6) * 32] = ld_q(p, c[h], e[h]);
                for (int t = 1; t < 6; t++) pool[(h * 6 + t) * 32] = z4;
            }
        }
        const bool any0 = __any_sync(0xffffffffu, (e[0] & 15u) != 0u), any1 = __any_sync(0xffffffffu, (e[1] & 15u) != 0u);
        float de = 0.0f;  // lane 0: d of the cell before the chunk, lane 31: of the one after
#pragma unroll 1
        for (; it < vld(sh.iters); it++) {
            // ---------------- phase 1: direction + SpMV + d.q ----------------
            // No branches per lane: d and r are zero in every cell that is not
            // liquid, and a zero term leaves a sum that starts at +0 unchanged.
            Acc acc[2] = {};
            if (mine) {
                Quad nr[2][4];  // -y, +y, -z, +z
                auto load = [&](int h) {
                    nr[h][0] = row(r, c[h] - nx, e[h]);
                    nr[h][1] = row(r, c[h] + nx, e[h]);
                    nr[h][2] = row(r, c[h] - nxy, e[h]);
                    nr[h][3] = row(r, c[h] + nxy, e[h]);
                };
                if (any0) load(0);
                if (any1) load(1);
                const float re = r[edge(c[0], e[0], c[1], e[1])];
                const Quad beta4 = qall(beta);
                auto dir = [&](Quad dv, Quad rv) { return qaddp(qmul(beta4, dv), one, rv); };  // cg_dir.wgsl:30
                dq[0] = dir(dq[0], r4[0]);
                dq[1] = dir(dq[1], r4[1]);
                float* const d_cur = (it & 1u) ? b.dB : b.dA;
                st_q(d_cur, c[0], e[0], dq[0]);  // for blocks of the other form
                st_q(d_cur, c[1], e[1], dq[1]);
                const float b0 = __shfl_sync(0xffffffffu, hi2(dq[0].b), 31), b1 = __shfl_sync(0xffffffffu, lo2(dq[1].a), 0);
                Quad prod[2] = {z4, z4};
                de = __fadd_rn(re, __fmul_rn(beta, de));
                auto stencil = [&](int h, float left0, float right31) {  // cg_spmv.wgsl:46-68, order -x,+x,-y,+y,-z,+z
                    Quad sum = xsum(dq[h], left0, right31);
#pragma unroll
                    for (int t = 0; t < 4; t++) {
                        Quad& d = pool[(h * 6 + 1 + t) * 32];
                        d = dir(d, nr[h][t]);
                        sum = qadd(sum, d);
                    }
                    const Quad q4 = liquid(qsubp(sum, one, qmul(counts(e[h]), dq[h])), e[h]);
                    pool[(h * 6 + 5) * 32] = q4;
                    if (f64) acc_quad(acc[h], dq[h], q4);
                    else prod[h] = qmul(dq[h], q4);
                };
                if (any0) stencil(0, de, b1);
                if (any1) stencil(1, b0, de);
                if (!f64) {
                    const float v = tree256_quads<VEC>(prod[0], prod[1], one, lane);
                    if (lane == 0) sh.part[warp] = v;
                }
            }
            tag++;
            if (!f64 && !whole) publish_parts(0, vld(sh.m), vld(sh.area[SLOT_A]), tag, false);
            float alpha;
            bool dn;
            if (!exchange(acc, tag, 1, alpha, dn, nothing)) return;
            // ---------------- phase 2: update + r.r (cg_update.wgsl:33-34) ----------------
            acc[0] = Acc{};
            acc[1] = Acc{};
            if (mine) {
                const Quad na4 = qall(-alpha);
                r4[0] = qaddp(qmul(na4, pool[5 * 32]), one, r4[0]);  // r - alpha q = r + (-alpha) q
                r4[1] = qaddp(qmul(na4, pool[11 * 32]), one, r4[1]);
                st_q(r, c[0], e[0], r4[0]);
                st_q(r, c[1], e[1], r4[1]);
                if (f64) {
                    acc_quad(acc[0], r4[0], r4[0]);
                    acc_quad(acc[1], r4[1], r4[1]);
                } else {
                    const float v = tree256_quads<VEC>(qmul(r4[0], r4[0]), qmul(r4[1], r4[1]), one, lane);
                    if (lane == 0) sh.part[warp] = v;
                }
            }
            tag++;
            if (!f64 && !whole) publish_parts(0, vld(sh.m), vld(sh.area[SLOT_B]), tag, true);
            if (mine) {
                const Quad a4 = qall(alpha);
                pool[0] = qaddp(qmul(a4, dq[0]), one, pool[0]);
                pool[6 * 32] = qaddp(qmul(a4, dq[1]), one, pool[6 * 32]);
            }
            if (!exchange(acc, tag, 2, beta, dn, nothing)) return;
            if (dn) {
                it++;
                break;
            }
        }
        if (mine) {
            st_q(p, c[0], e[0], pool[0]);
            st_q(p, c[1], e[1], pool[6 * 32]);
        }
    } else {
        HR = vld(sh.HR);  // not live in the loop above
#pragma unroll 1
        for (; it < vld(sh.iters); it++) {
            float* d_cur = (it & 1u) ? b.dB : b.dA;
            const float* d_src = (it & 1u) || it == 0 ? b.dA : b.dB;
            const Quad beta4 = qall(beta);
            auto dir = [&](Quad dv, Quad rv) { return qaddp(qmul(beta4, dv), one, rv); };  // cg_dir.wgsl:30
            // The warp's chunks of [jb, je), two at a time for their trees (256^3: 5,148 ->
            // 5,066 us; the extended forms have none, and the loop in the loop cost them
            // 1.5 %).
            auto chunks = [&](uint32_t jb, uint32_t je, auto&& phase) {
                if constexpr (f64) {
#pragma unroll 1
                    for (uint32_t j = jb + warp; j < je; j += CG_WARPS) phase(j);
                } else {
#pragma unroll 1
                    for (uint32_t j = jb + warp; j < je; j += 2u * CG_WARPS) {
                        Quad s0 = z4, s1 = z4;
#pragma unroll 1
                        for (uint32_t k = j; k < je && k <= j + CG_WARPS; k += CG_WARPS) {
                            s0 = s1;
                            s1 = phase(k);
                        }
                        const bool two = j + CG_WARPS < je;
                        if (!two) s0 = s1;
                        const float v = tree256_pair<VEC>(s0, s1, lane);
                        if (lane == 0u) sh.part[j - jb] = v;
                        if (two && lane == PAIR_LANE<VEC>) sh.part[j + CG_WARPS - jb] = v;
                    }
                }
            };
            // ---------------- phase 1: direction + SpMV + d.q ----------------
            Acc acc[2] = {};
            tag++;
            auto phase1 = [&](uint32_t j) -> Quad {
                const bool res = __any_sync(0xffffffffu, j < vld(sh.mres));
                const Quads o = quads_of(j);
                // One half's d and r rows in flight at a time (64 registers).
                Quad nd[4], nr[4];
                auto load = [&](int h) {
                    const uint32_t c = o.c[h];
                    const uint32_t off4[4] = {c - nx, c + nx, c - nxy, c + nxy};
#pragma unroll
                    for (int t = 0; t < 4; t++) {
                        nd[t] = row(d_src, off4[t], o.e[h]);
                        nr[t] = row(r, off4[t], o.e[h]);
                    }
                };
                if (o.any[0]) load(0);
                const uint32_t ce = edge(o.c[0], o.e[0], o.c[1], o.e[1]);
                const float de = __fadd_rn(r[ce], __fmul_rn(beta, d_src[ce]));
                Quad dq[2] = {z4, z4}, prod[2] = {z4, z4};
                auto own = [&](int h) {
                    if (res) dq[h] = dir(op(0, o.i[h]), op(1, o.i[h]));
                    else dq[h] = dir(ld_q(d_src, o.c[h], o.e[h]), ld_q(r, o.c[h], o.e[h]));
                };
                if (o.any[0]) own(0);
                if (o.any[1]) own(1);
                const float b0 = __shfl_sync(0xffffffffu, hi2(dq[0].b), 31), b1 = __shfl_sync(0xffffffffu, lo2(dq[1].a), 0);
                auto stencil = [&](int h, float left0, float right31) {
                    Quad sum = xsum(dq[h], left0, right31);
#pragma unroll
                    for (int t = 0; t < 4; t++) sum = qadd(sum, dir(nd[t], nr[t]));
                    const Quad q4 = liquid(qsubp(sum, one, qmul(counts(o.e[h]), dq[h])), o.e[h]);
                    st_q(d_cur, o.c[h], o.e[h], dq[h]);  // the first iteration writes back what is there
                    if (res) {
                        op(0, o.i[h]) = dq[h];
                        op(2, o.i[h]) = q4;
                    } else {
                        st_q(q, o.c[h], o.e[h], q4);
                    }
                    if (f64) acc_quad(acc[h], dq[h], q4);
                    else prod[h] = qmul(dq[h], q4);
                };
                if (o.any[0]) stencil(0, de, b1);
                if (o.any[1]) {
                    load(1);
                    stencil(1, b0, de);
                }
                return f64 ? z4 : qaddp(prod[0], one, prod[1]);  // level 128 of the chunk's tree
            };
#pragma unroll 1
            for (uint32_t jb = 0; jb < vld(sh.m); jb += KCH) {
                const uint32_t je = vld(sh.m) - jb < KCH ? vld(sh.m) : jb + KCH;
                chunks(jb, je, phase1);
                if (!f64 && !whole) {
                    publish_parts(jb, je - jb, vld(sh.area[SLOT_A]), tag, false);
                    if (je < vld(sh.m)) __syncthreads();
                }
            }
            float alpha;
            bool dn;
            if (!exchange(acc, tag, 1, alpha, dn, nothing)) return;
            // ---------------- phase 2: update + r.r (cg_update.wgsl:33-34) ----------------
            acc[0] = Acc{};
            acc[1] = Acc{};
            tag++;
            const Quad a4 = qall(alpha), na4 = qall(-alpha);
            auto phase2 = [&](uint32_t j) -> Quad {
                const bool res = __any_sync(0xffffffffu, j < vld(sh.mres));
                const Quads o = quads_of(j);
                Quad prod[2] = {z4, z4};
                auto update = [&](int h) {
                    const uint32_t c = o.c[h], e = o.e[h], i = o.i[h];
                    Quad q4, r4, d4 = z4, p4 = z4;
                    if (res) {
                        q4 = op(2, i); r4 = op(1, i);
                        if (!f64) { d4 = op(0, i); p4 = op(3, i); }
                    } else {
                        q4 = ld_q(q, c, e); r4 = ld_q(r, c, e);
                        d4 = ld_q(d_cur, c, e); p4 = ld_q(p, c, e);
                    }
                    r4 = qaddp(qmul(na4, q4), one, r4);  // r - alpha q = r + (-alpha) q
                    st_q(r, c, e, r4);
                    if (res) op(1, i) = r4;
                    if (!f64 || !res) {
                        p4 = qaddp(qmul(a4, d4), one, p4);
                        if (res) op(3, i) = p4;
                        else st_q(p, c, e, p4);
                    }
                    if (f64) acc_quad(acc[h], r4, r4);
                    else prod[h] = qmul(r4, r4);
                };
                if (o.any[0]) update(0);
                if (o.any[1]) update(1);
                return f64 ? z4 : qaddp(prod[0], one, prod[1]);  // level 128 of the chunk's tree
            };
#pragma unroll 1
            for (uint32_t jb = 0; jb < vld(sh.m); jb += KCH) {
                const uint32_t je = vld(sh.m) - jb < KCH ? vld(sh.m) : jb + KCH;
                chunks(jb, je, phase2);
                if (!f64 && !whole) {
                    publish_parts(jb, je - jb, vld(sh.area[SLOT_B]), tag, true);
                    if (je < vld(sh.m)) __syncthreads();
                }
            }
            // Extended forms: nothing waits for p, so the resident chunks' is advanced
            // while the words travel (full-depth 128^3 dam: 2,058 -> 1,980 us; the others'
            // loads are in the polls' way: with them 256^3 took 4,432 us, without 4,140, before 4,270).  FL_CG_F32's
            // exchange is busy with the segments (256^3, 5,205 -> 5,317 us).
            auto resident_p = [&] {
#pragma unroll 1
                for (uint32_t j = warp; j < vld(sh.mres); j += CG_WARPS) {
                    const uint4 t = sh.tab[j];
#pragma unroll
                    for (int h = 0; h < 2; h++)
                        if (h ? t.z : t.y) {
                            const uint32_t i = slot_of(t, h);
                            op(3, i) = qaddp(qmul(a4, op(0, i)), one, op(3, i));
                        }
                }
            };
            if (!exchange(acc, tag, 2, beta, dn, resident_p)) return;
            if (dn) {
                it++;
                break;
            }
        }
    }
    // the resident pressure, once
    HR = vld(sh.HR);
    for (uint32_t j = warp; j < vld(sh.mres); j += CG_WARPS) {
        const Quads o = quads_of(j);
#pragma unroll
        for (int h = 0; h < 2; h++)
            if (o.any[h]) st_q(p, o.c[h], o.e[h], op(3, o.i[h]));
    }
    if (blockIdx.x == 0 && tid == 0) {
        st->cg_iters = it;
        st->rs_final = ieee ? sh.rs_d : (f64 ? df_to_double(Df{sh.rs_hi, sh.rs_lo}) : (double)sh.rs_hi);
    }
}

typedef void (*CgKernel)(DevBufs);
static CgKernel cg_kernel(uint32_t precision, bool vec) {
    switch (precision) {
        case FL_CG_F64: return vec ? k_cg<FL_CG_F64, true> : k_cg<FL_CG_F64, false>;
        case FL_CG_F64_IEEE: return vec ? k_cg<FL_CG_F64_IEEE, true> : k_cg<FL_CG_F64_IEEE, false>;
        default: return vec ? k_cg<FL_CG_F32, true> : k_cg<FL_CG_F32, false>;
    }
}

int cg_max_blocks_per_sm() {
    int lo = 1 << 30;
    for (int i = 0; i < 6; i++) {
        const void* f = (const void*)cg_kernel((uint32_t)i / 2, i & 1);
        int n = 0;
        if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(CgShared)) != cudaSuccess)
            return 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, f, CG_THREADS, sizeof(CgShared)) != cudaSuccess) return 0;
        lo = n < lo ? n : lo;
    }
    return lo;
}

cudaError_t launch_cg_plan(const DevBufs& b, uint32_t G, cudaStream_t s) {
    if (G < 1 || G > MAX_CG_BLOCKS) return cudaErrorInvalidValue;
    launch_after(k_cg_plan, dim3(1), CHUNK, s, b, G, PLAN_RANGES);
    return cudaGetLastError();
}

cudaError_t launch_cg(const DevBufs& b, const LaunchCfg& L, cudaStream_t s, uint32_t precision, uint32_t nx) {
    if (precision > FL_CG_F64_IEEE) return cudaErrorInvalidValue;
    if (L.cg_blocks < 1 || (uint32_t)L.cg_blocks > MAX_CG_BLOCKS) return cudaErrorInvalidValue;
    launch_after(k_cg_plan, dim3(1), CHUNK, s, b, (uint32_t)L.cg_blocks, precision == FL_CG_F32 ? PLAN_F32 : PLAN_EXTENDED);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(L.cg_blocks);
    cfg.blockDim = dim3(CG_THREADS);
    cfg.dynamicSmemBytes = sizeof(CgShared);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const bool vec = (nx & 3u) == 0u && (((uintptr_t)b.p | (uintptr_t)b.r | (uintptr_t)b.q | (uintptr_t)b.dA |
                                          (uintptr_t)b.dB) & 15u) == 0u;
    return cudaLaunchKernelEx(&cfg, cg_kernel(precision, vec), b);
}

}  // namespace fl
