// fl_relax.cu — the reference's relaxation solvers for the pressure system,
// as CUDA kernels (fl_relax_pressure):
//
//   k_jacobi  sim/pressure.rs:72-117 jacobi_iteration: one sweep from p_in to
//             p_out over all cells; non-liquid cells get 0; air neighbours
//             count toward n (Dirichlet p = 0), solid ones are excluded
//             (Neumann).  jacobi_solve (:120-136) ping-pongs from zero.
//   k_rbgs    pressure.wgsl:26-61: the same update in place for the cells of
//             one colour (i+j+k)&1; non-liquid cells are not written (zero
//             from the start).  One iteration = red phase, then black.
//
//   k_relax   either, all sweeps in one cooperative launch, for grids whose cells
//             fit the blocks' lists
//
// All evaluate (sum - scale*div) / n in f32 with the neighbours in the order
// -x, +x, -y, +y, -z, +z, like the reference (no contraction: --fmad=false).
#include "fl_device.cuh"

namespace fl {

namespace {

__device__ __forceinline__ float relax_cell(const uint8_t* ct, const float* div, float scale, const float* p,
                                            uint32_t c, uint32_t nx, uint32_t nxy) {
    const uint32_t nb[6] = {c - 1, c + 1, c - nx, c + nx, c - nxy, c + nxy};
    float sum = 0.0f, n = 0.0f;
#pragma unroll
    for (int s = 0; s < 6; s++) {
        const uint8_t t = ct[nb[s]];
        if (t == CELL_SOLID) continue;
        if (t == CELL_LIQUID) sum = __fadd_rn(sum, p[nb[s]]);
        n = __fadd_rn(n, 1.0f);
    }
    return n > 0.0f ? __fdiv_rn(__fsub_rn(sum, __fmul_rn(scale, div[c])), n) : 0.0f;
}

__global__ void __launch_bounds__(256) k_jacobi(const uint8_t* __restrict__ ct, const float* __restrict__ div,
                                                float scale, const float* __restrict__ p_in,
                                                float* __restrict__ p_out, uint32_t nx, uint32_t ny, uint32_t C) {
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    // liquid cells are interior (the boundary layer is solid): neighbours exist
    p_out[c] = ct[c] == CELL_LIQUID ? relax_cell(ct, div, scale, p_in, c, nx, nx * ny) : 0.0f;
}

__global__ void __launch_bounds__(256) k_rbgs(const uint8_t* __restrict__ ct, const float* __restrict__ div,
                                              float scale, float* p, uint32_t nx, uint32_t ny, uint32_t C,
                                              uint32_t phase) {
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C || ct[c] != CELL_LIQUID) return;
    const uint32_t i = c % nx, j = (c / nx) % ny, k = c / (nx * ny);
    if (((i + j + k) & 1u) != phase) return;
    p[c] = relax_cell(ct, div, scale, p, c, nx, nx * ny);
}

// One launch for all sweeps.  A sweep of a grid of this size is a few hundred
// loads deep in latency and nothing else: as a kernel of its own it took 6.4 us
// at 64^3 (types, then each neighbour's type, then its value, half the threads
// of the other colour).  Here every block lists its liquid cells by colour once
// (place, neighbours, right-hand side: 10 B of shared memory each), so a sweep
// is six loads in flight per cell and a grid barrier: 2.1 us.  Cells are dealt
// out in groups of 32, so blocks get equal numbers of liquid ones.
constexpr uint32_t RELAX_CELLS = 20480;  // per block
constexpr int RELAX_THREADS = 1024;
// Grids below num_sms times this take fewer blocks, so that a barrier has fewer to wait
// for; a cell per thread measures best (red-black, per sweep: 2,048 cells 4.7 us at 48^3
// and 5.3 at 60^3, 1,024 4.1 and 4.7; more than twice that at 8,192).
constexpr uint32_t RELAX_PER_BLOCK = 1024;
constexpr uint32_t RELAX_SWEEPS = 8192;     // per launch; even: the next one starts in pa again

struct RelaxShared {
    uint32_t cell[RELAX_CELLS];
    float rhs[RELAX_CELLS];      // scale * div
    uint16_t info[RELAX_CELLS];  // liquid neighbours (bits 0-5), number of non-solid ones (bits 6-8)
    uint32_t wc[2][RELAX_THREADS / 32];
    int ok;
};

template <bool JACOBI>
__global__ void __launch_bounds__(RELAX_THREADS, 1) k_relax(const uint8_t* __restrict__ ct, const float* __restrict__ div,
                                                             float scale, float* pa, float* pb, uint32_t* bars, uint32_t nx,
                                                             uint32_t ny, uint32_t C, uint32_t iters, uint64_t wait_ns) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    RelaxShared& sh = *reinterpret_cast<RelaxShared*>(smem_raw);
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nxy = nx * ny;
    const uint32_t groups = (C + 31) / 32;
    uint32_t n0 = 0, n1 = 0;  // listed cells: red (or all) from the front, black from the back
    for (uint32_t g0 = 0; g0 * gridDim.x < groups; g0 += RELAX_THREADS / 32) {
        const uint32_t c = ((g0 + warp) * gridDim.x + blockIdx.x) * 32u + lane;
        const bool liquid = c < C && ct[c] == CELL_LIQUID;
        uint32_t info = 0, black = 0;
        float rhs = 0.0f;
        if (liquid) {  // interior (the boundary layer is solid): neighbours exist
            const uint32_t nb[6] = {c - 1, c + 1, c - nx, c + nx, c - nxy, c + nxy};
            uint8_t t[6];
#pragma unroll
            for (int s = 0; s < 6; s++) t[s] = ct[nb[s]];
            rhs = __fmul_rn(scale, div[c]);
#pragma unroll
            for (int s = 0; s < 6; s++) info += (t[s] == CELL_LIQUID ? 1u << s : 0u) + (t[s] != CELL_SOLID ? 64u : 0u);
            if (!JACOBI) black = (c % nx + (c / nx) % ny + c / nxy) & 1u;
        }
        const uint32_t m0 = __ballot_sync(0xffffffffu, liquid && !black), m1 = __ballot_sync(0xffffffffu, liquid && black);
        if (lane == 0) {
            sh.wc[0][warp] = (uint32_t)__popc(m0);
            sh.wc[1][warp] = (uint32_t)__popc(m1);
        }
        __syncthreads();
        uint32_t before[2] = {0, 0}, all[2] = {0, 0};
        for (uint32_t w = 0; w < RELAX_THREADS / 32; w++)
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const uint32_t v = sh.wc[k][w];
                before[k] += w < warp ? v : 0u;
                all[k] += v;
            }
        __syncthreads();
        if (liquid) {
            const uint32_t e = (black ? n1 + before[1] : n0 + before[0]) + (uint32_t)__popc((black ? m1 : m0) & ((1u << lane) - 1u));
            const uint32_t at = black ? RELAX_CELLS - 1 - e : e;
            sh.cell[at] = c;
            sh.rhs[at] = rhs;
            sh.info[at] = (uint16_t)info;
        }
        n0 += all[0];
        n1 += all[1];
    }
    __syncthreads();
    uint32_t epoch = 0;
    for (uint32_t it = 0; it < iters; it++) {
#pragma unroll
        for (uint32_t colour = 0; colour < (JACOBI ? 1u : 2u); colour++) {
            const float* const in = JACOBI && (it & 1u) ? pb : pa;
            float* const out = JACOBI ? ((it & 1u) ? pa : pb) : pa;
            for (uint32_t e = threadIdx.x; e < (colour ? n1 : n0); e += RELAX_THREADS) {
                const uint32_t at = colour ? RELAX_CELLS - 1 - e : e;
                const uint32_t c = sh.cell[at], info = sh.info[at];
                const uint32_t nb[6] = {c - 1, c + 1, c - nx, c + nx, c - nxy, c + nxy};
                float v[6];
#pragma unroll
                for (int s = 0; s < 6; s++) v[s] = ld_if(in + nb[s], (info >> s) & 1u);
                // the reference's order; a term of +0 (not liquid) changes nothing
                float sum = 0.0f;
#pragma unroll
                for (int s = 0; s < 6; s++) sum = __fadd_rn(sum, v[s]);
                const uint32_t cnt = info >> 6;
                out[c] = cnt ? __fdiv_rn(__fsub_rn(sum, sh.rhs[at]), (float)cnt) : 0.0f;
            }
            if (it + 1 == iters && (JACOBI || colour == 1u)) return;
            if (!grid_barrier(bars, ++epoch, wait_ns, bars + BAR_BYTES / 4, &sh.ok)) return;
        }
    }
}

}  // namespace

cudaError_t solve_relax(const uint8_t* ct, const float* div, float scale, float* pa, float* pb, uint32_t* bars,
                        uint32_t nx, uint32_t ny, uint32_t nz, uint32_t method, uint32_t iters, int num_sms,
                        uint64_t wait_ns, cudaStream_t s, float** result) {
    const uint32_t C = nx * ny * nz, grid = (C + 255) / 256;
    if (iters && (uint64_t)C + 32ull * num_sms <= (uint64_t)RELAX_CELLS * num_sms) {
        const bool jacobi = method == 0u;
        const uint32_t want = (C + RELAX_PER_BLOCK - 1) / RELAX_PER_BLOCK;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(want < (uint32_t)num_sms ? want : (uint32_t)num_sms);
        cfg.blockDim = dim3(RELAX_THREADS);
        cfg.dynamicSmemBytes = sizeof(RelaxShared);
        cfg.stream = s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        auto* const f = jacobi ? k_relax<true> : k_relax<false>;
        cudaError_t e = cudaFuncSetAttribute((const void*)f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(RelaxShared));
        for (uint32_t done = 0; e == cudaSuccess && done < iters; done += RELAX_SWEEPS) {
            if (done) e = cudaMemsetAsync(bars, 0, BAR_BYTES, s);
            const uint32_t now = iters - done < RELAX_SWEEPS ? iters - done : RELAX_SWEEPS;
            if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, f, ct, div, scale, pa, pb, bars, nx, ny, C, now, wait_ns);
        }
        uint32_t status = 0;
        if (e == cudaSuccess) e = cudaMemcpyAsync(&status, bars + BAR_BYTES / 4, 4, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        *result = jacobi && (iters & 1u) ? pb : pa;
        if (e == cudaErrorCooperativeLaunchTooLarge) (void)cudaGetLastError();
        else if (e != cudaSuccess || status == 0) return e;
        // The blocks cannot all be resident, or one waited too long for another (a GPU
        // shared with other work): a launch per sweep needs neither.
        if ((e = cudaMemsetAsync(pa, 0, 4 * (size_t)C, s)) != cudaSuccess) return e;
        if ((e = cudaMemsetAsync(pb, 0, 4 * (size_t)C, s)) != cudaSuccess) return e;
    }
    float* cur = pa;
    for (uint32_t it = 0; it < iters; it++) {
        if (method == 0u) {
            float* nxt = cur == pa ? pb : pa;
            k_jacobi<<<grid, 256, 0, s>>>(ct, div, scale, cur, nxt, nx, ny, C);
            cur = nxt;
        } else {
            k_rbgs<<<grid, 256, 0, s>>>(ct, div, scale, cur, nx, ny, C, 0u);
            k_rbgs<<<grid, 256, 0, s>>>(ct, div, scale, cur, nx, ny, C, 1u);
        }
    }
    *result = cur;
    return cudaGetLastError();
}

}  // namespace fl
