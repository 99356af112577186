"""The one-launch relaxation solve (csrc/fl_relax.cu) when a wait of its grid barrier
runs out: it ends, and a launch per sweep gives the same answer.  The limit is no
argument of fl_relax_pressure, so the test compiles the source with a caller of its
own.  Nothing traps or hangs: the expiry is an ordinary return path."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from fluidgb import FL_RELAX_JACOBI, FL_RELAX_RBGS

from test_gpu_relax_sizes import random_field

pytestmark = pytest.mark.gpu

CALLER = r"""
#include "fl_relax.cu"
using namespace fl;
// returns the CUDA error, or 1000 + the status word
extern "C" int relax(const uint8_t* ct, const float* div, float scale, uint32_t nx, uint32_t ny, uint32_t nz, uint32_t method,
                     uint32_t iters, uint64_t wait_ns, float* out) {
    const size_t C = (size_t)nx * ny * nz;
    uint8_t* dct = nullptr;
    float *ddiv = nullptr, *pa = nullptr, *pb = nullptr, *res = nullptr;
    uint32_t *bars = nullptr, status = 0;
    int sms = 0;
    cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, 0);
    if (!e) e = cudaMalloc(&dct, C);
    if (!e) e = cudaMalloc(&ddiv, 4 * C);
    if (!e) e = cudaMalloc(&pa, 4 * C);
    if (!e) e = cudaMalloc(&pb, 4 * C);
    if (!e) e = cudaMalloc(&bars, BAR_BYTES + 4);
    if (!e) e = cudaMemset(pa, 0, 4 * C);
    if (!e) e = cudaMemset(pb, 0, 4 * C);
    if (!e) e = cudaMemset(bars, 0, BAR_BYTES + 4);
    if (!e) e = cudaMemcpy(dct, ct, C, cudaMemcpyHostToDevice);
    if (!e) e = cudaMemcpy(ddiv, div, 4 * C, cudaMemcpyHostToDevice);
    if (!e) e = solve_relax(dct, ddiv, scale, pa, pb, bars, nx, ny, nz, method, iters, sms, wait_ns, 0, &res);
    if (!e) e = cudaMemcpy(out, res, 4 * C, cudaMemcpyDeviceToHost);
    if (!e) e = cudaMemcpy(&status, bars + BAR_BYTES / 4, 4, cudaMemcpyDeviceToHost);
    cudaFree(dct); cudaFree(ddiv); cudaFree(pa); cudaFree(pb); cudaFree(bars);
    return e ? (int)e : 1000 + (int)status;
}
"""


@pytest.fixture(scope="module")
def caller(tmp_path_factory):
    from fluidgb import build
    d = tmp_path_factory.mktemp("relax")
    (d / "caller.cu").write_text(CALLER)
    subprocess.run([build.nvcc()] + build.ARCH + build.NVCC_FLAGS + ["-shared", "-cudart", "static", str(d / "caller.cu"), "-o",
                                                                    str(d / "caller.so")], check=True)
    return ctypes.CDLL(str(d / "caller.so"))


@pytest.mark.parametrize("method", [FL_RELAX_JACOBI, FL_RELAX_RBGS])
@pytest.mark.parametrize("wait_ns,status", [(2000000000, 0), (1, 5)])
def test_an_expired_wait_is_solved_by_plain_launches(oracle, caller, method, wait_ns, status):
    dims, iters, scale = (64, 60, 66), 7, np.float32(0.5 * 0.5 / 0.25)
    ct, div = random_field(dims, 4)
    out = np.empty(ct.size, np.float32)
    got = caller.relax(ctypes.c_void_p(ct.ctypes.data), ctypes.c_void_p(div.ctypes.data), ctypes.c_float(scale), *dims, method, iters,
                       ctypes.c_uint64(wait_ns), ctypes.c_void_p(out.ctypes.data))
    assert got == 1000 + status
    ref = oracle.ref_jacobi_solve if method == FL_RELAX_JACOBI else oracle.ref_rbgs_solve
    assert np.array_equal(out, ref(dims, 0.5, 1.0, 0.25, ct, div, iters))
