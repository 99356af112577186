"""Float-float sums (csrc/fl_df.cuh, the header that the kernels compile) on the host's
C++ compiler: accumulated products and a tree of 32 accumulators lose no more than
Dekker's normalised additions one after the other do, against exact sums, for terms of
one sign and of both.  The conversion to double by integer operations is exact."""
import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fluid-simulation_gb300", "csrc")

SHIM = r"""
#include <cmath>
#include <cstring>
#define __device__
#define __forceinline__ inline
static float __fadd_rn(float a, float b) { return a + b; }
static float __fsub_rn(float a, float b) { return a - b; }
static float __fmul_rn(float a, float b) { return a * b; }
static float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
static unsigned __float_as_uint(float x) { unsigned b; std::memcpy(&b, &x, 4); return b; }
static double __hiloint2double(int hi, int lo) {
    const unsigned long long b = (unsigned long long)(unsigned)hi << 32 | (unsigned)lo;
    double d;
    std::memcpy(&d, &b, 8);
    return d;
}
#include "fl_df.cuh"
using namespace fl;
// Dekker 1971 with Knuth's two-sum: every sum normalised
static Df dekker(Df a, Df b) {
    const float s = a.hi + b.hi, t = s - a.hi, e = ((a.hi - (s - t)) + (b.hi - t)) + (a.lo + b.lo), h = s + e;
    return {h, e - (h - s)};
}
// x, y: [32][n]; out[0]: as the kernels do, out[1]: one after the other
extern "C" void dots(const float* x, const float* y, int n, Df* out) {
    Df a[32], b[32], all = {0.0f, 0.0f};
    for (int l = 0; l < 32; l++) {
        a[l] = b[l] = {0.0f, 0.0f};
        const float *p = x + l * n, *q = y + l * n;
        for (int j = 0; j < n; j++) {
            const float r = p[j] * q[j];
            a[l] = df_acc(a[l], p[j], q[j]);
            b[l] = dekker(b[l], {r, std::fma(p[j], q[j], -r)});
        }
        all = dekker(all, b[l]);
    }
    out[0] = df_tree(a);
    out[1] = all;
}
"""


SHIM += r"""
extern "C" void doubles(const float* x, int n, unsigned char* plain, double* out) {
    for (int i = 0; i < n; i++) {
        plain[i] = is_plain(x[i]);
        out[i] = plain_double(x[i]);
    }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("df")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run(["g++", "-O1", "-ffp-contract=off", "-std=c++17", "-shared", "-fPIC", "-I" + CSRC, str(d / "shim.cpp"),
                    "-o", str(d / "shim.so")], check=True)
    return ctypes.CDLL(str(d / "shim.so"))


def exact(values):
    return sum((Fraction(float(v)) for v in values), Fraction(0))


@pytest.mark.parametrize("n", [4, 8, 32, 64])
@pytest.mark.parametrize("signs", ["one", "both", "mostly one"])
def test_no_less_exact_than_one_by_one(lib, n, signs):
    rng = np.random.default_rng(n)
    squares = np.zeros(2)
    for _ in range(200):
        x = rng.standard_normal((32, n)).astype(np.float32)
        y = {"one": x, "both": rng.standard_normal((32, n)), "mostly one": x * (0.3 + rng.standard_normal((32, n)))}[signs]
        y = np.ascontiguousarray(y, np.float32)
        out = np.zeros((2, 2), np.float32)
        lib.dots(ctypes.c_void_p(x.ctypes.data), ctypes.c_void_p(y.ctypes.data), n, ctypes.c_void_p(out.ctypes.data))
        terms = (x.astype(np.float64) * y.astype(np.float64)).ravel()  # exact
        want, size = exact(terms), np.abs(terms).sum()
        err = np.array([float(exact(o) - want) / size for o in out])
        assert abs(err[0]) <= 3 * 2.0**-48 * (n + 5)  # at most that of its operands per addition, n + 5 in a row
        squares += err**2
    assert squares[0] <= squares[1]


def test_conversion_to_double(lib):
    rng = np.random.default_rng(1)
    mant = np.concatenate([[0, 1, 2, 2**22, 2**23 - 1], rng.integers(0, 2**23, 40)]).astype(np.uint32)
    bits = (np.arange(512, dtype=np.uint32)[:, None] << np.uint32(23)) | mant  # every sign and exponent
    x = np.ascontiguousarray(bits.ravel()).view(np.float32)
    plain, out = np.zeros(x.size, np.uint8), np.zeros(x.size)
    lib.doubles(ctypes.c_void_p(x.ctypes.data), x.size, ctypes.c_void_p(plain.ctypes.data), ctypes.c_void_p(out.ctypes.data))
    normal = np.isfinite(x) & ((x == 0) | (np.abs(x) >= np.finfo(np.float32).tiny))
    assert np.array_equal(plain.astype(bool), normal)
    assert np.array_equal(out[normal].view(np.uint64), x[normal].astype(np.float64).view(np.uint64))
