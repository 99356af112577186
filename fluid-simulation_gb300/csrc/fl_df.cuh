// fl_df.cuh — float-float sums and products, exact conversion to double.
//
// Float-float ("double-single") arithmetic: a value is hi + lo with two f32,
// |lo| <= ulp(hi)/2, about 48 significand bits.  GB300's FP64 pipe has a
// dependent-op latency of ~64 cycles for one warp and ~600 with a full SM
// issuing (DDIV ~640 for one warp), so the FL_CG_F64 inner products, residual
// norms and stopping test are carried in float-float on the FP32 pipe
// (df_add: ~32 cycles dependent latency) and converted to double only for the
// statistics.  Products use the exact two-product (fmaf), sums the two-sum.
// df_add rounds only among the low parts: its error is a few 2^-48 of |a| + |b|, also
// where the high parts cancel and its last step, exact while |s| >= |e|, rounds too.
#pragma once

namespace fl {

struct Df {
    float hi, lo;
};
__device__ __forceinline__ Df df_add(Df a, Df b) {
    const float s = __fadd_rn(a.hi, b.hi);
    const float bb = __fsub_rn(s, a.hi);
    float e = __fadd_rn(__fsub_rn(a.hi, __fsub_rn(s, bb)), __fsub_rn(b.hi, bb));
    e = __fadd_rn(e, __fadd_rn(a.lo, b.lo));
    const float hi = __fadd_rn(s, e);
    return {hi, __fsub_rn(e, __fsub_rn(hi, s))};
}
__device__ __forceinline__ Df df_prod(float x, float y) {
    const float p = __fmul_rn(x, y);
    return {p, __fmaf_rn(x, y, -p)};
}
// Sum of N values (a power of two), i with i + N/2 and so on: in pairs the adds do not
// wait for one another, and the rounding errors are those of log2 N of them.
template <int N>
__device__ __forceinline__ Df df_tree(Df (&v)[N]) {
#pragma unroll
    for (int w = N / 2; w > 0; w /= 2)
#pragma unroll
        for (int i = 0; i < w; i++) v[i] = df_add(v[i], v[i + w]);
    return v[0];
}
// a + x y.  (Left unnormalised within four products and within a tree, the sums of
// FL_CG_F64 were up to 1.4 times as far from exact ones; normalised the solve of the
// full-depth 128^3 dam takes 1,849 us instead of 1,757.)
__device__ __forceinline__ Df df_acc(Df a, float x, float y) { return df_add(a, df_prod(x, y)); }

// (double)x by integer operations, for x zero or normal (is_plain): sign, exponent and
// mantissa moved to their places, the exponent's bias raised by 896.  The conversion
// instruction shares the FP64 pipe, two lanes per clock and SM.
__device__ __forceinline__ bool is_plain(float x) {
    const unsigned a = __float_as_uint(x) & 0x7fffffffu;
    return a == 0u || a - 0x00800000u < 0x7f000000u;
}
__device__ __forceinline__ double plain_double(float x) {
    const unsigned b = __float_as_uint(x), hi = (unsigned)((int)b >> 3) & 0x8fffffffu;
    return __hiloint2double((int)(hi + (b << 1 ? 0x38000000u : 0u)), (int)(b << 29));
}

}  // namespace fl
