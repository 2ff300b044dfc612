// ct_fastmath.cuh — short forms of e^x, square root and division, each with the error bound that its callers
// count on.
//
// u = 2^-24.  The two approximate instructions are taken at their documented bounds: ex2.approx.ftz.f32
// and rsqrt.approx.ftz.f32 within 2^-22 relative (PTX ISA).
#pragma once
#include <cuda_runtime.h>

namespace ct {

// e^x = 2^(x log2 e).  With t = x log2 e rounded twice (the constant and the product), |dt| <= 1.23 u |t|, so
// the relative error is at most 2^-22 + 1.23 u |x|; results below 2^-126 are 0 (an absolute error that the
// sweep's 1e-30 covers).  The sweep's kernel-value bounds allow 1e-6 + 6e-8 d2 with |x| = d2 / 2 (RBF) and
// 1e-6 + 2.4e-7 |x| (Matern).
__device__ __forceinline__ float ex2_ftz(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float2 exp2x(float2 x) {
    const float2 t = __fmul2_rn(x, make_float2(1.4426950408889634f, 1.4426950408889634f));
    return make_float2(ex2_ftz(t.x), ex2_ftz(t.y));
}

// sqrt(x), x >= 0, by one step of Newton's iteration for s^2 = x: with r = 1/sqrt(x) to 2^-22 and s = x r, so
// s = sqrt(x) (1 + e), |e| < 2^-21.6, the step s + (x - s^2) r / 2 has the relative error e^2 / 2 plus
// roundings of the correction, together below 2^-43, and then one rounding: u (1 + 2^-19) in all.  Two values
// at once, without branches.  x is taken as at least 1e-30 (1e-15 for x = 0).
__device__ __forceinline__ float2 sqrt2x(float2 x) {
    x = make_float2(fmaxf(x.x, 1e-30f), fmaxf(x.y, 1e-30f));
    float2 r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(x.x));
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(x.y));
    const float2 s = __fmul2_rn(x, r);
    const float2 e = __ffma2_rn(make_float2(-s.x, -s.y), s, x);
    return __ffma2_rn(e, __fmul2_rn(r, make_float2(0.5f, 0.5f)), s);
}

// x / b, correctly rounded, from y = the correctly rounded 1 / b: q = x y, then one residual step (Markstein's
// theorem), three operations on a chip with two FP64 operations a clock per SM.  An infinite or NaN quotient
// is returned as it is.
__device__ __forceinline__ double div_by(double x, double b, double y) {
    const double q = x * y;
    if ((__double2hiint(q) & 0x7ff00000) == 0x7ff00000) return q;
    return fma(fma(-b, q, x), y, q);
}

}  // namespace ct
