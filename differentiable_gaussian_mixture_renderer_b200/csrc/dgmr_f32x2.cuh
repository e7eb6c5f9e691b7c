// Two floats per instruction (sm_100's packed fma / mul / add.rn.f32x2): each
// half is the scalar IEEE operation, so the results are the scalar code's bits.
// A packed operation holds the FP32 pipe for two cycles (measured: 72 TFLOP/s
// of scalar fma, 74 of packed), so it saves issue slots, not FP32 time: for
// kernels bound by instruction issue.  The functions below are compared with their
// scalar forms over every float of their ranges (tests/test_gpu_packed_math.py).
#pragma once

#include <cstdint>

#include "dgmr_device_math.cuh"

namespace dgmr {

struct F2 {
    unsigned long long v;
};

__device__ __forceinline__ F2 f2(float lo, float hi)
{
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ F2 f2(float x) { return f2(x, x); }
__device__ __forceinline__ void split2(F2 a, float* lo, float* hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(*lo), "=f"(*hi) : "l"(a.v)); }
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c)
{
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b)
{
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
// a * b for a product that an add2 takes: rounded on its own.  The assembler
// contracts mul.rn.f32x2 and a following add.rn.f32x2 into one fma, whatever
// -fmad says; a * b + (-0) with a -0 that it cannot see (constant memory) is the
// same value and stays.
static __constant__ float2 c_neg_zero = { -0.0f, -0.0f };
__device__ __forceinline__ F2 mul2_rounded(F2 a, F2 b) { return fma2(a, b, f2(c_neg_zero.x, c_neg_zero.y)); }
__device__ __forceinline__ F2 add2(F2 a, F2 b)
{
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}

// 1 / x of both halves for x in [0.0099, 1]: the approximate reciprocal (within an
// ulp there) and one Newton step y + y (1 - x y).  The division's result for every
// float of that range (a test compares all of them).  The division itself carries a
// slow path for operands that this range never has: the splat backward, with two
// reciprocals per record and lane, took 324 us instead of 281 with it at 1M, 1080p.
__device__ __forceinline__ F2 recip2(F2 x)
{
    float x0, x1, y0, y1;
    split2(x, &x0, &x1);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(x0));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y1) : "f"(x1));
    const F2 y = f2(y0, y1);
    return fma2(y, fma2(f2(-x0, -x1), y, f2(1.f)), y);
}

// exp_f_nonpos (dgmr_fmath.h) of both halves, for x in [-87, 85]: the 2^n scaling
// as an add to the exponent (the scaled value is normal there, so the product
// is that bit pattern).
__device__ __forceinline__ F2 exp2_nonpos(F2 x)
{
    const F2 tm = add2(mul2_rounded(x, f2(1.44269504088896341f)), f2(12582912.0f));
    const F2 n = add2(tm, f2(-12582912.0f));
    F2 r = fma2(n, f2(-0.693145751953125f), x);
    r = fma2(n, f2(-1.42860682030941723e-06f), r);
    F2 p = fma2(f2(1.98412698412698413e-04f), r, f2(1.38888888888888889e-03f));
    p = fma2(p, r, f2(8.33333333333333333e-03f));
    p = fma2(p, r, f2(4.16666666666666667e-02f));
    p = fma2(p, r, f2(1.66666666666666667e-01f));
    p = fma2(p, r, f2(0.5f));
    p = fma2(p, r, f2(1.0f));
    p = fma2(p, r, f2(1.0f));
    float p0, p1, t0, t1;
    split2(p, &p0, &p1);
    split2(tm, &t0, &t1);
    // the shifted integer sits in tm's low bits; the magic's own bits leave by the shift
    return f2(__uint_as_float(__float_as_uint(p0) + (__float_as_uint(t0) << 23)), __uint_as_float(__float_as_uint(p1) + (__float_as_uint(t1) << 23)));
}

// erf_f (dgmr_fmath.h) of both halves: the same branches by |x| -- a branch is
// run when one of the two needs it -- and the same operations in each.
__device__ __forceinline__ F2 erf2(F2 z)
{
    float z0, z1;
    split2(z, &z0, &z1);
    const float a0 = fabsf(z0), a1 = fabsf(z1);
    const bool series0 = a0 < 1.0f, series1 = a1 < 1.0f;
    const bool tail0 = !series0 && !(a0 >= 3.92f), tail1 = !series1 && !(a1 >= 3.92f); // NaN takes the tail and stays NaN
    const F2 ax = f2(a0, a1), zz = mul2(z, z);
    float y0 = 1.0f, y1 = 1.0f;
    if (tail0 || tail1) {
        // Abramowitz & Stegun 7.1.26 with recip_hastings
        const F2 d = fma2(f2(0.3275911f), ax, f2(1.0f)), nd = fma2(f2(-0.3275911f), ax, f2(-1.0f));
        F2 y = fma2(fma2(f2(0.17927061f), d, f2(-0.971220434f)), d, f2(1.72301638f));
        y = fma2(y, fma2(nd, y, f2(1.0f)), y);
        y = fma2(y, fma2(nd, y, f2(1.0f)), y);
        y = fma2(y, fma2(nd, y, f2(1.0f)), y);
        float d0, d1, t0, t1;
        split2(d, &d0, &d1);
        split2(y, &t0, &t1);
        const F2 t = f2(d0 == 0x1.fffffep+0f ? 0x1.000002p-1f : t0, d1 == 0x1.fffffep+0f ? 0x1.000002p-1f : t1);
        // the negated polynomial: -p, so that 1 - p e is one add
        F2 p = fma2(f2(-1.061405429f), t, f2(1.453152027f));
        p = fma2(p, t, f2(-1.421413741f));
        p = fma2(p, t, f2(0.284496736f));
        p = fma2(p, t, f2(-0.254829592f));
        p = mul2(p, t);
        const F2 e = exp2_nonpos(mul2(zz, f2(-1.0f)));
        const F2 r = add2(mul2_rounded(p, e), f2(1.0f));
        float r0, r1;
        split2(r, &r0, &r1);
        y0 = tail0 ? r0 : y0;
        y1 = tail1 ? r1 : y1;
    }
    if (series0 || series1) {
        F2 p = fma2(f2(-1.22905553017179263e-09f), zz, f2(1.48071928158792176e-08f));
        p = fma2(p, zz, f2(-1.63658446912349245e-07f));
        p = fma2(p, zz, f2(1.64621143658892463e-06f));
        p = fma2(p, zz, f2(-1.49256503584062504e-05f));
        p = fma2(p, zz, f2(1.20553329817896636e-04f));
        p = fma2(p, zz, f2(-8.54832702345085225e-04f));
        p = fma2(p, zz, f2(5.22397762544218793e-03f));
        p = fma2(p, zz, f2(-2.68661706451312522e-02f));
        p = fma2(p, zz, f2(1.12837916709551261e-01f));
        p = fma2(p, zz, f2(-3.76126389031837538e-01f));
        p = fma2(p, zz, f2(1.12837916709551256e+00f));
        const F2 r = mul2(ax, p);
        float r0, r1;
        split2(r, &r0, &r1);
        y0 = series0 ? r0 : y0;
        y1 = series1 ? r1 : y1;
    }
    return f2(copysignf(y0, z0), copysignf(y1, z1));
}

// cdf_inv_SD (dgmr_device_math.cuh) at two positions x; nc = -centre in both halves
__device__ __forceinline__ F2 cdf2_inv_SD(F2 nc, F2 inv_sd, F2 x)
{
    const F2 z = mul2(mul2(add2(x, nc), inv_sd), f2(0.70710678118654752440f));
    return mul2(f2(0.5f), add2(f2(1.0f), erf2(z)));
}

} // namespace dgmr
