// The overlap area of two neurons' radii (ConnGrowth.cpp:319-376), in double as the reference
// promotes and in float-float arithmetic with certified rounding.
//
// pair_area_fp64 is two double acos, two double sin and two double divisions a pair, and this
// chip's FP64 pipe runs at 1/64 of the FP32 rate: the weight pass over 7.6 M synapses spent 2.09 ms
// there.  pair_area_ff evaluates each double expression to within a bound E in pairs of floats
// (~400 FP32 instructions a pair) and rounds it to float where the rounding is certain (ff_round);
// a pair with any uncertain value (about 1 in 4,000) is evaluated in double.  The same bits, in
// 0.23 ms.
#pragma once
#include "bg3_internal.cuh"

namespace bg3 {

static __device__ __noinline__ float pair_area_fp64(float len, float len2, float ri, float rj)
{
    float r12 = ri * ri, r22 = rj * rj;
    float cosCBA = (float)((double)(r22 + len2 - r12) / (2.0 * (double)rj * (double)len));
    float angCBA = acos_cr(cosCBA);
    float angCBD = (float)(2.0 * (double)angCBA);
    float cosCAB = (float)((double)(r12 + len2 - r22) / (2.0 * (double)ri * (double)len));
    float angCAB = acos_cr(cosCAB);
    float angCAD = (float)(2.0 * (double)angCAB);
    return (float)(0.5 * (double)(r22 * (angCBD - sin_cr(angCBD)) + r12 * (angCAD - sin_cr(angCAD))));
}

__device__ __forceinline__ FF ff_mul(FF a, FF b)
{
    const float p = a.hi * b.hi;
    float e = __fmaf_rn(a.hi, b.hi, -p);
    e = __fmaf_rn(a.hi, b.lo, e);
    e = __fmaf_rn(a.lo, b.hi, e);
    return ff_fast_two_sum(p, e);
}
__device__ __forceinline__ FF ff_add_big(FF a, FF b)  // |a| >= |b|
{
    FF s = ff_fast_two_sum(a.hi, b.hi);
    s.lo = s.lo + (a.lo + b.lo);
    return ff_fast_two_sum(s.hi, s.lo);
}

// cos(t) - 1 (odd = true) or sin(t) / t - 1 (odd = false) from z = t t, |t| <= pi/4 (a little
// beyond is fine): Taylor's series, the first three terms in float-float and four more in float.
// Terms left out and the float tail's rounding: below 2^-40.
__device__ __forceinline__ FF ff_series(FF z, bool cosine)
{
    float p = cosine ? -0x1.93974ap-37f : -0x1.ae7f3ep-41f;               // -1/14!, -1/15!
    p = __fmaf_rn(p, z.hi, cosine ? 0x1.1eed8ep-29f : 0x1.612462p-33f);   // 1/12!, 1/13!
    p = __fmaf_rn(p, z.hi, cosine ? -0x1.27e4fcp-22f : -0x1.ae6456p-26f); // -1/10!, -1/11!
    p = __fmaf_rn(p, z.hi, cosine ? 0x1.a01a02p-16f : 0x1.71de3ap-19f);   // 1/8!, 1/9!
    FF q = ff_fast_two_sum(cosine ? -0x1.6c16c2p-10f : -0x1.a01a02p-13f, p * z.hi);  // -1/6!, -1/7!
    q.lo += cosine ? 0x1.27d27ep-35f : 0x1.7f97fap-39f;
    q = ff_mul(q, z);
    q = ff_add_big(cosine ? FF{0x1.555556p-5f, -0x1.555556p-30f} : FF{0x1.111112p-7f, -0x1.dddddep-32f},
                   q);  // 1/4!, 1/5!
    q = ff_mul(q, z);
    q = ff_add_big(cosine ? FF{-0.5f, 0.0f} : FF{-0x1.555556p-3f, 0x1.555556p-28f}, q);  // -1/2!, -1/3!
    return ff_mul(q, z);
}

// a / (2 r l) rounded to double and then to float, where that is certain: one correction of the
// approximate quotient by its residual against the exact 48-bit product.
__device__ __forceinline__ float area_cos(float a, float r, float l, bool &ok)
{
    const float r2 = 2.0f * r, dh = r2 * l, dl = __fmaf_rn(r2, l, -dh);
    const float inv = __fdividef(1.0f, dh);
    const float q0 = a * inv;
    const float res = __fmaf_rn(-q0, dl, __fmaf_rn(-q0, dh, a));
    const FF q = ff_fast_two_sum(q0, res * inv);
    float c = 0.0f;
    ok = ff_round(q, fabsf(q.hi) * 0x1p-41f, c) && fabsf(a) > 0x1p-60f && ok;
    return c;
}

// (float)acos((double)x) where certain: one Newton step y0 + (cos(y0) - |x|) / sin(y0) from the
// float acos of |x| (two ulp, so the step's remainder is below 2^-45 of y), the difference in
// float-float, about 1 for small y0 (1 - |x| is exact there) and from sin(pi/2 - y0) otherwise.
__device__ __forceinline__ float area_acos(float x, bool &ok)
{
    const float ax = fabsf(x);
    const float y0 = acosf(ax);
    const bool near0 = ax >= 0.703125f;  // y0 < 0.7910
    FF t = near0 ? FF{y0, 0.0f} : ff_two_sum(0x1.921fb6p+0f - y0, -0x1.777a5cp-25f);
    const float zh = t.hi * t.hi;
    const FF z = ff_fast_two_sum(zh, __fmaf_rn(2.0f * t.hi, t.lo, __fmaf_rn(t.hi, t.hi, -zh)));
    FF d = ff_series(z, near0);
    if (!near0) d = ff_add_big(t, ff_mul(d, t));  // sin(t)
    const FF m = ff_two_sum(d.hi, near0 ? 1.0f - ax : -ax);
    const float c = (m.hi + (m.lo + d.lo)) * rsqrtf((1.0f - ax) * (1.0f + ax));
    FF y = ff_fast_two_sum(y0, c);
    float err = y0 * 0x1p-39f;
    if (x < 0.0f) {  // pi - y
        FF s = ff_two_sum(0x1.921fb6p+1f, -y.hi);
        s.lo = s.lo + (-0x1.777a5cp-24f - y.lo);
        y = ff_fast_two_sum(s.hi, s.lo);
        err += 0x1p-45f;
    }
    float r = 0.0f;
    ok = ff_round(y, err, r) && ok;
    return r;
}

// (float)sin((double)a) for 0 <= a <= 2 pi, where certain: reduced by a multiple k of pi/2 held as
// two floats; the first subtraction is exact (the result is a whole number of units of 2^-24 or
// of a's last place below pi/4, or a itself).
__device__ __forceinline__ float area_sin(float a, bool &ok)
{
    const float k = rintf(a * 0x1.45f306p-1f);
    const FF t = ff_two_sum(__fmaf_rn(-k, 0x1.921fb6p+0f, a), k * 0x1.777a5cp-25f);
    const int ki = (int)k;
    const bool cosine = (ki & 1) != 0;
    const float zh = t.hi * t.hi;
    const FF z = ff_fast_two_sum(zh, __fmaf_rn(2.0f * t.hi, t.lo, __fmaf_rn(t.hi, t.hi, -zh)));
    const FF d = ff_series(z, cosine);
    const FF one = cosine ? FF{1.0f, 0.0f} : t;
    FF s = ff_add_big(one, ff_mul(d, one));
    if (ki & 2) s = FF{-s.hi, -s.lo};
    float r = 0.0f;
    ok = ff_round(s, fabsf(s.hi) * 0x1p-39f + 0x1p-45f, r) && ok;
    return r;
}

// pair_area_fp64 with every double expression rounded from its float-float value, where certain.
// The doublings and the halving are exact in float.
__device__ __forceinline__ float pair_area_ff(float len, float len2, float ri, float rj, bool &ok)
{
    // products and quotients far from float's limits; false for NaN too
    ok = ri > 0x1p-30f && rj > 0x1p-30f && len > 0x1p-30f && ri < 0x1p+30f && rj < 0x1p+30f &&
         len < 0x1p+30f;
    const float r12 = ri * ri, r22 = rj * rj;
    const float angCBD = 2.0f * area_acos(area_cos(r22 + len2 - r12, rj, len, ok), ok);
    const float angCAD = 2.0f * area_acos(area_cos(r12 + len2 - r22, ri, len, ok), ok);
    return 0.5f * (r22 * (angCBD - area_sin(angCBD, ok)) + r12 * (angCAD - area_sin(angCAD, ok)));
}

// Frontier distance and overlap area of the pair (i = source, j = dest)
// (Connections/ConnGrowth.cpp:319-376; dist from Layouts/Layout.cpp:54-69).  Returns 0 for pairs
// that do not overlap.
__device__ __forceinline__ float pair_area(float xi, float yi, float ri, float xj, float yj,
                                           float rj)
{
    float dx = xi - xj, dy = yi - yj;
    float len2 = dx * dx + dy * dy;
    float len = sqrtf(len2);
    float delta = len - (ri + rj);
    if (!(delta < 0.0f)) return 0.0f;
    float rmin = fminf(ri, rj), rmax = fmaxf(ri, rj);
    if (len + rmin <= rmax) {
        const float pi = 3.1415926536f;  // Utils/Global.cpp:90
        return pi * rmin * rmin;
    }
    bool ok;
    const float a = pair_area_ff(len, len2, ri, rj, ok);
    return ok ? a : pair_area_fp64(len, len2, ri, rj);
}

}  // namespace bg3
