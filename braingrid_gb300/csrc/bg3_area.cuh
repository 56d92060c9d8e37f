// The overlap area of two neurons' radii (ConnGrowth.cpp:319-376), in double as the reference
// promotes and in float-float arithmetic with certified rounding.
//
// pair_area_fp64 is two double acos, two double sin and two double divisions a pair, and this
// chip's FP64 pipe runs at 1/64 of the FP32 rate: the weight pass over 7.6 M synapses spent 2.09 ms
// there.  pair_area_ff evaluates each double expression to within a bound in pairs of floats and
// rounds it to float where every value within the bound rounds the same; a pair with any uncertain
// value (about 1 in 10,000) is evaluated in double.  The same bits, in 160 us; the instructions of the
// areas bound it.  (Newton steps on acosf and Taylor series for the sines: 239 us.)
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

__device__ __forceinline__ float rcp_approx(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rsqrt_approx(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// cos and asin values at s = i / 128 up to sin(pi/4): {sqrt(1 - s s), asin(s)}, each as two floats.
static __device__ const float4 area_nodes[92] = {
    {0x1p+0f, 0x0p+0f, 0x0p+0f, 0x0p+0f},
    {0x1.fffcp-1f, -0x1.0002p-31f, 0x1.0000aap-7f, 0x1.57bbc2p-32f},
    {0x1.fffp-1f, -0x1.0008p-27f, 0x1.0002aap-6f, 0x1.7bbd2ap-31f},
    {0x1.ffdbfep-1f, 0x1.77d26cp-26f, 0x1.8009p-6f, 0x1.23b204p-31f},
    {0x1.ffbffcp-1f, -0x1.002808p-34f, 0x1.000aacp-5f, -0x1.0fa31cp-32f},
    {0x1.ff9bf6p-1f, 0x1.d0ba06p-28f, 0x1.4014d8p-5f, 0x1.ff5f16p-30f},
    {0x1.ff6fecp-1f, -0x1.16d006p-27f, 0x1.80240ap-5f, -0x1.c049eap-30f},
    {0x1.ff3bdap-1f, 0x1.b67254p-27f, 0x1.c0393ep-5f, 0x1.970b24p-31f},
    {0x1.feffcp-1f, -0x1.00a07p-28f, 0x1.002abep-4f, -0x1.6ac9e6p-32f},
    {0x1.febb9ap-1f, -0x1.8a260cp-26f, 0x1.203ce2p-4f, 0x1.67019ap-29f},
    {0x1.fe6f64p-1f, -0x1.751372p-26f, 0x1.40539p-4f, 0x1.20737ep-31f},
    {0x1.fe1b1ap-1f, 0x1.8af76cp-27f, 0x1.606f4ap-4f, -0x1.19e668p-29f},
    {0x1.fdbebap-1f, 0x1.22f87ep-26f, 0x1.809092p-4f, 0x1.227ca6p-29f},
    {0x1.fd5a4p-1f, -0x1.2a1292p-26f, 0x1.a0b7fp-4f, 0x1.dd3c56p-31f},
    {0x1.fceda4p-1f, 0x1.0f7edap-28f, 0x1.c0e5e8p-4f, 0x1.ee2e5ap-33f},
    {0x1.fc78e4p-1f, -0x1.fa07a4p-27f, 0x1.e11bp-4f, 0x1.3c4d36p-29f},
    {0x1.fbfbf8p-1f, -0x1.438aa2p-29f, 0x1.00abep-3f, 0x1.8253c4p-28f},
    {0x1.fb76dcp-1f, -0x1.4ebdacp-26f, 0x1.10ce5ap-3f, -0x1.16d5dp-29f},
    {0x1.fae988p-1f, -0x1.57d6dp-26f, 0x1.20f53p-3f, 0x1.84661p-30f},
    {0x1.fa53f4p-1f, 0x1.f9897p-26f, 0x1.3120aap-3f, -0x1.04b42ep-29f},
    {0x1.f9b61ep-1f, -0x1.fb91b6p-26f, 0x1.41510cp-3f, 0x1.602284p-28f},
    {0x1.f90ff8p-1f, -0x1.740accp-27f, 0x1.5186ap-3f, 0x1.5bd2e8p-32f},
    {0x1.f8617cp-1f, 0x1.557adep-26f, 0x1.61c1acp-3f, -0x1.8aa8b4p-29f},
    {0x1.f7aaa4p-1f, -0x1.1fcbb2p-26f, 0x1.720278p-3f, 0x1.299a78p-32f},
    {0x1.f6eb62p-1f, 0x1.a4ee62p-26f, 0x1.82494ep-3f, 0x1.a1cf2p-28f},
    {0x1.f623b2p-1f, -0x1.90cbecp-26f, 0x1.92967ap-3f, 0x1.8e36cep-29f},
    {0x1.f55384p-1f, 0x1.1249dp-26f, 0x1.a2ea46p-3f, 0x1.5a4cc6p-30f},
    {0x1.f47ad2p-1f, 0x1.8f53a4p-28f, 0x1.b344fep-3f, 0x1.352f8ap-28f},
    {0x1.f3999p-1f, -0x1.c9cef2p-26f, 0x1.c3a6f2p-3f, -0x1.8aa2f6p-28f},
    {0x1.f2afbp-1f, -0x1.5b1fc2p-27f, 0x1.d4106cp-3f, 0x1.748b62p-28f},
    {0x1.f1bd28p-1f, -0x1.1bff4ep-27f, 0x1.e481cp-3f, 0x1.f9ce26p-28f},
    {0x1.f0c1eap-1f, 0x1.37f48cp-26f, 0x1.f4fb4p-3f, -0x1.aa5f0cp-28f},
    {0x1.efbdecp-1f, -0x1.d61624p-26f, 0x1.02be9cp-2f, 0x1.c170fap-27f},
    {0x1.eeb11cp-1f, -0x1.577a02p-26f, 0x1.0b0402p-2f, 0x1.491734p-28f},
    {0x1.ed9b6cp-1f, 0x1.e788ccp-26f, 0x1.134dfap-2f, 0x1.300a28p-27f},
    {0x1.ec7cdp-1f, 0x1.e56b5cp-26f, 0x1.1b9cb2p-2f, -0x1.b57434p-27f},
    {0x1.eb5538p-1f, -0x1.3af2cap-27f, 0x1.23f052p-2f, 0x1.e2ee16p-29f},
    {0x1.ea249p-1f, 0x1.d7bad8p-26f, 0x1.2c490ap-2f, 0x1.f17bdp-27f},
    {0x1.e8eaccp-1f, -0x1.26ddbcp-27f, 0x1.34a70ap-2f, -0x1.4d0aaap-27f},
    {0x1.e7a7d6p-1f, 0x1.d99e12p-27f, 0x1.3d0a7cp-2f, 0x1.312f66p-28f},
    {0x1.e65b9ep-1f, 0x1.bd7472p-26f, 0x1.457394p-2f, -0x1.1bc756p-28f},
    {0x1.e50612p-1f, -0x1.77294ap-29f, 0x1.4de28p-2f, 0x1.1b9ca2p-27f},
    {0x1.e3a71cp-1f, -0x1.914e12p-28f, 0x1.565774p-2f, 0x1.96cdep-27f},
    {0x1.e23ea8p-1f, 0x1.5a58d2p-32f, 0x1.5ed2a4p-2f, -0x1.b512bcp-28f},
    {0x1.e0cca2p-1f, -0x1.a2d0eep-26f, 0x1.675442p-2f, -0x1.9accf2p-27f},
    {0x1.df50f2p-1f, -0x1.b608b2p-26f, 0x1.6fdc84p-2f, -0x1.93611cp-27f},
    {0x1.ddcb8p-1f, 0x1.bb810cp-26f, 0x1.786bap-2f, 0x1.d3fbe4p-28f},
    {0x1.dc3c38p-1f, 0x1.b42b82p-27f, 0x1.8101d2p-2f, -0x1.bc825ap-27f},
    {0x1.daa2fep-1f, 0x1.f55c3ap-26f, 0x1.899f4ep-2f, 0x1.b92c5ap-27f},
    {0x1.d8ffbap-1f, 0x1.7228bap-26f, 0x1.924454p-2f, 0x1.88c598p-27f},
    {0x1.d7525p-1f, 0x1.b738f2p-26f, 0x1.9af12p-2f, -0x1.d91678p-28f},
    {0x1.d59aa6p-1f, -0x1.ce6e38p-27f, 0x1.a3a5eep-2f, -0x1.f49ab2p-28f},
    {0x1.d3d89cp-1f, -0x1.e89f8ep-29f, 0x1.ac62fep-2f, 0x1.816552p-27f},
    {0x1.d20c16p-1f, -0x1.75ad8ep-28f, 0x1.b52896p-2f, -0x1.b592eap-27f},
    {0x1.d034f4p-1f, 0x1.34c10ap-28f, 0x1.bdf6f4p-2f, 0x1.eb9a42p-28f},
    {0x1.ce5316p-1f, 0x1.cd80ccp-27f, 0x1.c6ce62p-2f, 0x1.1ba266p-27f},
    {0x1.cc665cp-1f, -0x1.f9af3cp-26f, 0x1.cfaf28p-2f, -0x1.73e02cp-27f},
    {0x1.ca6e9ep-1f, 0x1.98ad38p-26f, 0x1.d8998cp-2f, 0x1.87cc0ap-27f},
    {0x1.c86bbep-1f, -0x1.3ecbb4p-26f, 0x1.e18dep-2f, -0x1.04bdf2p-27f},
    {0x1.c65d9p-1f, 0x1.b8a13ep-26f, 0x1.ea8c6ep-2f, 0x1.7d79ap-28f},
    {0x1.c443f2p-1f, -0x1.596ea8p-28f, 0x1.f3958ap-2f, 0x1.d9bbdep-27f},
    {0x1.c21eb8p-1f, -0x1.74e346p-26f, 0x1.fca98ap-2f, -0x1.34e8aap-27f},
    {0x1.bfedb6p-1f, 0x1.ef84ecp-27f, 0x1.02e46p-1f, 0x1.d5e168p-27f},
    {0x1.bdb0c4p-1f, -0x1.fcf57p-26f, 0x1.0779c6p-1f, -0x1.5905a4p-28f},
    {0x1.bb67aep-1f, 0x1.0b0996p-26f, 0x1.0c1524p-1f, -0x1.f4a326p-27f},
    {0x1.b91248p-1f, 0x1.87130ep-26f, 0x1.10b6aap-1f, -0x1.bc6bdp-29f},
    {0x1.b6b06p-1f, -0x1.2d328cp-26f, 0x1.155e8cp-1f, -0x1.abfff6p-26f},
    {0x1.b441bep-1f, -0x1.52aap-31f, 0x1.1a0cfcp-1f, -0x1.2782c2p-26f},
    {0x1.b1c62ep-1f, -0x1.36a6cp-27f, 0x1.1ec23p-1f, 0x1.8e2952p-26f},
    {0x1.af3d76p-1f, -0x1.3cac78p-26f, 0x1.237e64p-1f, -0x1.0c6408p-26f},
    {0x1.aca75ap-1f, -0x1.657668p-26f, 0x1.2841cep-1f, 0x1.0c52eap-30f},
    {0x1.aa039cp-1f, -0x1.f22db2p-26f, 0x1.2d0caep-1f, -0x1.40de3cp-26f},
    {0x1.a751fap-1f, -0x1.77091cp-26f, 0x1.31df4p-1f, 0x1.f7a63ap-26f},
    {0x1.a4923p-1f, -0x1.314ddp-27f, 0x1.36b9ccp-1f, -0x1.d90f24p-26f},
    {0x1.a1c3f6p-1f, 0x1.9403e6p-26f, 0x1.3b9c9p-1f, 0x1.88652ep-26f},
    {0x1.9ee704p-1f, -0x1.bc84fp-27f, 0x1.4087dap-1f, 0x1.11cca6p-27f},
    {0x1.9bfb08p-1f, -0x1.25b922p-26f, 0x1.457bf4p-1f, -0x1.ce035ep-26f},
    {0x1.98ffbp-1f, -0x1.e131dp-29f, 0x1.4a792ap-1f, 0x1.3c9854p-27f},
    {0x1.95f4a6p-1f, 0x1.37b36ap-27f, 0x1.4f7fd2p-1f, 0x1.785f66p-26f},
    {0x1.92d99p-1f, -0x1.74f2a8p-27f, 0x1.549044p-1f, -0x1.7b148ep-26f},
    {0x1.8fae0cp-1f, 0x1.5ad38ap-29f, 0x1.59aad8p-1f, -0x1.c625fep-26f},
    {0x1.8c71b6p-1f, 0x1.918936p-26f, 0x1.5ecfeep-1f, 0x1.8e4b74p-28f},
    {0x1.892426p-1f, -0x1.281758p-26f, 0x1.63ffeep-1f, -0x1.25cce2p-26f},
    {0x1.85c4e8p-1f, -0x1.5afa28p-28f, 0x1.693b4p-1f, -0x1.b7623ep-26f},
    {0x1.825388p-1f, -0x1.d4747ep-27f, 0x1.6e8254p-1f, -0x1.f0cefep-27f},
    {0x1.7ecf88p-1f, -0x1.69ef24p-26f, 0x1.73d5a2p-1f, -0x1.f08432p-26f},
    {0x1.7b3862p-1f, 0x1.e75efcp-27f, 0x1.7935a6p-1f, -0x1.fca0b2p-26f},
    {0x1.778d8cp-1f, 0x1.13b85p-26f, 0x1.7ea2e4p-1f, 0x1.64813ep-28f},
    {0x1.73ce7p-1f, 0x1.3edec8p-27f, 0x1.841decp-1f, -0x1.5dd68ap-26f},
    {0x1.6ffa7p-1f, -0x1.79b87ep-26f, 0x1.89a75p-1f, -0x1.9e5ae2p-32f},
    {0x1.6c10ep-1f, 0x1.53cbacp-26f, 0x1.8f3fb2p-1f, -0x1.636d2ap-26f},
    {0x1.68111p-1f, 0x1.530baap-26f, 0x1.94e7b8p-1f, 0x1.b479fp-26f},
};

// Rounds a float-float value to float where every value within err of it rounds the same.
__device__ __forceinline__ float area_round(FF a, float err, bool &ok)
{
    const float up = a.hi + (a.lo + err), dn = a.hi + (a.lo - err);
    ok = ok && up == dn;  // false for NaN
    return up;
}

// a / (2 r l) rounded to double and then to float, where that is certain: one correction of the
// approximate quotient by its residual against the exact 48-bit product.
__device__ __forceinline__ float area_cos(float a, float r, float l, bool &ok)
{
    const float r2 = 2.0f * r, dh = r2 * l, dl = __fmaf_rn(r2, l, -dh);
    const float inv = rcp_approx(dh);
    const float q0 = a * inv;
    const float res = __fmaf_rn(-q0, dl, __fmaf_rn(-q0, dh, a));
    const FF q = ff_fast_two_sum(q0, res * inv);
    ok = ok && fabsf(a) > 0x1p-40f;
    return area_round(q, fabsf(q.hi) * 0x1p-41f, ok);
}

// r - sin(r) for r = (float)(2 (float)acos((double)x)) with the sine rounded as (float)sin((double)r),
// where both roundings are certain, in float as the reference subtracts; *angle = r.
//
//   s = sqrt(1 - x x) in float-float.  Of |x| and s the smaller is the sine m of an angle up to pi/4
//   and the larger its cosine M.  At the node i / 128 nearest to m, with cosine c and angle g,
//   asin(m) = g + asin(m c - M i / 128), the last argument below 1/181 so that its series is the
//   argument itself and two terms in float.  acos(|x|) is that or pi/2 minus it, acos(x) pi minus that
//   for x < 0.
//   sin(2 y) = 2 x s; rounding y to y - lo turned the angle by -2 lo, so
//   sin(r) = 2 x s - 2 lo cos(2 y); the next term, 2 lo^2 sin(2 y), is below 2^-45 of it.
//
//   Errors.  w is exact for x x >= 1/2 and to 2^-48 below.  rsqrt.approx is good to 2^-22.9 and s0 to
//   2^-22.3, so one correction leaves 2^-44.4, its roundings (three of 2^-24 on a part of 2^-22.3) 2^-44.7:
//   s to 2^-43.5 of itself.  That moves an asin(s) of a by 2^-43.5 tan a (at most 2^-43.2 a), and by way of
//   M t, at most 1/2, an asin(|x|) by 2^-44.5.  The products' low parts, the node's and the sums are below
//   2^-24 and round by 2^-48 each, about five of them; the base's low part, up to 2^-23.5, by 2^-47.5 twice:
//   2^-45.7 in all, and 2^-47 without a base.  So y is within 2^-43.2 y + 2^-45.7 (2^-47 where y is an asin
//   itself and may be small) of the angle, and 2^-41 y + 2^-45 is allowed for.  The sine takes 2^-43.5 of
//   itself from s and twice the angle's error times the cosine: 2^-41.9 where it is near 1, 2^-41.5 of a for a
//   small a, 2^-42.2 near pi; 2^-41 of it + 2^-42 is allowed for.  (Largest seen in 3e7 random pairs: 0.35
//   and 0.43 of what is allowed.)
__device__ __forceinline__ float area_segment(float x, bool &ok)
{
    const float ax = fabsf(x);
    const float xx = x * x, xl = __fmaf_rn(x, x, -xx);
    FF w = ff_fast_two_sum(1.0f, -xx);
    w = ff_fast_two_sum(w.hi, w.lo - xl);
    const float rs = rsqrt_approx(w.hi);
    const float s0 = w.hi * rs;
    const FF s = ff_fast_two_sum(s0, 0.5f * rs * (__fmaf_rn(-s0, s0, w.hi) + w.lo));
    const bool sine = ax < s.hi;  // acos = pi/2 - asin(|x|)
    const FF m = sine ? FF{ax, 0.0f} : s, M = sine ? s : FF{ax, 0.0f};
    const int i = min((int)__fmaf_rn(m.hi, 128.0f, 0.5f), 91);  // |x| > 1: any node, s is NaN
    const float4 node = area_nodes[i];
    const float t = (float)i * 0x1p-7f;
    // u = m c - M t
    const float p1 = m.hi * node.x, p2 = M.hi * t;
    const float e1 = __fmaf_rn(m.lo, node.x, __fmaf_rn(m.hi, node.y, __fmaf_rn(m.hi, node.x, -p1)));
    const float e2 = __fmaf_rn(M.lo, t, __fmaf_rn(M.hi, t, -p2));
    // p1 - p2 is exact: within a factor of two, both multiples of its last place at the first node's lower
    // edge, or p2 = 0
    const FF d = ff_fast_two_sum(p1 - p2, e1 - e2);
    const float uu = d.hi * d.hi;
    const float tail = __fmaf_rn(d.hi * uu, __fmaf_rn(uu, 0.075f, 0x1.555556p-3f), d.lo);
    FF y = ff_two_sum(node.z, d.hi);
    y.lo = y.lo + (node.w + tail);
    // (k pi/2) +- y
    const float base = sine ? 0x1.921fb6p+0f : (x < 0.0f ? 0x1.921fb6p+1f : 0.0f);
    const bool minus = sine ? x > 0.0f : x < 0.0f;
    const FF a = ff_two_sum(base, minus ? -y.hi : y.hi);
    const float al = a.lo + (base * (-0x1.777a5cp-25f / 0x1.921fb6p+0f) + (minus ? -y.lo : y.lo));
    y = ff_fast_two_sum(a.hi, al);
    const float r = area_round(y, __fmaf_rn(y.hi, 0x1p-41f, 0x1p-45f), ok);
    const float x2 = 2.0f * x;
    const float ph = x2 * s.hi;
    const float pl = __fmaf_rn(x2, s.lo, __fmaf_rn(x2, s.hi, -ph));
    const FF v = ff_fast_two_sum(ph, __fmaf_rn(-2.0f * y.lo, __fmaf_rn(x2, x, -1.0f), pl));
    const float sn = area_round(v, __fmaf_rn(fabsf(v.hi), 0x1p-41f, 0x1p-42f), ok);
    const float angle = 2.0f * r;
    return angle - sn;
}

// pair_area_fp64 with every double expression rounded from its float-float value, where certain.
// The doublings and the halving are exact in float.
__device__ __forceinline__ float pair_area_ff(float len, float len2, float ri, float rj, bool &ok)
{
    // products and quotients far from float's limits; false for NaN too
    ok = fminf(fminf(ri, rj), len) > 0x1p-20f && fmaxf(fmaxf(ri, rj), len) < 0x1p+20f;
    const float r12 = ri * ri, r22 = rj * rj;
    const float segj = area_segment(area_cos(r22 + len2 - r12, rj, len, ok), ok);
    const float segi = area_segment(area_cos(r12 + len2 - r22, ri, len, ok), ok);
    return 0.5f * (r22 * segj + r12 * segi);
}

// The frontier distance of a pair; negative where the radii overlap.
__device__ __forceinline__ float pair_delta(float xi, float yi, float ri, float xj, float yj, float rj)
{
    const float dx = xi - xj, dy = yi - yj;
    return sqrtf(dx * dx + dy * dy) - (ri + rj);
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
