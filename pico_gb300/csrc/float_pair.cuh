// Float pairs: a value as the unevaluated sum of two floats (about 48 bits), for the few places where the
// reference computes in double and rounds the result to float.
//
// The chip's FP64 rate is a 64th of its FP32 rate, and the shade kernel kept the FP64 pipe 78 % busy (its FP32 pipe
// 9 %) on the sine, cosine, square root and quotient of each sampled lobe.  The functions here evaluate them in
// pairs (error-free sums and products after Dekker 1971 and Knuth, products through FMA) and give the float that the
// double evaluation rounds to: a result is taken only if it rounds to the same float over the whole interval that
// the pair's and the double's errors allow (Ziv's rounding test, 1991); the rest, about one in 2^18, is evaluated
// in double as before.  So results are those of the double evaluation bit for bit.  The 1080p lit-field render's
// shading: 16.5 -> 7.9 ms of 75.4 -> 66.8, the Cornell box's at 256 x 256: 0.41 -> 0.24 ms of 1.38 -> 1.20.
#pragma once

#include "exact_math.cuh"

namespace pico {
namespace pair {

struct P { float h, l; };   // h + l, |l| at most half an ulp of h

__device__ __forceinline__ P fast_sum(float a, float b)   // exact for |a| >= |b|
{
    const float s = __fadd_rn(a, b);
    return P{s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ P sum(float a, float b)   // exact
{
    const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
    return P{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t))};
}
__device__ __forceinline__ P mul(P a, float b)
{
    const float p = __fmul_rn(a.h, b);
    return fast_sum(p, __fmaf_rn(a.l, b, __fmaf_rn(a.h, b, -p)));
}
__device__ __forceinline__ P mul(P a, P b)
{
    const float p = __fmul_rn(a.h, b.h);
    return fast_sum(p, __fmaf_rn(a.h, b.l, __fmaf_rn(a.l, b.h, __fmaf_rn(a.h, b.h, -p))));
}
__device__ __forceinline__ P add(P a, P b)   // |a| >= |b|, or of either order with sum
{
    const P s = sum(a.h, b.h);
    return fast_sum(s.h, __fadd_rn(s.l, __fadd_rn(a.l, b.l)));
}

// The float nearest to h + l where every value within |h| * rel of it rounds to the same one; false elsewhere
// (and for anything not finite).
__device__ __forceinline__ bool rounds(P a, float rel, float& out)
{
    const float up = __fadd_rn(a.h, __fmaf_rn(fabsf(a.h), rel, a.l));
    const float dn = __fadd_rn(a.h, __fmaf_rn(-fabsf(a.h), rel, a.l));
    out = up;
    return up == dn;
}

// Bounds of the pair evaluations' relative errors (measured against 64-bit-mantissa arithmetic over 4M arguments and
// the neighbourhoods of the quadrants: 2^-47.6, 2^-45.0 before the product with the radius, 2^-44.9), with the double
// evaluation's own (under 2^-50) and a margin on top.
constexpr float kRelPhi = 0x1p-45f, kRelCircle = 0x1p-43f, kRelQuotient = 0x1p-43f;

// pi and pi / 2 as sums of floats: 3.14159265358979323846 in steps of 24 bits.
constexpr float kPi0 = 0x1.921fb6p+1f, kPi1 = -0x1.777a5cp-24f;
constexpr float kHalf0 = 0x1.921fb6p+0f, kHalf1 = -0x1.777a5cp-25f, kHalf2 = -0x1.ee59dap-50f;

// (float)((double)a * pi * 2) for a in [0, 2): the product's rounding errors are below 2^-46 of it.
static __device__ __noinline__ float two_pi_times_double(float a) { return (float)((double)a * 3.14159265358979323846 * 2.0); }
__device__ __forceinline__ float two_pi_times(float a)
{
    float out;
    if (rounds(mul(P{kPi0, kPi1}, a), kRelPhi, out)) return copysignf(2.0f * out, a);   // the sum loses a zero's sign
    return two_pi_times_double(a);
}

static __device__ __noinline__ float2 circle_double(float r, float phi)
{
    const double c = cos((double)phi), s = sin((double)phi);
    return make_float2((float)((double)r * c), (float)((double)r * s));
}

// ((float)(r * cos(phi)), (float)(r * sin(phi))) evaluated in double.
//
// phi = k pi/2 + y with |y| <= pi/4: phi - k kHalf0 is exact (both are multiples of the smaller one's ulp and the
// difference is below 1), and the two further parts of pi/2 leave y with an error below 2^-72.  sin y and cos y are
// their Taylor series in z = y^2 up to y^15 and y^16 (the rest is below 2^-48); coefficients from 1 / 3! and 1 / 2!
// on as pairs while the term can reach 2^-20 of the sum, in float beyond.
__device__ __forceinline__ float2 circle(float r, float phi)
{
    if (!(phi >= 0.0f && phi <= 6.5f)) return circle_double(r, phi);
    const float k = rintf(__fmul_rn(phi, 0.636619772f));
    const float p1 = __fmul_rn(k, kHalf1), e1 = __fmaf_rn(k, kHalf1, -p1);
    P y = sum(__fmaf_rn(-k, kHalf0, phi), -p1);
    y = fast_sum(y.h, __fsub_rn(y.l, __fmaf_rn(k, kHalf2, e1)));
    const P z = mul(y, y);
    // sine: y + y z (-1/6 + z (1/120 + z (-1/5040 + z (1/9! - z / 11! + z^2 / 13! - z^3 / 15!))))
    float t = __fmaf_rn(z.h, -7.6471637e-13f, 1.6059044e-10f);
    t = __fmaf_rn(z.h, t, -2.5052108e-8f);
    t = __fmaf_rn(z.h, t, 2.7557319e-6f);
    P s = add(P{-0x1.a01a02p-13f, 0x1.7f97fap-39f}, mul(z, t));
    s = add(P{0x1.111112p-7f, -0x1.dddddep-32f}, mul(z, s));
    s = add(P{-0x1.555556p-3f, 0x1.555556p-28f}, mul(z, s));
    s = add(y, mul(mul(y, z), s));
    // cosine: 1 + z (-1/2 + z (1/24 + z (-1/720 + z (1/8! - z / 10! + z^2 / 12! - z^3 / 14! + z^4 / 16!))))
    float v = __fmaf_rn(z.h, 4.7794773e-14f, -1.1470746e-11f);
    v = __fmaf_rn(z.h, v, 2.0876757e-9f);
    v = __fmaf_rn(z.h, v, -2.7557319e-7f);
    P c = add(P{0x1.a01a02p-16f, -0x1.7f97fap-42f}, mul(z, v));
    c = add(P{-0x1.6c16c2p-10f, 0x1.27d27ep-35f}, mul(z, c));
    c = add(P{0x1.555556p-5f, -0x1.555556p-30f}, mul(z, c));
    c = add(P{-0.5f, 0.0f}, mul(z, c));
    c = add(P{1.0f, 0.0f}, mul(z, c));
    // cos phi and sin phi are +-cos y, +-sin y by the quadrant
    const int q = (int)k & 3;
    P cp = (q & 1) ? s : c, sp = (q & 1) ? c : s;
    if (q == 1 || q == 2) cp = P{-cp.h, -cp.l};
    if (q >= 2) sp = P{-sp.h, -sp.l};
    float2 out;
    // a sine or cosine next to its zero, or a radius next to 0, could lose bits to underflow
    const bool a = rounds(mul(cp, r), kRelCircle, out.x), b = rounds(mul(sp, r), kRelCircle, out.y);
    if (a && b && fabsf(out.x) > 1e-20f && fabsf(out.y) > 1e-20f) return out;
    return circle_double(r, phi);
}

static __device__ __noinline__ float quotient_double(float e, float a, float c)
{
    return (float)((double)e / (3.14159265358979323846 * (double)a * (double)a * (double)c));
}

// (float)(e / (pi * a * a * c)) evaluated in double; the range test keeps the residuals clear of underflow.
__device__ __forceinline__ float quotient_by_pi(float e, float a, float c)
{
    const P d = mul(mul(mul(P{kPi0, kPi1}, a), a), c);
    if (e == 0.0f && d.h > 1e-12f && d.h < 1e12f) return e;
    if (e > 1e-20f && e < 1e20f && d.h > 1e-12f && d.h < 1e12f) {
        const float i = __frcp_rn(d.h), q = __fmul_rn(e, i);
        const float res = __fmaf_rn(-q, d.l, __fmaf_rn(-q, d.h, e));
        float out;
        if (rounds(fast_sum(q, __fmul_rn(res, i)), kRelQuotient, out)) return out;
    }
    return quotient_double(e, a, c);
}

}  // namespace pair
}  // namespace pico
