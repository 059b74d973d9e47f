// scaled.h -- the numbers the sweeps run on: (1 + x.x) * 2^-x.y with x.y a whole number, +inf for zero (a dead
// state or edge), and the sums of exponentials of the posterior pass.  Plain arithmetic, compiled for the
// device by the kernels and for the host by tests/test_scaled_numbers.py, which holds it against doubles.
//
// The mantissa is kept as its distance from one: a score s near zero, the negative log of a probability near
// one, becomes x.x = expm1(-s) with the relative precision of s itself.  As a plain mantissa 1 - s it would be
// rounded to 2^-24, and the sum over the frames of a model that is sure of its labels (a whole sequence at a
// negative log of 1e-3) would be lost in those roundings: 4e-4 of it for 50 frames, where sums of logarithms
// lose 1e-7.  The exponent is a float so that +inf needs no special case and scores of any magnitude fit
// (above 2^24 its spacing exceeds one, as the spacing of a score of that magnitude does).
#pragma once
#include <math.h>
#include <string.h>

#ifdef __CUDACC__
#define FBW_HD __host__ __device__ __forceinline__
#else
#define FBW_HD static inline
struct float2 { float x, y; };
static inline float2 make_float2(float x, float y) { float2 r = {x, y}; return r; }
#endif

FBW_HD unsigned float_bits(float x) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(x);
#else
    unsigned u;
    memcpy(&u, &x, 4);
    return u;
#endif
}
FBW_HD float bits_float(unsigned u) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float x;
    memcpy(&x, &u, 4);
    return x;
#endif
}

#define FBW_INF bits_float(0x7f800000u)

// expm1(y) for |y| <= 0.52: y + y^2 P(y), P fitted by linear programming to a relative error of 3.1e-10 for
// |y| <= 0.36 (the remainders of to_scaled; beyond lie scores above 2^20 only, whose own spacing is larger)
FBW_HD float expm1_near_zero(float y) {
    float p = fmaf(1.99207249e-4f, y, 1.39451124e-3f);
    p = fmaf(p, y, 8.33326145e-3f);
    p = fmaf(p, y, 4.16663036e-2f);
    p = fmaf(p, y, 1.66666669e-1f);
    p = fmaf(p, y, 0.5f);
    return fmaf(y * y, p, y);
}

// log1p(x) for -0.25 <= x <= 0.5: x - x^2 Q(x), Q fitted the same way to a relative error of 5.0e-9
FBW_HD float log1p_near_zero(float x) {
    float q = fmaf(0.0450432624f, x, -0.104773388f);
    q = fmaf(q, x, 0.131797821f);
    q = fmaf(q, x, -0.144835828f);
    q = fmaf(q, x, 0.166463173f);
    q = fmaf(q, x, -0.199903390f);
    q = fmaf(q, x, 0.250000843f);
    q = fmaf(q, x, -0.333334600f);
    q = fmaf(q, x, 0.500000007f);
    return fmaf(-x * x, q, x);
}

// exp(-s) of a negative log score below kPlainScore in magnitude: s is split into a whole multiple of log 2 (the
// rounding of an addition to 1.5 * 2^23) and a remainder, formed with fused multiply-adds and log 2 in two
// parts.  The mantissa is 0.70 .. 1.42.
constexpr float kPlainScore = 2.0e6f;
FBW_HD float2 plain_to_scaled(float s) {
    const float c = fmaf(s, 1.44269502f, 12582912.f) - 12582912.f;
    float r = fmaf(c, -0.693147182f, s);
    r = fmaf(c, 1.90465421e-9f, r);
    return make_float2(expm1_near_zero(-r), c);
}
// The same for any score: +inf and NaN give zero, finite scores beyond the exponent's range saturate and stay
// finite.
FBW_HD float2 to_scaled(float s) {
    if (fabsf(s) < kPlainScore) return plain_to_scaled(s);
    const float c = rintf(fminf(fmaxf(s * 1.44269502f, -3.4e38f), 3.4e38f));
    float r = fmaf(c, -0.693147182f, s);
    r = fmaf(c, 1.90465421e-9f, r);
    r = fminf(fmaxf(r, -0.52f), 0.52f);
    return make_float2(expm1_near_zero(-r), s < FBW_INF ? c : FBW_INF);
}

// x of the product of two mantissas: (1 + a)(1 + b) - 1
FBW_HD float mul_scaled(float a, float b) { return fmaf(a, b, a + b); }

// 2^d for a whole number d <= 0; zero below 2^-126 and for NaN (the difference of two +inf)
FBW_HD float pow2_neg(float d) { return bits_float(float_bits(fmaxf(d, -127.f) + 8388735.f) << 23); }

// adds (1 + p) * 2^-k to (1 + x) * 2^-c; the exponent of the sum is the smaller one, its mantissa is not
// brought into range.  The term with the smaller exponent keeps its distance from one.
FBW_HD void add_scaled(float& x, float& c, float p, float k) {
    const bool  lead = c <= k;
    const float e = pow2_neg(-fabsf(c - k));
    const float other = lead ? p : x;
    x = (lead ? x : p) + fmaf(e, other, e);
    c = fminf(c, k);
}

// (1 + x) * 2^-c with the mantissa brought into [0.75, 1.5); the mantissa must be a normal positive number
FBW_HD float2 normalised(float x, float c) {
    const unsigned u = float_bits(1.f + x) + 0x00400000u;            // exponent of the nearest power of two
    const float  inv = bits_float(0x7f000000u - (u & 0xff800000u));  // 2^-n
    return make_float2(fmaf(x, inv, inv - 1.f), c - (bits_float(0x4b000000u | (u >> 23)) - 8388735.f));
}

// the natural negative log of a normalised number
FBW_HD float from_scaled(float2 v) {
    return v.y < 3.4e38f ? fmaf(v.y, 0.693147181f, -log1p_near_zero(v.x)) : v.y;
}
