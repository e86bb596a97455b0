// Reciprocals, quotients and square roots of doubles on the integer and FP32
// pipes.
//
// GB300 has one FP64 unit per SM, which takes 16 clocks for a warp
// instruction; in that time the SM's other pipes issue up to 64.  A division
// in FP64 instructions costs eight or nine of them, a root as many.  Here a
// significand X (53 bits) is worked on as a 64-bit integer:
//   * an FP32 estimate of 1/X (or of its root), corrected once in FP32 by its
//     residual, is good to about 44 bits;
//   * its exact residual against X is small, so the low 64 bits of an integer
//     product give it (three 32-bit multiplies), and one more FP32 correction
//     brings the estimate to 60 bits or more;
//   * rounding that to 53 bits is within 0.504 ulp (a root 0.508) of the value (rcp_t and
//     sqrt_t of the fast precisions); where IEEE rounding is needed (the
//     strict sweeps), the remainder of the rounded result, again exact in 64
//     bits, says whether its neighbour is nearer.
// No FP64 instruction is issued.  Arguments outside the ranges stated at each
// function (subnormal or non-finite values, results near the ends of the
// exponent range) go to the hardware's own operations.
// The scheme is Newton's iteration in fixed point with exact integer
// remainders (Brent and Zimmermann, Modern Computer Arithmetic, 2010, chapters
// 1 and 3).
#pragma once

#include <cstdint>

#ifndef IBTFO_DEVICE
#define IBTFO_DEVICE __device__ __forceinline__
#endif

namespace ibtfo {

#ifdef __CUDACC__
IBTFO_DEVICE float rcp_estimate(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
IBTFO_DEVICE float rsqrt_estimate(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
IBTFO_DEVICE uint64_t double_bits(double x) { return (uint64_t)__double_as_longlong(x); }
IBTFO_DEVICE double bits_double(uint64_t b) { return __longlong_as_double((long long)b); }
IBTFO_DEVICE float bits_float(uint32_t b) { return __uint_as_float(b); }
IBTFO_DEVICE uint32_t float_bits(float x) { return __float_as_uint(x); }
IBTFO_DEVICE int round_int(float x) { return __float2int_rn(x); }
IBTFO_DEVICE uint64_t mul_high(uint64_t a, uint64_t b) { return __umul64hi(a, b); }
// the rare arguments; calls, so that a face does not hold a copy of each
static __device__ __noinline__ double divide_hardware(double a, double b) { return a / b; }
static __device__ __noinline__ double sqrt_hardware(double x) { return sqrt(x); }
#endif

constexpr uint64_t SIG_HIDDEN = 1ull << 52;

// the 53-bit significand of a normal double
IBTFO_DEVICE uint64_t significand(uint64_t bits) { return (bits & (SIG_HIDDEN - 1)) | SIG_HIDDEN; }
IBTFO_DEVICE int exponent_field(uint64_t bits) { return (int)((uint32_t)(bits >> 52) & 0x7ffu); }

// the significand as a float mh (24 bits) and the next 23 bits, ml 2^-23
IBTFO_DEVICE float leading(uint64_t X) { return bits_float(0x3f800000u | ((uint32_t)(X >> 29) & 0x007fffffu)); }
IBTFO_DEVICE float following(uint64_t X) { return bits_float(0x3f800000u | (((uint32_t)X >> 6) & 0x007fffffu)) - 1.0f; }

// 2^114 / X for a significand X in [2^52, 2^53), within two units
IBTFO_DEVICE uint64_t reciprocal62(uint64_t X)
{
    const float mh = leading(X), ml = following(X);
    float y = rcp_estimate(mh);
    y = fminf(fmaxf(y, 0.5f), 0x1.fffffep-1f); // the binade [1/2, 1)
    const float e = fmaf(ml * -0x1p-23f, y, fmaf(-mh, y, 1.0f));
    // units of 2^-48: 24 bits of y and the correction y e, |y e| < 2^-21
    const uint64_t Y = ((uint64_t)((float_bits(y) & 0x007fffffu) | 0x00800000u) << 24) +
                       (uint64_t)(int64_t)round_int((y * e) * 0x1p48f);
    const int64_t T = (int64_t)(0ull - X * Y); // 2^100 - X Y, below 2^58
    const float d = (float)(int)(T >> 32);
    return (Y << 14) + (uint64_t)(int64_t)round_int((y * d) * 0x1p-6f);
}

// a biased exponent and a significand (2^52 ... 2^53) as a double's bits
IBTFO_DEVICE uint64_t assemble(uint64_t sig, int ex) { return sig + ((uint64_t)(int64_t)(ex - 1) << 52); }

// 1/x within half an ulp and two units of the estimate, 0.504 ulp (0.502 seen in 20 million); |x| in [2^-1021, 2^1020)
IBTFO_DEVICE bool rcp_range(uint64_t bits) { return (unsigned)exponent_field(bits) - 2u < 2041u; }
IBTFO_DEVICE double rcp_int(uint64_t bits)
{
    const uint64_t Y = reciprocal62(significand(bits));
    return bits_double(assemble((Y + 256) >> 9, 2045 - exponent_field(bits)) | (bits & (1ull << 63)));
}

// 2^60 sqrt(X2 / 2^52) for X2 in [2^52, 2^54), within two units; y receives the
// FP32 estimate of 1/sqrt
IBTFO_DEVICE uint64_t root60(uint64_t X, int odd)
{
    const float mh = bits_float(float_bits(leading(X)) + ((uint32_t)odd << 23));
    const float ml = following(X);
    const float y = rsqrt_estimate(mh);
    const float s = fminf(fmaxf(mh * y, 1.0f), 0x1.fffffep0f); // the binade [1, 2)
    const float r = fmaf(ml, odd ? 0x1p-22f : 0x1p-23f, fmaf(-s, s, mh));
    // units of 2^-46: 24 bits of s and the correction y r / 2, below 2^-20
    const uint64_t S = ((uint64_t)((float_bits(s) & 0x007fffffu) | 0x00800000u) << 23) +
                       (uint64_t)(int64_t)round_int((y * r) * 0x1p45f);
    const int64_t T = (int64_t)((X << (40 + odd)) - S * S); // 2^92 m - S^2, below 2^56
    const float d = (float)(int)(T >> 28);
    return (S << 14) + (uint64_t)(int64_t)round_int((y * d) * 0x1p-5f);
}

// sqrt(x) within half an ulp and two units, 0.508 ulp (0.503 seen); x positive and normal
IBTFO_DEVICE bool sqrt_range(uint64_t bits) { return (uint32_t)(bits >> 32) - 0x00100000u < 0x7fe00000u; }
IBTFO_DEVICE double sqrt_int(uint64_t bits)
{
    const int E = exponent_field(bits) - 1023;
    const uint64_t S = root60(significand(bits), E & 1);
    return bits_double(assemble((S + 128) >> 8, 1023 + (E >> 1)));
}

// sqrt(x) correctly rounded; x positive and normal.  With R = X 2^52 - S^2 the
// root lies above S + 1/2 exactly when R > S and below S - 1/2 when R <= -S.
IBTFO_DEVICE double sqrt_rn_int(uint64_t bits)
{
    const int E = exponent_field(bits) - 1023, odd = E & 1;
    const uint64_t X = significand(bits);
    uint64_t S = (root60(X, odd) + 128) >> 8;
    const int64_t R = (int64_t)((X << odd << 52) - S * S);
    S += (uint64_t)(int64_t)((R > (int64_t)S) - (R <= -(int64_t)S));
    return bits_double(assemble(S, 1023 + (E >> 1)));
}

// sqrt(x), IEEE for every x
#ifdef __CUDACC__
IBTFO_DEVICE double sqrt_rn(double x)
{
    const uint64_t b = double_bits(x);
    return sqrt_range(b) ? sqrt_rn_int(b) : sqrt_hardware(x);
}
#endif

// A divisor: its reciprocal serves every quotient by it.
struct Divisor
{
    double b;
    uint64_t B, Y; // significand, reciprocal62
    uint64_t sign;
    int ex;        // exponent field; 0 for a b that divide_rn hands to the hardware
};
IBTFO_DEVICE Divisor divisor(double b)
{
    Divisor d;
    const uint64_t bits = double_bits(b);
    d.b = b;
    d.B = significand(bits);
    d.Y = reciprocal62(d.B);
    d.ex = exponent_field(bits);
    if (d.ex == 0x7ff)
        d.ex = 0;
    d.sign = bits & (1ull << 63);
    return d;
}

// a / b correctly rounded (round to nearest; a quotient of two doubles is
// never half way between two).  Q, the quotient of the significands from the
// reciprocal, is the floor or one less of the 53-bit quotient; R = A 2^s - Q B
// is exact in 64 bits, and Q + 1 is nearer when 2 R > B.
IBTFO_DEVICE double divide_rn(double a, const Divisor &d)
{
    const uint64_t bits = double_bits(a);
    const int ea = exponent_field(bits);
    const uint64_t A = significand(bits);
    const int less = A < d.B ? 1 : 0;
    const int ex = ea - d.ex + 1023 - less;
    // a normal a and b, and a normal quotient away from both ends
    if (d.ex == 0 || (unsigned)(ea - 1) >= 0x7feu || (unsigned)(ex - 1) >= 0x7fcu)
    {
        if ((bits << 1) == 0 && d.ex != 0) // gas at rest: zero momenta and flux differences are common
            return bits_double(bits ^ d.sign);
        return divide_hardware(a, d.b);
    }
    const uint64_t Q = mul_high(A << (2 + less), d.Y);
    const int64_t R = (int64_t)((A << less << 52) - Q * d.B);
    const uint64_t q = Q + (2 * R > (int64_t)d.B ? 1 : 0);
    return bits_double(assemble(q, ex) | ((bits ^ d.sign) & (1ull << 63)));
}

} // namespace ibtfo
