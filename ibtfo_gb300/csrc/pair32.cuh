// Doubles and (hi, lo) pairs of floats into each other, on the integer and
// FP32 pipes: the conversion instructions share the FP64 unit, which takes 16
// clocks for each warp instruction, and a pair costs three of them each way.
// Same results, bit for bit; numbers outside the stated ranges go to the
// hardware's conversions, in calls.
#pragma once

#include "int64math.cuh"

namespace ibtfo {

#ifdef __CUDACC__
static __device__ __noinline__ double widen_hardware(float f) { return (double)f; }
static __device__ __noinline__ float2 split_hardware(double v)
{
    const float hi = (float)v;
    return make_float2(hi, (float)(v - (double)hi));
}
#endif

// (double)f
IBTFO_DEVICE double widen(float f)
{
    const uint32_t b = float_bits(f), m = b & 0x7fffffffu;
    if (m - 0x00800000u >= 0x7f000000u) // not a normal number
    {
        if (m == 0)
            return bits_double((uint64_t)b << 32);
        return widen_hardware(f);
    }
    const uint32_t high = (b & 0x80000000u) | ((m >> 3) + 0x38000000u);
    return bits_double(((uint64_t)high << 32) | (uint32_t)(b << 29));
}

// hi = (float)v, lo = (float)(v - hi); |v| in [2^-74, 2^127) or zero.  The
// significand's upper 24 bits rounded to even are hi's, and what that leaves
// (29 bits, signed) lo's.
IBTFO_DEVICE void split_pair(double v, float &hi, float &lo)
{
    const uint64_t b = double_bits(v);
    const uint32_t bh = (uint32_t)(b >> 32), bl = (uint32_t)b, sign = bh & 0x80000000u;
    const uint32_t e = (bh >> 20) & 0x7ffu;
    if (e - 949u > 200u)
    {
        if ((b << 1) == 0)
        {
            hi = bits_float(sign);
            lo = 0.0f;
            return;
        }
        const float2 p = split_hardware(v);
        hi = p.x;
        lo = p.y;
        return;
    }
    uint32_t q = 0x00800000u | ((bh & 0x000fffffu) << 3) | (bl >> 29);
    const uint32_t rest = bl & 0x1fffffffu;
    const uint32_t up = rest + (q & 1u) > 0x10000000u ? 1u : 0u;
    q += up;
    const int r = (int)rest - (int)(up << 29);
    hi = bits_float(sign | (q + ((e - 897u) << 23)));
    lo = (float)(sign ? -r : r) * bits_float((e - 948u) << 23);
}

} // namespace ibtfo
