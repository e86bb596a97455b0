"""The integer-pipe reciprocal, square root and quotient of
ibtfo_gb300/csrc/int64math.cuh, compiled for the host.

The FP32 hardware estimates are stood in for by the rounded value moved by up
to three units in the last place (the hardware's are within two).  Bounds, from
the scheme: the estimate is good to 2^-59 of the result before it is rounded
to 53 bits, so rcp_int and sqrt_int lie within 1/2 + 2^-6 ulp; sqrt_rn_int and
divide_rn are the IEEE values, whatever the arguments (special values, results
at the ends of the exponent range, significands of all ones or zeros, and
dividends next to a divisor times a half-way point)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
static int off = 0;
#define IBTFO_DEVICE static inline
namespace ibtfo {
IBTFO_DEVICE uint64_t double_bits(double x) { uint64_t i; memcpy(&i, &x, 8); return i; }
IBTFO_DEVICE double bits_double(uint64_t i) { double x; memcpy(&x, &i, 8); return x; }
IBTFO_DEVICE uint32_t float_bits(float x) { uint32_t i; memcpy(&i, &x, 4); return i; }
IBTFO_DEVICE float bits_float(uint32_t i) { float x; memcpy(&x, &i, 4); return x; }
IBTFO_DEVICE float rcp_estimate(float x) { return bits_float(float_bits(1.0f / x) + off); }
IBTFO_DEVICE float rsqrt_estimate(float x) { return bits_float(float_bits((float)(1.0 / sqrt((double)x))) + off); }
IBTFO_DEVICE int round_int(float x) { if (!(fabsf(x) < 2147483000.0f)) { puts("overflow"); exit(1); } return (int)rintf(x); }
IBTFO_DEVICE uint64_t mul_high(uint64_t a, uint64_t b) { return (uint64_t)(((unsigned __int128)a * b) >> 64); }
IBTFO_DEVICE double divide_hardware(double a, double b) { return a / b; }
}
#include "int64math.cuh"
using namespace ibtfo;
static uint64_t state = 88172645463325252ull;
static uint64_t rnd() { state ^= state << 13; state ^= state >> 7; state ^= state << 17; return state; }
static uint64_t mantissa()
{
    const uint64_t all = (1ull << 52) - 1;
    uint64_t m = rnd() & all;
    switch (rnd() % 8)
    {
    case 0: return (rnd() % 64) * (rnd() % 3);
    case 1: return all - rnd() % 64;
    case 2: return m & ~((1ull << 29) - 1);
    case 3: return m | ((1ull << 29) - 1);
    case 4: return (~0ull << (rnd() % 52)) & all;
    default: return m;
    }
}
static double number(int lo, int hi) { return bits_double(((uint64_t)(lo + rnd() % (hi - lo)) << 52) | mantissa() | (rnd() << 63)); }
static double ulps(long double got, long double want) { int e; frexpl(want, &e); return (double)(fabsl(got - want) / ldexpl(1.0L, e - 53)); }
int main(int argc, char **argv)
{
    const long n = atol(argv[1]);
    const double special[] = {0.0, -0.0, INFINITY, -INFINITY, NAN, 5e-324, 1e-310, 2.2250738585072014e-308, 1.79e308};
    double worst_rcp = 0, worst_sqrt = 0;
    for (long i = 0; i < n; i++)
    {
        off = (int)(rnd() % 7) - 3;
        double x = number(2, 2043);
        if (!rcp_range(double_bits(x))) { printf("range %a\n", x); return 1; }
        worst_rcp = fmax(worst_rcp, ulps(rcp_int(double_bits(x)), 1.0L / (long double)x));
        x = fabs(number(1, 2047));
        if (!sqrt_range(double_bits(x))) { printf("range %a\n", x); return 1; }
        worst_sqrt = fmax(worst_sqrt, ulps(sqrt_int(double_bits(x)), sqrtl((long double)x)));
        if (sqrt_rn_int(double_bits(x)) != sqrt(x)) { printf("sqrt %a\n", x); return 1; }
        double a = i & 1 ? number(1, 2047) : number(1000, 1040), b = i & 2 ? number(1, 2047) : number(1000, 1040);
        if (i % 16 == 0) (rnd() & 1 ? a : b) = special[rnd() % 9];
        if (i % 5 == 0) a = (double)(((long double)(mantissa() | (1ull << 52)) + 0.5L) * 0x1p-52L * (long double)b);
        const double q = divide_rn(a, divisor(b)), want = a / b;
        if (double_bits(q) != double_bits(want) && !(std::isnan(q) && std::isnan(want))) { printf("divide %a %a: %a, not %a\n", a, b, q, want); return 1; }
    }
    printf("%.6f %.6f\n", worst_rcp, worst_sqrt);
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_reciprocals_roots_and_quotients(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "ibtfo_gb300", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    p = subprocess.run([str(exe), "3000000"], capture_output=True, text=True)
    assert p.returncode == 0, p.stdout
    rcp, sqrt = map(float, p.stdout.split())
    # long double has 64 bits here or more, 11 beyond a double's
    assert rcp <= 0.5 + 2 ** -6 + 2 ** -10 and sqrt <= 0.5 + 2 ** -6 + 2 ** -10
