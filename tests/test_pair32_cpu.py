"""Doubles to (hi, lo) float pairs and back on integers
(ibtfo_gb300/csrc/pair32.cuh), compiled for the host: bit for bit the values
of the conversions they stand for, over random bits, ties, special values and
the ends of the ranges handed to the hardware."""
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
#include <random>
#define IBTFO_DEVICE static inline
struct float2 { float x, y; };
namespace ibtfo {
IBTFO_DEVICE uint64_t double_bits(double x) { uint64_t i; memcpy(&i, &x, 8); return i; }
IBTFO_DEVICE double bits_double(uint64_t i) { double x; memcpy(&x, &i, 8); return x; }
IBTFO_DEVICE uint32_t float_bits(float x) { uint32_t i; memcpy(&i, &x, 4); return i; }
IBTFO_DEVICE float bits_float(uint32_t i) { float x; memcpy(&x, &i, 4); return x; }
IBTFO_DEVICE float rcp_estimate(float x) { return 1.0f / x; }
IBTFO_DEVICE float rsqrt_estimate(float x) { return 1.0f / sqrtf(x); }
IBTFO_DEVICE int round_int(float x) { return (int)rintf(x); }
IBTFO_DEVICE uint64_t mul_high(uint64_t a, uint64_t b) { return (uint64_t)(((unsigned __int128)a * b) >> 64); }
IBTFO_DEVICE double divide_hardware(double a, double b) { return a / b; }
IBTFO_DEVICE double widen_hardware(float f) { return (double)f; }
IBTFO_DEVICE float2 split_hardware(double v) { const float h = (float)v; return {h, (float)(v - (double)h)}; }
}
#include "pair32.cuh"
using namespace ibtfo;
static bool same(float a, float b) { return float_bits(a) == float_bits(b) || (std::isnan(a) && std::isnan(b)); }
static long bad = 0;
static void check(double v)
{
    float hi, lo;
    split_pair(v, hi, lo);
    const float h = (float)v, l = (float)(v - (double)h);
    if (!same(hi, h) || !same(lo, l)) bad++;
}
static void check(float f)
{
    const double a = widen(f), b = (double)f;
    if (double_bits(a) != double_bits(b) && !(std::isnan(a) && std::isnan(b))) bad++;
}
int main(int argc, char **argv)
{
    std::mt19937_64 g(3);
    const long n = atol(argv[1]);
    for (long i = 0; i < n; i++)
    {
        uint64_t x = g();
        if (i % 3 == 1) x = (x & ~(0x7ffull << 52)) | ((940ull + g() % 220) << 52);
        if (i % 3 == 2) x = (x & ~((1ull << (g() % 40)) - 1) & ~(0x7ffull << 52)) | ((1000ull + g() % 40) << 52);
        check(bits_double(x));
        check(bits_float((uint32_t)(x >> 16)));
    }
    for (int e = 0; e < 2048; e++)
        for (uint64_t m : {0ull, 1ull, 0x10000000ull, 0x10000001ull, 0x0fffffffull, 0x30000000ull, (1ull << 52) - 1})
            for (uint64_t s : {0ull, 1ull}) check(bits_double((s << 63) | ((uint64_t)e << 52) | m));
    for (uint32_t e = 0; e < 256; e++)
        for (uint32_t m : {0u, 1u, 0x7fffffu})
            for (uint32_t s : {0u, 1u}) check(bits_float((s << 31) | (e << 23) | m));
    printf("%ld\n", bad);
    return bad != 0;
}
"""


@pytest.mark.parametrize("n", [6000000])
def test_pairs_are_the_conversions(tmp_path, n):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host compiler")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "ibtfo_gb300", "csrc"), "-o",
                    str(exe), str(src)], check=True)
    assert subprocess.run([str(exe), str(n)], stdout=subprocess.PIPE, text=True, check=True).stdout.split() == ["0"]
