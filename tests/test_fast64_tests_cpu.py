"""The comparisons of the fp64_fast faces and cells that read bit patterns
(csrc/physics_fast64.cuh), compiled for the host, with signed overflow trapped:
what they give for zeros, negative values, infinities and NaN."""
import device_on_host

TWICE = r"""
#include "physics_fast64.cuh"
using namespace ibtfo;
static std::mt19937_64 rg(5);
static double normal(bool sign)
{
    return bits_double(((uint64_t)(1 + rg() % 2046) << 52) | (rg() & ((1ull << 52) - 1)) | (sign ? rg() & (1ull << 63) : 0));
}
int main()
{
    const double inf = INFINITY, nan = bits_double(0x7ff8000000000000ull), nan_max = bits_double(0x7fffffffffffffffull);
    long bad = 0;
    for (double w : {0.0, 2.2250738585072014e-308, 1.0, 1.79e308, inf})
    {
        bad += exceeds_twice(w, inf) + exceeds_twice(w, nan) + exceeds_twice(w, nan_max);
        for (double p : {-0.0, -5e-324, -1.0, -1.79e308}) bad += !exceeds_twice(w, p);
    }
    bad += exceeds_twice(0.0, 0.0) + !exceeds_twice(inf, 8e307) + exceeds_twice(inf, 1e308) + !exceeds_twice(1.0, 0.0);
    for (int i = 0; i < 1000000; i++)
    {
        const double w = normal(false);
        double p = normal(true);
        if (i % 2) p = bits_double(double_bits(0.5 * w) + (rg() % 5) - 2); // next to w / 2
        if (std::fabs(p) < 2.3e-308) continue;
        bad += exceeds_twice(w, p) != (0.5L * w > (long double)p);
    }
    printf("%ld", bad);
}
"""


def test_exceeds_twice(tmp_path):
    exe = device_on_host.build(tmp_path, TWICE, "-fsanitize=signed-integer-overflow", "-fsanitize-undefined-trap-on-error")
    assert device_on_host.run(exe) == b"0"
