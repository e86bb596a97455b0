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


FLOOR = r"""
#include "physics_fast64.cuh"
using namespace ibtfo;
static std::mt19937_64 rg(6);
static double u01() { return (double)(rg() >> 11) * 0x1p-53; }
// the floor as stated: E becomes (E - e) + f where the density is positive and not e >= f = 1e-5 |E|
static double plain(const double *U, double e)
{
    const double f = 1e-5 * std::fabs(U[3]);
    return U[0] > 0 && !(e >= f) ? (U[3] - e) + f : U[3];
}
static bool same(double a, double b) { return double_bits(a) == double_bits(b) || (a != a && b != b); }
int main()
{
    const double odd[] = {NAN, INFINITY, -INFINITY, 0.0, -0.0, -1.0, 1e300, 1e-300};
    long bad = 0;
    for (int i = 0; i < 400000; i++)
    {
        const double r = 1 + u01(), u = 3 * (2 * u01() - 1), v = 3 * (2 * u01() - 1), k = 0.5 * r * (u * u + v * v);
        double U[4] = {r, r * u, r * v, k * (1 + std::pow(10.0, -8 * u01()) * (i % 3 ? 1 : -1))};
        if (i % 4 == 0) U[rg() % 4] = odd[rg() % 8];
        Cell64 c = cell64(U);
        const double e = c.ei, want = plain(U, e), f = 1e-5 * std::fabs(U[3]);
        pressure_floor64(U, c);
        bad += !same(U[3], want);
        // the internal energy of the statistics: the floor's where it raised E, NaN for a cell that is NaN
        bad += want != want ? c.ei == c.ei : !same(c.ei, same(want, U[3]) && U[0] > 0 && !(e >= f) ? f : e);
    }
    printf("%ld", bad);
}
"""


def test_pressure_floor(tmp_path):
    assert device_on_host.run(device_on_host.build(tmp_path, FLOOR)) == b"0"
