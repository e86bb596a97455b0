"""The FP64 arithmetic of a cut cell (csrc/physics_fast64.cuh), compiled for the
host: wall length, unit normal and update bit for bit the IEEE expressions, over
volume fractions and apertures down to 1e-12, walls along an axis and no wall."""
import device_on_host

PROGRAM = r"""
#include "physics_fast64.cuh"
using namespace ibtfo;
static std::mt19937_64 rg(3);
static double u01() { return (double)(rg() >> 11) * 0x1p-53; }
static bool same(double a, double b) { return double_bits(a) == double_bits(b); }
int main(int, char **v)
{
    long bad = 0;
    for (long i = 0; i < atol(v[1]); i++)
    {
        const double al = std::pow(10.0, -12 * u01()), dx = 0.01 * (1 + u01()), dy = 0.01 * (1 + u01());
        double ax = std::pow(10.0, -12 * u01()) * (u01() < 0.5 ? -1 : 1), ay = (2 * u01() - 1) * ax;
        if (i % 8 == 0) ax = 0;
        if (i % 12 == 0) ay = 0;
        const double nLx = ax * dy, nLy = ay * dx, L = std::sqrt(nLx * nLx + nLy * nLy);
        const CutWall w = cut_wall(nLx, nLy);
        bad += !same(w.L, L);
        if (L > 0) bad += !same(w.nx, nLx / L) + !same(w.ny, nLy / L);
        const double U = 2 * u01(), fx = u01() - 0.5, gy = u01() - 0.5, W = u01(), lx = u01(), ly = u01(), lw = 50 * L;
        bad += !same(cut_update(divisor(al), U, lx, fx, ly, gy, lw, W), (al * U - lx * fx - ly * gy - lw * W) / al);
    }
    printf("%ld", bad);
}
"""


def test_cut_cell_arithmetic_is_ieee(tmp_path):
    assert device_on_host.run(device_on_host.build(tmp_path, PROGRAM), 1000000) == b"0"
