"""The FP32 difference form's faces, solved two at a time (GPU).

FP32 (HLL_Toro) against fp64_fast over a few steps of smooth flow, at sizes
where a pair has one face (odd rows and columns), at the edges of the 32x16
tile, at the smallest grid, with a body whose tiles solve a list of pairs, and
with more tiles than CTAs (a CTA sweeps several).

The bar: one step moves a cell by at most CFL x the jump to its neighbour,
under 0.2 of the scale here; its increment passes about a hundred FP32
roundings of 6e-8, which add to at most 16 of them (1e-6 of the increment,
2e-7 of the scale); six steps of two stages at most, 2.4e-6.  A face read from
or written to a wrong place changes cells by the jump, 1e-3 and more."""
import numpy as np
import pytest

ib = pytest.importorskip("ibtfo_gb300")
from ibtfo_gb300 import cases  # noqa: E402

pytestmark = pytest.mark.gpu
BAR = 2.4e-6


def run(n_x, n_y, body, scheme, time, precision):
    g = cases.Grid(n_x, n_y, 2, 0.0, 0.0, 1.0, n_y / n_x)
    with ib.Case(n_x, n_y, lo=(0, 0), hi=(g.hi_x, g.hi_y), cfl=0.4, t_end=1e300, max_iter=2 ** 31 - 1, scheme=scheme,
                 riemann="HLL_Toro", boundary="IDWBaseGFM" if body else "Regular", precision=precision, time=time) as c:
        x, y = g.coords()
        phi = cases.cylinder_phi(g, 0.55, 0.5 * g.hi_y, 0.3 * g.hi_y) if body else np.ones(g.N * g.M)
        c.setup_geometry(phi)
        wave = 0.2 * np.sin(7 * x) * np.cos(5 * y)
        u = cases.conserved(1.0 + wave, 0.3 + wave, 0.1 - wave, 1.0 + 0.5 * wave, 1.4)
        c.set_state(cases._solid_fill(u, c.cell_types().reshape(g.N, g.M)).reshape(-1))
        fluid = c.cell_types() == 0
        c.advance(6)
        assert c.progress()["nan_cells"] == 0
        return c.get_state().reshape(-1, 4)[fluid]


@pytest.mark.parametrize("n_x,n_y,body,scheme,time", [
    (2, 2, False, "MUSCL", "SingleStep"),
    (31, 15, False, "MUSCL", "RK2"),
    (32, 16, False, "Godunov", "SingleStep"),
    (33, 17, False, "MHM", "RK2"),
    (65, 49, False, "MHM", "SingleStep"),
    (161, 97, True, "MUSCL", "RK2"),
    (160, 96, True, "MHM", "RK2"),
    (961, 500, False, "MUSCL", "RK2"),   # 992 tiles
])
def test_pairs_track_fp64(n_x, n_y, body, scheme, time):
    a = run(n_x, n_y, body, scheme, time, "fp32c")
    b = run(n_x, n_y, body, scheme, time, "fp64_fast")
    assert np.isfinite(a).all()
    assert np.abs(a - b).max() <= BAR * np.abs(b).max()
