"""The 16x8 tiles that the FP64 device steps of small grids sweep (GPU).

A case alone (16x8 tiles) against the same case in a batch of 32x16 tiles:
state, loop scalars and the mass sum bit for bit.  Sizes at the edges of both
tiles, one cell less and more, the smallest grid, and either side of the
number of 32x16 tiles up to which a case takes the small ones; with a body,
the tiles it leaves out and those it cuts."""
import numpy as np
import pytest

ib = pytest.importorskip("ibtfo_gb300")
from ibtfo_gb300 import cases  # noqa: E402

pytestmark = pytest.mark.gpu


def make(n_x, n_y, body, scheme, riemann, time):
    g = cases.Grid(n_x, n_y, 2, 0.0, 0.0, 1.0, n_y / n_x)
    c = ib.Case(n_x, n_y, lo=(0, 0), hi=(g.hi_x, g.hi_y), cfl=0.4, t_end=1e300, max_iter=2 ** 31 - 1, scheme=scheme,
                riemann=riemann, boundary="IDWBaseGFM" if body else "Regular", precision="fp64_fast", time=time)
    x, y = g.coords()
    phi = cases.cylinder_phi(g, 0.55, 0.5 * g.hi_y, 0.3 * g.hi_y) if body else np.ones(g.N * g.M)
    c.setup_geometry(phi)
    wave = 0.2 * np.sin(7 * x) * np.cos(5 * y)
    u = cases.conserved(1.0 + wave, 0.3 + wave, 0.1 - wave, 1.0 + 0.5 * wave, 1.4)
    c.set_state(cases._solid_fill(u, c.cell_types().reshape(g.N, g.M)).reshape(-1))
    return c


@pytest.mark.parametrize("n_x,n_y,body,scheme,riemann,time", [
    (2, 2, False, "MUSCL", "HLL", "SingleStep"),
    (15, 7, False, "MHM", "HLL", "SingleStep"),
    (16, 8, False, "MUSCL", "StegerWarming", "RK2"),
    (17, 9, False, "Godunov", "HLL", "SingleStep"),
    (33, 17, False, "MUSCL", "HLL_Toro", "RK2"),
    (61, 47, True, "MUSCL", "HLL", "SingleStep"),
    (160, 97, True, "MHM", "HLL_Toro", "SingleStep"),
    (511, 255, False, "MUSCL", "HLL", "SingleStep"),   # 256 32x16 tiles
    (512, 257, False, "MUSCL", "HLL", "SingleStep"),   # 272: the case's tiles are 32x16
])
def test_small_tiles_give_the_bits_of_32x16_tiles(n_x, n_y, body, scheme, riemann, time):
    with make(n_x, n_y, body, scheme, riemann, time) as a, make(n_x, n_y, body, scheme, riemann, time) as b:
        with ib.Batch(scheme=scheme, riemann=riemann, precision="fp64_fast", tile_shape="32x16", time=time) as batch:
            batch.add(b)
            for steps in (1, 5):
                a.advance(steps)
                batch.advance(steps)
                batch.synchronize()
                assert np.array_equal(a.get_state(), b.get_state())
                pa, pb = a.progress(), b.progress()
                assert pa == pb
            assert pa["iter"] == 6 and pa["nan_cells"] == 0
