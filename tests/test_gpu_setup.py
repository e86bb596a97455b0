"""Geometry set-up does its work once (GPU): kernels launched by
ibtfo_setup_geometry, the tile counts of all tilings a case needs among them, and the
tile lists it leaves (the results of the steps that follow)."""
import numpy as np
import pytest

ib = pytest.importorskip("ibtfo_gb300")
from ibtfo_gb300 import cases  # noqa: E402

pytestmark = pytest.mark.gpu


def make(n_x, n_y, riemann, precision, boundary="Regular"):
    g = cases.Grid(n_x, n_y, 2, 0.0, 0.0, 1.0, n_y / n_x)
    c = ib.Case(n_x, n_y, lo=(0, 0), hi=(g.hi_x, g.hi_y), cfl=0.4, t_end=1e300, max_iter=2 ** 31 - 1,
                scheme="MUSCL", riemann=riemann, boundary=boundary, precision=precision, time="SingleStep")
    return g, c


# normals, cell types, and one count for each tiling the steps use: the case's
# tiles; 16x8 on grids of few tiles; with PVRS also the 32x16 tiles that group the mass sums
@pytest.mark.parametrize("n_x,n_y,riemann,precision,launches", [
    (64, 48, "HLL", "fp64", 4),
    (700, 400, "HLL", "fp64_fast", 4),     # 550 tiles: counted with the others, none used
    (2048, 1024, "HLL", "fp64", 3),        # 4096 tiles
    (512, 256, "HLL", "fp32c", 3),
    (96, 64, "PVRS", "fp64", 5),
])
def test_launches_of_the_setup(n_x, n_y, riemann, precision, launches):
    g, c = make(n_x, n_y, riemann, precision)
    with c:
        before = ib.launch_count()
        c.setup_geometry(np.ones(g.N * g.M))
        assert ib.launch_count() - before == launches


def test_few_active_tiles_of_a_large_grid():
    """A narrow channel of a 2048x1024 grid (4096 tiles, fewer than 256 active) sweeps the
    16x8 tiles, a wide one the case's own; both are what the same case gives from new
    geometry after another was set up."""
    for width in (0.012, 0.4):
        g, c = make(2048, 1024, "HLL", "fp64_fast", "IDWBaseGFM")
        x, y = g.coords()
        phi = np.broadcast_to(0.5 * width - np.abs(y - 0.25), (g.N, g.M)).reshape(-1).copy()
        r = 1.0 + 0.2 * np.sin(9 * x) * np.ones_like(y)
        out = []
        with c:
            for other in (False, True):
                if other:
                    c.setup_geometry(np.ones(g.N * g.M))
                c.setup_geometry(phi)
                u = cases.conserved(r, 0.3, 0.0, 1.0 + 0.1 * r, 1.4)
                c.set_state(cases._solid_fill(u, c.cell_types().reshape(g.N, g.M)).reshape(-1))
                c.advance(3)
                out.append((c.get_state(), c.progress()))
        assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]
        assert out[0][1]["iter"] == 3 and out[0][1]["nan_cells"] == 0
