"""Cut-cell sweeps at the edges of their tiles (GPU, against oracle/ccm_oracle.c).

Grids with partial tiles in both directions, bodies small enough to lie within
one tile, across a tile corner and along a whole tile row (the tile's list of
cut cells from a handful to several rows of it), and a ghost width other than
two, with which no tile is staged by the tensor copy; a gas in motion, so that
every component has a scale.  FP64 state of the
updated cells within 1e-12 relative after 12 steps, the bar of the cut-cell
parity test; the FP32 form's density within 1e-5 (L1) of FP64."""
import numpy as np
import pytest

ib = pytest.importorskip("ibtfo_gb300")
oracle = pytest.importorskip("oracle")
from ibtfo_gb300 import cases  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_x,n_y,ng,bodies", [
    (131, 77, 2, [(0.5, 0.3, 0.03), (0.99, 0.25, 0.05)]),     # inside a tile; across the corner of four
    (96, 48, 2, [(0.75, 0.25, 0.2)]),                          # whole tiles, many cut cells in each
    (65, 33, 2, [(0.7, 0.26, 0.1)]),                           # one column and one row beyond whole tiles
    (70, 40, 3, [(0.6, 0.3, 0.12)]),
])
def test_tile_edges(n_x, n_y, ng, bodies):
    hi = (1.5, 1.5 * n_y / n_x)
    g = cases.Grid(n_x, n_y, ng, 0.0, 0.0, *hi)
    phi = np.full(g.M * g.N, 1e300)
    for b in bodies:
        phi = np.minimum(phi, cases.cylinder_phi(g, *b))
    rho = {}
    o = oracle.CcmOracle(n_x, n_y, ng, (0, 0), hi, 1.4, 0.3, 1e300, "MUSCL", "HLL_Toro", "minmod", "walls")
    for precision in ("fp64_fast", "fp32c"):
        with ib.Case(n_x, n_y, ng=ng, lo=(0, 0), hi=hi, cfl=0.3, t_end=1e300, max_iter=2 ** 31 - 1,
                     riemann="HLL_Toro", boundary="CCM", precision=precision) as c:
            c.setup_geometry(phi)
            t = c.cell_types()
            x, y = g.coords()
            r = 1.0 + 0.2 * np.sin(5 * x) * np.cos(7 * y)
            u0 = cases.conserved(r, 0.6, 0.25, 1.0 + 0.1 * r, 1.4)
            u0 = cases._solid_fill(np.ascontiguousarray(u0), t.reshape(g.N, g.M)).reshape(-1)
            c.set_state(u0)
            c.advance(12)
            p = c.progress()
            assert p["iter"] == 12 and p["nan_cells"] == 0 and p["status"] == 0
            u = c.get_state().reshape(-1, 4)
        upd = (t == 0) | (t == 3)
        rho[precision] = u[upd, 0]
        if precision == "fp64_fast":
            o.setup(phi)
            o.set_state(u0)
            o.run(12)
            uo = o.get_state().reshape(-1, 4)
            for k in range(4):
                assert np.abs(u[upd, k] - uo[upd, k]).max() <= 1e-12 * np.abs(uo[upd, k]).max()
            assert abs(p["now_t"] - o.scalars()["now_t"]) <= 1e-12 * p["now_t"]
    d = rho["fp32c"] - rho["fp64_fast"]
    assert np.abs(d).sum() <= 1e-5 * np.abs(rho["fp64_fast"]).sum()
