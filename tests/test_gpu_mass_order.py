"""The mass of a step has the same bits whichever way the step is taken (GPU):
device steps (16x8 tiles on small grids and with PVRS, the case's tiles longest
first otherwise) and host-array steps (the case's tiles in row order, by bands).

Strict and fp64_fast, every solver with its own tiles, sizes at the edges of the tiles
and on either side of the number of 32x16 tiles up to which the device steps take
the small ones, with a body; one case stepped both ways in turn."""
import numpy as np
import pytest

ib = pytest.importorskip("ibtfo_gb300")
from ibtfo_gb300 import cases  # noqa: E402

pytestmark = pytest.mark.gpu


def make(n_x, n_y, body, scheme, riemann, precision):
    g = cases.Grid(n_x, n_y, 2, 0.0, 0.0, 1.0, n_y / n_x)
    c = ib.Case(n_x, n_y, lo=(0, 0), hi=(g.hi_x, g.hi_y), cfl=0.4, t_end=1e300, max_iter=2 ** 31 - 1, scheme=scheme,
                riemann=riemann, boundary="HBCGFM" if body else "Regular", precision=precision)
    x, y = g.coords()
    phi = cases.cylinder_phi(g, 0.55, 0.5 * g.hi_y, 0.3 * g.hi_y) if body else np.ones(g.N * g.M)
    c.setup_geometry(phi)
    wave = 0.2 * np.sin(7 * x) * np.cos(5 * y)
    u = cases.conserved(1.0 + wave, 0.3 + wave, 0.1 - wave, 1.0 + 0.5 * wave, 1.4)
    c.set_state(cases._solid_fill(u, c.cell_types().reshape(g.N, g.M)).reshape(-1))
    return c


@pytest.mark.parametrize("n_x,n_y,body,scheme,riemann,precision", [
    (2, 2, False, "MUSCL", "PVRS", "fp64"),
    (31, 17, False, "MUSCL", "PVRS", "fp64"),
    (161, 97, True, "MHM", "PVRS", "fp64"),
    (300, 151, False, "MUSCL", "PVRS", "fp64_fast"),
    (33, 9, False, "Godunov", "HLL", "fp64"),
    (161, 97, True, "MUSCL", "HLL", "fp64"),
    (511, 255, False, "MUSCL", "StegerWarming", "fp64"),      # 256 32x16 tiles
    (700, 401, True, "MHM", "HLL_Toro", "fp64"),              # 32x16 on the device too
    (700, 401, True, "MUSCL", "HLL", "fp64_fast"),
    (200, 120, True, "MUSCL", "HLLC_Toro", "fp64_fast"),
    (130, 70, False, "Lax", "HLL", "fp64"),
])
def test_mass_of_host_steps(n_x, n_y, body, scheme, riemann, precision):
    key = (n_x, n_y, body, scheme, riemann, precision)
    with make(*key) as a, make(*key) as b, make(*key) as both:
        u = np.ascontiguousarray(b.get_state().reshape(-1))
        w = np.ascontiguousarray(both.get_state().reshape(-1))
        for step in range(4):
            a.advance(1)
            want = a.progress()
            assert b.step_host_ptr(u.ctypes.data, u.ctypes.data) == want
            if step % 2:
                both.advance(1)
                assert both.progress() == want
                w = np.ascontiguousarray(both.get_state().reshape(-1))
            else:
                assert both.step_host_ptr(w.ctypes.data, w.ctypes.data) == want
        assert np.array_equal(a.get_state().reshape(-1), u) and np.array_equal(both.get_state().reshape(-1), u)
        assert want["iter"] == 4 and want["nan_cells"] == 0
