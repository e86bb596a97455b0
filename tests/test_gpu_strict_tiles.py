"""The strict sweeps' two tile sizes (GPU): 16x8 on grids of few tiles, 32x16
above and in the host-array step.

Device steps against host-array steps of the same case: state and loop scalars
bit for bit (every cell is the same sequence of IEEE operations whatever its
tile; the mass adds up over the same tree).  Sizes at the edges of both tiles,
the smallest grid, and either side of the number of 32x16 tiles up to which the
device steps take the small ones."""
import numpy as np
import pytest

ib = pytest.importorskip("ibtfo_gb300")
from ibtfo_gb300 import cases  # noqa: E402

pytestmark = pytest.mark.gpu


def make(n_x, n_y, body, scheme, riemann, time):
    g = cases.Grid(n_x, n_y, 2, 0.0, 0.0, 1.0, n_y / n_x)
    c = ib.Case(n_x, n_y, lo=(0, 0), hi=(g.hi_x, g.hi_y), cfl=0.4, t_end=1e300, max_iter=2 ** 31 - 1, scheme=scheme,
                riemann=riemann, boundary="IDWBaseGFM" if body else "Regular", precision="fp64", time=time)
    x, y = g.coords()
    phi = cases.cylinder_phi(g, 0.55, 0.5 * g.hi_y, 0.3 * g.hi_y) if body else np.ones(g.N * g.M)
    c.setup_geometry(phi)
    wave = 0.2 * np.sin(7 * x) * np.cos(5 * y)
    u = cases.conserved(1.0 + wave, 0.3 + wave, 0.1 - wave, 1.0 + 0.5 * wave, 1.4)
    c.set_state(cases._solid_fill(u, c.cell_types().reshape(g.N, g.M)).reshape(-1))
    return c


@pytest.mark.parametrize("n_x,n_y,body,scheme,riemann,time", [
    (2, 2, False, "MUSCL", "HLL", "SingleStep"),
    (31, 15, False, "MHM", "HLL", "SingleStep"),
    (32, 16, False, "MUSCL", "StegerWarming", "SingleStep"),
    (33, 17, False, "Godunov", "HLL", "SingleStep"),
    (161, 97, True, "MUSCL", "HLL", "SingleStep"),
    (511, 255, False, "MUSCL", "HLL", "SingleStep"),            # 256 32x16 tiles
    (512, 257, False, "MUSCL", "HLL", "SingleStep"),            # 272: 32x16 on the device too
    (700, 401, True, "MHM", "StegerWarming", "SingleStep"),
])
def test_device_steps_equal_host_steps(n_x, n_y, body, scheme, riemann, time):
    with make(n_x, n_y, body, scheme, riemann, time) as a, make(n_x, n_y, body, scheme, riemann, time) as b:
        u = np.ascontiguousarray(b.get_state().reshape(-1))
        a.advance(4)
        for _ in range(4):
            p = b.step_host_ptr(u.ctypes.data, u.ctypes.data)
        assert np.array_equal(a.get_state().reshape(-1), u)
        q = a.progress()
        assert {k: v for k, v in p.items() if k != "mass"} == {k: v for k, v in q.items() if k != "mass"}
        assert abs(p["mass"] - q["mass"]) <= 1e-14 * abs(q["mass"])
