"""Batches that hold cases with tensor maps and cases without (GPU).

A ghost width other than two has no tensor map: its tiles are staged
element-wise, those of the other cases by bulk copies, and a persistent CTA
takes both in turn (more tiles than resident CTAs in each case), so that a copy
lands on planes that ordinary stores wrote just before.  Each case bit for
bit as it is alone: state, loop scalars and mass."""
import numpy as np
import pytest

ib = pytest.importorskip("ibtfo_gb300")
from ibtfo_gb300 import cases  # noqa: E402

pytestmark = pytest.mark.gpu


def make(n_x, n_y, ng, scheme, riemann, precision, time):
    g = cases.Grid(n_x, n_y, ng, 0.0, 0.0, 1.0, n_y / n_x)
    c = ib.Case(n_x, n_y, ng=ng, lo=(0, 0), hi=(g.hi_x, g.hi_y), cfl=0.4, t_end=1e300, max_iter=2 ** 31 - 1,
                scheme=scheme, riemann=riemann, boundary="IDWBaseGFM", precision=precision, time=time)
    x, y = g.coords()
    c.setup_geometry(cases.cylinder_phi(g, 0.55, 0.5 * g.hi_y, 0.2 * g.hi_y))
    wave = 0.2 * np.sin(7 * x) * np.cos(5 * y)
    u = cases.conserved(1.0 + wave, 0.3 + wave, 0.1 - wave, 1.0 + 0.5 * wave, 1.4)
    c.set_state(cases._solid_fill(u, c.cell_types().reshape(g.N, g.M)).reshape(-1))
    return c


@pytest.mark.parametrize("scheme,riemann,precision,time", [
    ("MUSCL", "HLL_Toro", "fp32c", "SingleStep"),
    ("MHM", "HLL_Toro", "fp32c", "RK2"),
    ("MUSCL", "HLL", "fp32c", "SingleStep"),
    ("MUSCL", "HLL", "fp64_fast", "RK2"),
])
def test_ghost_widths_mixed_in_a_batch(scheme, riemann, precision, time):
    sizes = [(512, 500, 3), (760, 771, 2), (500, 519, 3), (769, 760, 2)]
    key = (scheme, riemann, precision, time)
    batched = [make(*s, *key) for s in sizes]
    with ib.Batch(scheme, riemann, "minmod", precision, tile_shape="32x16", time=time) as b:
        for c in batched:
            b.add(c)
        b.advance(6)
        b.synchronize()
        for s, c in zip(sizes, batched):
            with make(*s, *key) as alone:
                alone.advance(6)
                assert np.array_equal(c.get_state(), alone.get_state())
                p = c.progress()
                assert p == alone.progress()
                assert p["iter"] == 6 and p["nan_cells"] == 0 and p["status"] == 0
    for c in batched:
        c.close()
