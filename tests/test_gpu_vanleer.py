"""The van Leer branches of the paired FP32 faces and of the two FP64 tile sizes (GPU).

The reference's van Leer macro is no slope of a smooth flow (its states lie
near 7/4 and 1/4 of the cell's), so flows last a step or two; one step of a ramp
in every conserved variable, whose differences keep their sign, is compared.

FP32 (HLL_Toro) against the same arithmetic in float32, one face at a time
(difference_form.py): an update is at most CFL x 7/4 = 0.7 of the scale in face
fluxes, each of which passes about a hundred FP32 roundings of 6e-8 that add to
16 of them, and a limiter that triples the relative error of a quotient of
differences (four roundings): 2e-6 of a flux, four fluxes a cell, 6e-6 of the
scale; 1e-5 allowed.  With minmod the same step differs by 1e-3 and more.  (FP64 is
no yardstick here: the macro takes the difference of two cells from their
rounded FP32 values, and its result moves by the scale times that rounding over the
difference: 7e-5 at 31 cells, 5e-3 at 961, the restatement as the kernel.)
Device steps (16x8 tiles) against host-array steps (32x16): bit for bit."""
import numpy as np
import pytest

import difference_form

ib = pytest.importorskip("ibtfo_gb300")
from ibtfo_gb300 import cases  # noqa: E402

pytestmark = pytest.mark.gpu


def make(n_x, n_y, scheme, riemann, precision, limiter="VanLeer"):
    g = cases.Grid(n_x, n_y, 2, 0.0, 0.0, 1.0, n_y / n_x)
    c = ib.Case(n_x, n_y, lo=(0, 0), hi=(g.hi_x, g.hi_y), cfl=0.4, t_end=1e300, max_iter=2 ** 31 - 1, scheme=scheme,
                riemann=riemann, limiter=limiter, precision=precision)
    c.setup_geometry(np.ones(g.N * g.M))
    x, y = g.coords()
    u = cases.conserved(1 + 0.5 * x + 0.3 * y, 0.3 + 0.2 * x + 0.1 * y, 0.1 + 0.2 * x + 0.1 * y, 1 + 0.4 * x + 0.2 * y, 1.4)
    c.set_state(np.ascontiguousarray(u).reshape(-1))
    return c


@pytest.mark.parametrize("n_x,n_y,scheme", [
    (31, 15, "MUSCL"), (32, 16, "MHM"), (33, 17, "MUSCL"), (65, 49, "MHM"), (961, 500, "MUSCL"),
])
def test_van_leer_pairs(n_x, n_y, scheme):
    with make(n_x, n_y, scheme, "HLL_Toro", "fp32c") as c:
        u, dt, g = c.get_state().reshape(c.N, c.M, 4), c.progress()["dt"], cases.Grid(n_x, n_y, 2, 0, 0, 1.0, n_y / n_x)
        c.advance(1)
        assert c.progress()["nan_cells"] == 0
        got = c.get_state().reshape(c.N, c.M, 4)[2:-2, 2:-2]
    want = difference_form.step(u, 1.0 / n_x, g.hi_y / n_y, dt, scheme, "VanLeer")
    other = difference_form.step(u, 1.0 / n_x, g.hi_y / n_y, dt, scheme, "minmod")
    scale = np.abs(want).max()
    assert np.abs(got - want).max() <= 1e-5 * scale
    assert np.abs(want - other).max() >= 50 * 1e-5 * scale  # the limiter shows


@pytest.mark.parametrize("scheme,riemann,precision", [
    ("MUSCL", "HLL", "fp64"), ("MHM", "StegerWarming", "fp64"), ("MUSCL", "HLL_Toro", "fp64_fast"),
    ("MHM", "HLL", "fp64_fast"), ("MUSCL", "PVRS", "fp64"),
])
def test_van_leer_on_both_tiles(scheme, riemann, precision):
    with make(161, 97, scheme, riemann, precision) as a, make(161, 97, scheme, riemann, precision) as b:
        u = np.ascontiguousarray(b.get_state().reshape(-1))
        a.advance(1)
        b.step_host_ptr(u.ctypes.data, u.ctypes.data)
        got = a.get_state().reshape(-1)
        assert np.array_equal(got, u, equal_nan=True) and np.isfinite(got).mean() > 0.9
