"""The float64 form of difference_form.py against the cut-cell oracle's HLL_Toro on a
grid without bodies: the same algorithm, so rounding apart (some hundred
operations of 1.1e-16 on values up to 4: 1e-13 allowed)."""
import numpy as np
import pytest

import difference_form
from ibtfo_gb300 import cases

oracle = pytest.importorskip("oracle")


@pytest.mark.parametrize("scheme", ["MUSCL", "MHM"])
@pytest.mark.parametrize("limiter", ["minmod", "VanLeer"])
def test_restatement_is_the_oracles_step(scheme, limiter):
    g = cases.Grid(65, 49, 2, 0.0, 0.0, 1.0, 49 / 65)
    x, y = g.coords()
    u = cases.conserved(1 + 0.5 * x + 0.3 * y, 0.3 + 0.2 * x + 0.1 * y, 0.1 + 0.2 * x + 0.1 * y, 1 + 0.4 * x + 0.2 * y, 1.4)
    o = oracle.CcmOracle(g.n_x, g.n_y, g.ng, (0, 0), (g.hi_x, g.hi_y), 1.4, 0.4, 1e300, scheme, "HLL_Toro", limiter,
                         "walls")
    o.setup(np.ones(g.N * g.M))
    o.set_state(u.reshape(-1))
    first, dt = o.get_state().reshape(g.N, g.M, 4).copy(), o.scalars()["dt"]
    o.run(1)
    want = o.get_state().reshape(g.N, g.M, 4)[2:-2, 2:-2]
    got = difference_form.step(first, 1.0 / g.n_x, g.hi_y / g.n_y, dt, scheme, limiter, np.float64)
    assert np.abs(got - want).max() <= 1e-13
