"""States at the ends of the number range and of the shape bound (marked
``gpu``): what the force evaluation and the update give where a square
overflows or a contour's radius vanishes."""

import numpy as np
import pytest

from conftest import fcc, oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,big", [(np.float64, 1e150), (np.float64, 1e155), (np.float64, 1e200), (np.float64, -1e308),
                                   (np.float32, 1e15), (np.float32, 1e25), (np.float32, -1e38)])
def test_amplitudes_whose_squares_overflow(T, big):
    """enforce_shape! scales one huge amplitude to the shape bound, or, where
    its norm is infinite, to zero: the oracle's body, when it is loaded and
    after three steps."""
    b, box = fcc.polydisperse_monolayer(8, 8, packing=0.95, maxmode=10, seed=3)
    b.coef[3, 7] = big
    kw = dict(types=(fcc.BodyType(v0=0.1, Dr=0.01, μab=0.1),), energies=(fcc.Tension(0.01), fcc.Overlap(1.0)), dt=0.005,
              seed=3, T=T)
    g, o = fcc.Simulation(b, box, **kw), oracle.OracleSimulation(b, box, **kw)
    rtol = 1e-8 if T is np.float64 else 1e-3
    for steps in (0, 3):
        if steps:
            g.run(steps)
            o.step(steps)
        a, c = g.bodies, o.bodies
        assert np.isfinite(c.coef).all()
        assert np.allclose(a.coef, c.coef, rtol=rtol, atol=rtol) and np.allclose(a.x, c.x, rtol=rtol)
    assert g.health() == {"nonfinite": False, "barrier_error": False}
