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


@pytest.mark.parametrize("a", [-0.9, -5.0])
@pytest.mark.parametrize("term", [fcc.Tension(0.01), fcc.PerimeterElasticity(0.1, 3.7),
                                  fcc.ShapeIndexElasticity(0.05, 3.7)])
def test_contour_that_touches_its_centre(term, a):
    """One elliptic mode at the shape bound: R = R' = 0 at node 0, where the
    perimeter has no gradient (0 / 0).  Its integrals do not see that: energies
    and the other nodes' gradients are the oracle's (1e-12 of their scale), the
    node's own are not finite, in both."""
    b, box = fcc.hexagonal_monolayer(4, 4, packing=0.5, maxmode=2, rng=2)
    b.θ[:] = 0.0
    b.coef[1, 5] = a
    kw = dict(types=(fcc.BodyType(),), energies=(term, fcc.Overlap(1.0)), nθ=40, T=np.float64)
    g, o = (cls(b, box, **kw).refresh().grad for cls in (fcc.Simulation, oracle.OracleSimulation))
    assert np.isfinite(o.Ebody).all()
    assert np.allclose(g.Ebody, o.Ebody, rtol=1e-12, atol=0)
    node = np.isfinite(o.GR)
    assert not node[0, 5] and node.sum() == node.size - 1
    assert np.array_equal(np.isfinite(g.GR), node)
    assert np.abs(g.GR[node] - o.GR[node]).max() <= 1e-12 * np.abs(o.GR[node]).max()

