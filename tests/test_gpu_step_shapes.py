"""The step kernels' dispatch at its edges (marked ``gpu``), against the CPU
oracle and against each other:

- FP64 contractions on the tensor cores: contours of one chunk that do not
  fill it, of two chunks (table in shared memory) and of three (table read
  where it is), every number of modes, body counts that leave a warp's last
  group ragged, boxes of fewer than 3 cells a side, and neighbour lists longer
  than the stage of 8 records.  Forces at 1e-12 of each field's scale (sums of
  at most nθ · modes products of order one in FP64), 30 noisy steps at rtol
  1e-8 with equal rebuild counts, as the other parity tests;
- more body terms than the four read ahead;
- the kernels for one round of warp groups, at the largest size of one block's
  warp and just beyond it, and on both sides of the size where the other
  shapes take over: FP32 launch shapes give the same bits."""

import numpy as np
import pytest

from conftest import fcc, oracle

pytestmark = pytest.mark.gpu

FIELDS = ("GR", "GD", "GDD", "P", "gx", "gy", "gθ", "glab", "gcoef", "Ebody")


def relerr(a, b):
    a, b = np.asarray(a, float), np.asarray(b, float)
    return float(np.abs(a - b).max() / max(float(np.abs(b).max()), 1e-300)) if a.size else 0.0


def deformed(nx, ny, maxmode, seed, packing=0.97, nuclei=False):
    rng = np.random.default_rng(seed)
    bodies, box = fcc.hexagonal_monolayer(nx, ny, packing=packing, maxmode=maxmode, rng=rng)
    if nuclei:
        bodies = fcc.with_nuclei(bodies, rng=rng)
    bodies.coef[1:] = 0.1 / bodies.ncoef * rng.standard_normal((bodies.ncoef - 1, bodies.n))
    bodies.coef[0] = np.sqrt(1 - 0.5 * np.sum(bodies.coef[1:] ** 2, axis=0))
    bodies.x[:] = (bodies.x + 0.03 * rng.standard_normal(bodies.n)) % box.Lx
    bodies.y[:] = (bodies.y + 0.03 * rng.standard_normal(bodies.n)) % box.Ly
    return bodies, box


def take(bodies, n):
    return fcc.Bodies(*(np.asfortranarray(getattr(bodies, f)[..., :n]) for f in
                        ("x", "y", "θ", "imgx", "imgy", "coef", "R0", "type", "parent")))


KW = dict(types=(fcc.BodyType(v0=0.06, Dr=0.05, μab=0.1), fcc.BodyType(Dr=0.05, μab=0.1)),
          energies=(fcc.Tension(0.02), fcc.PerimeterElasticity(0.1, 3.7),
                    fcc.Overlap([[1.0, 0.8], [0.8, 0.6]], related=[[1.0, -2.0], [-2.0, 1.0]]),
                    fcc.LinearRepulsion(0.5)), seed=11)


def check_against_oracle(bodies, box, steps=30, **kw):
    kw = {**KW, **kw}
    g, o = fcc.Simulation(bodies, box, T=np.float64, **kw), oracle.OracleSimulation(bodies, box, T=np.float64, **kw)
    g.refresh()
    o.refresh()
    assert np.array_equal(g.neighbors.count, o.neighbors.count)
    for f in FIELDS:
        assert relerr(getattr(g.grad, f), getattr(o.grad, f)) < 1e-12, f
    g.run(steps)
    o.step(steps)
    a, b = g.bodies, o.bodies
    for f in ("x", "y", "θ"):
        assert np.allclose(getattr(a, f), getattr(b, f), rtol=1e-8, atol=1e-9), f
    assert np.allclose(a.coef, b.coef, rtol=1e-8, atol=1e-11)
    assert g.builds == o.builds and np.array_equal(a.imgx, b.imgx)
    return g, o


@pytest.mark.parametrize("nθ,maxmode,n", [(24, 10, 1), (33, 10, 2), (40, 2, 3), (40, 3, 5), (40, 9, 63), (40, 10, 64),
                                          (41, 10, 30), (64, 10, 33), (79, 6, 31), (80, 10, 64), (81, 10, 29),
                                          (121, 7, 30)])
def test_fp64_contractions_match_the_oracle(nθ, maxmode, n):
    bodies, box = deformed(8, 8, maxmode, 3 + n)
    check_against_oracle(take(bodies, n), box, nθ=nθ)


@pytest.mark.parametrize("nx,ny,nθ", [(2, 2, 40), (3, 4, 40), (2, 4, 64), (6, 6, 41)])
def test_fp64_small_boxes_and_long_lists(nx, ny, nθ):
    """Boxes that collapse the cell grid, with nuclei: every body lists most of
    the others, more than one stage of records at 24 and 72 bodies."""
    bodies, box = deformed(nx, ny, 8, 7, packing=0.95, nuclei=True)
    g, o = check_against_oracle(bodies, box, nθ=nθ, skin=0.6, bonds=fcc.parent_bonds(bodies))
    if nx * ny >= 12:
        assert g.neighbors.count.max() > 8


def test_more_body_terms_than_are_read_ahead():
    bodies, box = deformed(6, 6, 6, 5, nuclei=True)
    terms = tuple(fcc.OnTypes(fcc.Tension(0.01 * (k + 1)), 1 + k % 2) if k % 3 else fcc.PerimeterElasticity(0.02 * (k + 1), 3.6)
                  for k in range(7)) + (fcc.Overlap(1.0),)
    check_against_oracle(bodies, box, energies=terms)


@pytest.mark.parametrize("n", [5, 588, 596, 4732, 4740])
def test_one_round_shapes_give_the_bits_of_the_others(n, monkeypatch):
    """FP32: the kernel that keeps its bodies' state from step to step (the
    choice while 8 warps per SM hold every group: 4736 bodies on 148 SMs)
    against the two-blocks-per-SM shapes, over rebuilds and several launches."""
    bodies, box = deformed(70, 70, 10, n)
    bodies = take(bodies, n)
    kw = {**KW, "types": (fcc.BodyType(v0=0.3, Dr=0.2, Dt=0.02, μab=0.1),), "energies": KW["energies"][:2] + (fcc.Overlap(1.0),)}
    out = []
    for v in (None, "0", "5", "6"):
        if v is None:
            monkeypatch.delenv("FCC_VARIANT", raising=False)
        else:
            monkeypatch.setenv("FCC_VARIANT", v)
        s = fcc.Simulation(bodies, box, T=np.float32, **kw)
        s.run(150)
        s.dt = 0.004
        s.run(90)
        s.step(3)
        out.append((s.bodies, s.builds))
    a, builds = out[0]
    assert np.isfinite(a.x).all() and builds > 2
    for b, nb in out[1:]:
        assert nb == builds
        for f in ("x", "y", "θ", "coef", "imgx", "imgy"):
            assert np.array_equal(getattr(a, f), getattr(b, f)), f


@pytest.mark.parametrize("nθ,n", [(41, 61), (48, 62), (57, 64), (64, 30)])
def test_fp64_shapes_of_finer_contours_give_the_same_bits(nθ, n, monkeypatch):
    """Contours of 41 to 64 nodes in one chunk of 8 nodes a lane (the choice for
    one round of warp groups) against two chunks, and in a pool: a simulation's
    result does not depend on the shape its size, or its pool's, selects."""
    bodies, box = deformed(8, 8, 10, n)
    bodies = take(bodies, n)
    out = []
    for v in (None, "0", "5", "7"):
        if v is None:
            monkeypatch.delenv("FCC_VARIANT", raising=False)
        else:
            monkeypatch.setenv("FCC_VARIANT", v)
        s = fcc.Simulation(bodies, box, T=np.float64, nθ=nθ, **KW)
        s.run(60)
        out.append(s.bodies)
    pool = fcc.Pool(T=np.float64, nθ=nθ, max_bodies=256, max_cells=256, max_sims=2)
    slot = pool.add(bodies, box, horizon=60, **KW)
    pool.run(60)
    out.append(pool.bodies(slot))
    for b in out[1:]:
        for f in ("x", "y", "θ", "coef"):
            assert np.array_equal(getattr(out[0], f), getattr(b, f)), f


def test_user_body_terms_on_alternating_types():
    """User terms restricted to one type each, the types alternating within a
    warp's bodies: forces of both precisions against the FP64 oracle (FP64 at
    1e-12 of each field's scale, FP32 at 1e-5 on an FP32-representable state, as
    the other user-term tests; no contacts, so no Heaviside flips)."""
    bodies, box = deformed(6, 6, 6, 17, packing=0.6)
    bodies.type[:] = 1 + np.arange(bodies.n) % 2
    for f in ("x", "y", "θ", "coef", "R0"):
        getattr(bodies, f)[...] = np.asarray(getattr(bodies, f), np.float32)
    kw = {**KW, "energies": (fcc.Tension(0.02), fcc.OnTypes(fcc.ShapeIndexElasticity(0.05, 3.7), 1),
                             fcc.OnTypes(fcc.Bending(0.02), 2))}
    o = oracle.OracleSimulation(bodies, box, T=np.float64, **kw).refresh()
    for T, tol in ((np.float64, 1e-12), (np.float32, 1e-5)):
        g = fcc.Simulation(bodies, box, T=T, **kw).refresh()
        for f in ("GR", "GD", "GDD", "glab", "gcoef", "Ebody"):
            assert relerr(getattr(g.grad, f), getattr(o.grad, f)) < tol, (T, f)
        g.run(3)
        assert np.isfinite(g.bodies.coef).all()


@pytest.mark.parametrize("T", [np.float32, np.float64])
@pytest.mark.parametrize("nx,ny,n,cap", [(8, 8, 1, None), (8, 8, 33, 1), (18, 16, 257, None), (150, 140, 20999, 4)])
def test_update_neighbors_lists_and_flags(nx, ny, n, cap, T):
    """The stand-alone rebuild over its grids (one block, a remainder, more
    bodies than the grid's lanes) and with lists that have to grow: the
    oracle's lists (FP64; integers: equality), a rebuild only where one is due,
    and steps that go on from it as from the rebuild of a first step."""
    bodies, box = deformed(nx, ny, 6, 23)
    bodies = take(bodies, n)
    kw = {**KW, "T": T, **({} if cap is None else {"nl_capacity": cap})}
    g = fcc.Simulation(bodies, box, **kw)
    g.update_neighbors()
    a = g.neighbors
    if cap is not None:
        assert a.cap >= a.count.max() > cap
    if T is np.float64:
        o = oracle.OracleSimulation(bodies, box, **{**KW, "T": T})
        o.update_neighbors()
        b = o.neighbors
        for f in ("cellid", "perm", "start", "stop", "count"):
            assert np.array_equal(getattr(a, f), getattr(b, f)), f
        listed = np.arange(min(a.idx.shape[0], b.idx.shape[0]))[:, None] < a.count
        assert np.array_equal(a.idx[:len(listed)][listed], b.idx[:len(listed)][listed])
    builds = g.builds
    assert g.update_neighbors().builds == builds
    assert g.update_neighbors(force=True).builds == builds + 1
    fresh = fcc.Simulation(bodies, box, **kw)
    g.run(5)
    fresh.run(5)
    for f in ("x", "y", "θ", "coef"):
        assert np.array_equal(getattr(g.bodies, f), getattr(fresh.bodies, f)), f


def test_a_tuned_shape_does_not_bind_other_contours():
    """The tuner remembers a launch shape by size and precision; a pool of that
    size whose contour the shape does not take (here 80 nodes, after one of 64
    was tuned, where the shape of one chunk of 8 nodes a lane is the fastest)
    runs with its own and equals the simulation alone."""
    bodies, box = deformed(8, 8, 10, 5)
    tuned = fcc.Pool(T=np.float64, nθ=64, max_bodies=256, max_cells=256, max_sims=2)
    tuned.add(bodies, box, horizon=1 << 20, **KW)
    tuned.run(5)
    tuned.tune(steps=40, reorder=True)
    pool = fcc.Pool(T=np.float64, nθ=80, max_bodies=256, max_cells=256, max_sims=2)
    slot = pool.add(bodies, box, horizon=60, **KW)
    pool.run(60)
    alone = fcc.Simulation(bodies, box, T=np.float64, nθ=80, **KW)
    alone.run(60)
    a, b = alone.bodies, pool.bodies(slot)
    for f in ("x", "y", "θ", "coef"):
        assert np.array_equal(getattr(a, f), getattr(b, f)), f


@pytest.mark.parametrize("nθ", [48, 64])
def test_finer_contours_in_a_pool_of_two_rounds_equal_lone_runs(nθ):
    """FP64 contours of 41 to 64 nodes: members of a pool of more bodies than one
    round holds (two chunks, two blocks per SM) against the same simulations
    alone (one chunk of 8 nodes a lane), over many rebuilds: the same bits."""
    pool = fcc.Pool(T=np.float64, nθ=nθ, max_bodies=8192, max_cells=8192, max_sims=8)
    lone, slots = [], []
    for k in range(5):
        bodies, box = deformed(32, 32 + 2 * k, 10, 40 + k)
        kw = {**KW, "types": (fcc.BodyType(v0=0.3, Dr=0.2, Dt=0.02, μab=0.1),), "seed": 3 + k}
        slots.append(pool.add(bodies, box, horizon=1 << 20, **kw))
        lone.append(fcc.Simulation(bodies, box, T=np.float64, nθ=nθ, **kw))
    assert sum(s.N for s in lone) > 4736 and pool.variant()["slots"] == 5
    pool.run(300)
    for s, slot in zip(lone, slots):
        s.run(300)
        assert s.builds > 10 and pool.builds(slot) == s.builds
        a, b = s.bodies, pool.bodies(slot)
        for f in ("x", "y", "θ", "coef"):
            assert np.array_equal(getattr(a, f), getattr(b, f)), f
