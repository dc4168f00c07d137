"""Results written by the device into page-locked arrays (marked ``gpu``):
the same values as through ordinary memory (the path of a caller's own arrays,
and of results beyond the page-locked limit), and a stateless neighbour build
that keeps its workspace between calls of other sizes, precisions and threads.
Integers and doubles that are only copied or widened: the tolerance is
equality."""

from concurrent.futures import ThreadPoolExecutor

import ctypes as C

import numpy as np
import pytest

from conftest import fcc, oracle

pytestmark = pytest.mark.gpu

abi, simulation = fcc.simulation.abi, fcc.simulation


def sim(T, n=(7, 8), maxmode=6, nθ=24):
    bodies, box = fcc.hexagonal_monolayer(*n, packing=0.98, maxmode=maxmode, rng=2)
    bodies.coef[1:, :] = 0.03 * np.random.default_rng(5).standard_normal((bodies.ncoef - 1, bodies.n))
    return bodies, box, dict(types=(fcc.BodyType(v0=0.06, Dr=0.01, μab=0.1),),
                             energies=(fcc.Tension(0.01), fcc.Overlap(1.0)), nθ=nθ, T=T, seed=3)


@pytest.mark.parametrize("T", [np.float32, np.float64])
@pytest.mark.parametrize("maxmode,nθ", [(6, 24), (10, 40), (3, 64)])
def test_results_in_place_equal_copied_ones(T, maxmode, nθ, monkeypatch):
    bodies, box, kw = sim(T, maxmode=maxmode, nθ=nθ)
    s = fcc.Simulation(bodies, box, **kw).refresh()
    s.run(3)
    s.refresh()
    grad, state = s.grad, s.bodies
    monkeypatch.setattr(simulation, "_BLOCKS", simulation._ResultBlocks())
    monkeypatch.setattr(simulation._ResultBlocks, "LIMIT", 0)
    for a, b in zip(grad, s.grad):
        assert a.shape == b.shape and np.array_equal(a, b)
    other = s.bodies
    for f in ("x", "y", "θ", "imgx", "imgy", "coef", "R0", "type", "parent"):
        a, b = getattr(state, f), getattr(other, f)
        assert a.dtype == b.dtype and np.array_equal(a, b), f
    # some buffers only, in the caller's own memory
    gx, glab = np.zeros(s.N), np.zeros((s.N, s.ncoef))
    g = abi.FccGradientsHost(None, None, None, None, abi.dptr(gx), None, None, abi.dptr(glab), None, None)
    s._call("get_gradients", s._h, C.byref(g))
    assert np.array_equal(gx, grad.gx) and np.array_equal(glab.T, grad.glab)


def test_result_blocks_are_bounded_and_reused(monkeypatch):
    monkeypatch.setattr(simulation, "_BLOCKS", simulation._ResultBlocks())
    monkeypatch.setattr(simulation._ResultBlocks, "LIMIT", 1 << 20)
    blocks, lib = simulation._BLOCKS, fcc.native_library()
    kept = [blocks.take(lib, 200_000) for _ in range(8)]
    assert sum(k is not None for k in kept) == (1 << 20) // blocks.size_of(200_000)
    assert blocks.take(lib, 200_000) is None
    address = kept[0].ctypes.data
    view = kept[0][10:20]
    kept[0] = None
    assert blocks.take(lib, 200_000) is None      # a view keeps the block
    del view
    again = blocks.take(lib, 200_000)
    assert again.ctypes.data == address
    kept.clear()
    del again                                     # every block is idle
    big = blocks.take(lib, 900_000)               # idle blocks of other sizes make room
    assert big is not None and blocks._total <= 1 << 20


def neighbors(seed, n, T, cap=32):
    rng = np.random.default_rng(seed)
    L = np.sqrt(3.5 * n) + 4
    x, y = rng.random(n) * L, rng.random(n) * L * 1.1
    rmax = 0.9 + 0.3 * rng.random(n)
    return (x, y, rmax, L, L * 1.1, 3.0, 0.3), dict(cap=cap, T=T)


def same(a, b):
    for u, v in zip(a[:4], b[:4]):
        assert np.array_equal(u, v)
    assert np.array_equal(a[5], b[5])
    # the oracle orders and fills the first `cap` entries; the rest are zero here
    cap = a[4].shape[0]
    for i in range(a[4].shape[1]):
        k = min(a[5][i], cap)
        assert np.array_equal(a[4][:k, i], b[4][:k, i]) and not a[4][k:, i].any()


def test_neighbor_workspace_over_sizes_precisions_and_threads():
    jobs = [neighbors(k, n, T, cap) for k, (n, T, cap) in enumerate(
        [(700, np.float64, 32), (5, np.float64, 3), (9000, np.float32, 20), (1, np.float32, 1), (700, np.float64, 2),
         (9001, np.float64, 40), (300, np.float32, 33)])]
    want = [oracle.build_neighbors(*a, **k) for a, k in jobs]
    for _ in range(2):
        for (a, k), w in zip(jobs, want):
            same(fcc.build_neighbors(*a, **k), w)
    with ThreadPoolExecutor(4) as ex:
        for got, w in zip(ex.map(lambda j: fcc.build_neighbors(*j[0], **j[1]), jobs * 3), want * 3):
            same(got, w)
    with pytest.raises(fcc.ArgumentError):
        fcc.build_neighbors(*jobs[0][0][:5], -1.0, 0.3)
    same(fcc.build_neighbors(*jobs[0][0], **jobs[0][1]), want[0])


@pytest.mark.parametrize("nx,ny,n", [(3, 3, 5), (7, 73, 200), (16, 32, 4000), (27, 19, 300), (32, 32, 1), (33, 31, 3000),
                                     (200, 190, 50), (171, 180, 30000)])
def test_cell_scan_over_its_ranges(nx, ny, n):
    """Grids of fewer, exactly and more cells than one range of the scan (512),
    densely and sparsely filled: cell lists and neighbour lists equal the
    oracle's, in a build of its own and inside the step kernel."""
    rng = np.random.default_rng(nx * ny + n)
    cutoff = 3.2
    Lx, Ly = nx * cutoff * 1.0001, ny * cutoff * 1.0001
    x, y = rng.random(n) * Lx, rng.random(n) * Ly
    same(fcc.build_neighbors(x, y, np.full(n, 1.1), Lx, Ly, cutoff, 0.3, cap=64),
         oracle.build_neighbors(x, y, np.full(n, 1.1), Lx, Ly, cutoff, 0.3, cap=64))
    R0 = (cutoff - 0.3) / (2 * (1 + np.sqrt(2 / 3)))  # the radius whose grid has this cutoff
    coef = np.zeros((7, n), order="F")
    coef[0] = 1.0
    bodies = fcc.Bodies.new(x, y, np.zeros(n), coef, np.full(n, R0))
    kw = dict(types=(fcc.BodyType(v0=0.5),), energies=(fcc.Overlap(0.1),), nθ=16, nl_capacity=64)
    s, o = (cls(bodies, fcc.PeriodicBox(Lx, Ly), T=np.float64, **kw) for cls in (fcc.Simulation, oracle.OracleSimulation))
    s.run(2)
    o.step(2)
    a, b = s.neighbors, o.neighbors
    assert a.ncx * a.ncy == b.ncx * b.ncy and s.builds == o.builds
    for f in ("cellid", "perm", "start", "stop", "count"):
        assert np.array_equal(getattr(a, f), getattr(b, f)), f


def test_a_refused_page_lock_does_not_fail_the_next_call():
    """Page-locked memory that the system does not give (4 PB here) is an error
    of that request alone: results come in ordinary arrays then, and the calls
    that follow, kernel launches among them, do not see it."""
    bodies, box, kw = sim(np.float64)
    s, lib = fcc.Simulation(bodies, box, **kw), fcc.native_library()
    p = C.c_void_p()
    for query in (lambda: s.bodies, s.shape_index, lambda: s.refresh().grad, lambda: s.run(2)):
        assert lib.fcc_host_alloc(1 << 52, C.byref(p)) == abi.FCC_ERR_NOMEM
        query()


def odd(a):
    """A page-locked array like `a`, half an element off its alignment."""
    block = simulation._ResultBlocks().take(fcc.native_library(), a.nbytes + 64)
    v = np.ndarray(a.shape, a.dtype, block, a.itemsize // 2)
    v[...] = a
    return v


def test_misaligned_page_locked_arrays():
    """Page-locked arrays off their alignment, which the device cannot access,
    are copied like ordinary ones: states, gradients and lists equal those
    through aligned arrays."""
    bodies, box, kw = sim(np.float64, n=(32, 32))
    s = fcc.Simulation(bodies, box, **kw).refresh()
    s.run(3)
    want, grad = s.bodies, s.refresh().grad
    GR = odd(np.zeros((s.N, s.nθ)))
    g = abi.FccGradientsHost(abi.dptr(GR), *[None] * 9)
    s._call("get_gradients", s._h, C.byref(g))
    assert np.array_equal(GR.T, grad.GR)
    b = want.copy()
    for f in ("x", "y", "θ", "imgx", "imgy"):
        setattr(b, f, odd(getattr(want, f)))
    b.coef = odd(np.ascontiguousarray(want.coef.T)).T
    s.set_state(b)
    for f in ("x", "y", "θ", "imgx", "imgy", "coef"):
        getattr(b, f)[...] = 0
    s.get_state(out=b)
    for f in ("x", "y", "θ", "imgx", "imgy", "coef"):
        assert np.array_equal(getattr(b, f), getattr(want, f)), f
    (x, y, rmax, *rest), kwl = neighbors(3, 4000, np.float64)
    same(fcc.build_neighbors(odd(x), odd(y), odd(rmax), *rest, **kwl), oracle.build_neighbors(x, y, rmax, *rest, **kwl))


@pytest.mark.parametrize("T", [np.float32, np.float64])
def test_results_change_to_page_locked_memory(T, monkeypatch):
    """The same query again and again, its results dropped: ordinary arrays
    first, page-locked ones once enough came back, equal values throughout, for
    gradients, states, pool states and neighbour lists."""
    bodies, box, kw = sim(T, n=(32, 32))
    s = fcc.Simulation(bodies, box, **kw).refresh()
    s.run(3)
    s.refresh()
    nθ = kw.pop("nθ")
    pool = fcc.Pool(nθ=nθ, T=kw.pop("T"), max_bodies=2048, max_cells=2048, max_sims=2)
    slot = pool.add(bodies, box, horizon=1 << 20, **kw)
    pool.run(3)
    args, kwl = neighbors(5, 4000, T)
    for query in (lambda: list(s.grad), lambda: [getattr(s.bodies, f) for f in ("x", "y", "θ", "coef", "imgx", "R0", "type")],
                  lambda: [getattr(pool.bodies(slot), f) for f in ("x", "y", "θ", "coef", "imgy", "R0", "parent")],
                  lambda: list(fcc.build_neighbors(*args, **kwl))):
        monkeypatch.setattr(simulation, "_BLOCKS", simulation._ResultBlocks())
        first, places = query(), []
        for _ in range(200):
            got = query()
            assert all(np.array_equal(a, b) for a, b in zip(first, got))
            places.append(any(v.at <= got[0].ctypes.data < v.at + v.size for v in simulation._BLOCKS._slabs))
        assert not places[0] and places[-1] and places == sorted(places)


def test_gradients_into_ordinary_memory_keep_their_device_area():
    """Queries of gradients into a caller's own arrays allocate device memory
    once: what the first one took is still held after it, and later ones take
    no more."""
    import torch
    bodies, box, kw = sim(np.float64, n=(128, 128), nθ=40)
    s = fcc.Simulation(bodies, box, **kw).refresh()
    P = np.zeros((s.N, s.nθ))
    g = abi.FccGradientsHost(None, None, None, abi.dptr(P), *[None] * 6)
    free = [torch.cuda.mem_get_info()[0]]
    for _ in range(3):
        s._call("get_gradients", s._h, C.byref(g))
        free.append(torch.cuda.mem_get_info()[0])
    assert free[0] - free[1] >= P.nbytes - (2 << 20) and free[1] == free[2] == free[3]
