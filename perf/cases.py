"""Work that programs have this framework do, through its public entry points.

Kinds of case:

- ``run``: load a body state (``set_state``), advance it (``run``) and read the
  new state back (``get_state``) through page-locked arrays, as a parameter
  scan, a restart or a recorder of snapshots does; ``observe`` adds the shape
  index of every body, which recorders store beside the snapshot.
- ``step``: one time step and a read of the state: interactive and analysis
  loops that look at every step.
- ``gradients``: load a state, rebuild its lists, evaluate every gradient buffer
  and read them: force analysis and fitting.
- ``pool``: many simulations of uneven size advanced together and read back.
- ``neighbors``: cell and neighbour lists of positions a program holds.

Models are those of the tests and the benchmark: the plain monolayer
(Tension + Overlap), the polydisperse one (+ PerimeterElasticity), cells with
nuclei (parent drag, bonds, related couplings), contours of more nodes with
LinearRepulsion, and compiled user terms.  States are deformed monolayers with
the mode amplitudes that such a run reaches after some hundred steps.
"""

import importlib.util
import math
import os
import sys

import numpy as np

ROOT = os.getcwd()


def package():
    """The repository's package (its directory name is not an identifier)."""
    if "fcc_b200" not in sys.modules:
        home = os.path.join(ROOT, "fouriercontourcells.jl_b200")
        spec = importlib.util.spec_from_file_location("fcc_b200", os.path.join(home, "__init__.py"),
                                                      submodule_search_locations=[home])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["fcc_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["fcc_b200"]


# ------------------------------------------------------------------ cases
def listed():
    return [
        # one step of the smallest published system (8 x 8, modes 2..6), read back: latency
        dict(name="step_n64_f64", kind="step", model="plain", nx=8, ny=8, maxmode=6, ntheta=40, bits=64, steps=1),
        # the plain 32 x 32 monolayer in double precision, between two snapshots
        dict(name="run_n1024_f64", kind="run", model="plain", nx=32, ny=32, maxmode=10, ntheta=40, bits=64, steps=100),
        # a small single-precision study of an odd size, with its shape index recorded
        dict(name="run_n1054_f32_observed", kind="run", model="poly", nx=31, ny=34, maxmode=10, ntheta=40, bits=32,
             steps=100, observe=True),
        # the benchmark's workload: 128 x 128 polydisperse, 20 steps per exchange
        dict(name="run_n16384_f32", kind="run", model="poly", nx=128, ny=128, maxmode=10, ntheta=40, bits=32, steps=20),
        # the same in double precision at a ragged size
        dict(name="run_n16002_f64", kind="run", model="poly", nx=127, ny=126, maxmode=10, ntheta=40, bits=64, steps=20),
        # the largest monolayer of the tests and the benchmark's sweep
        dict(name="run_n262144_f32", kind="run", model="poly", nx=512, ny=512, maxmode=10, ntheta=40, bits=32, steps=20),
        # cells with nuclei dragged along and bonded: forces and motion in two phases
        dict(name="nuclei_n8192_f32", kind="run", model="nuclei", nx=64, ny=64, maxmode=10, ntheta=40, bits=32, steps=40,
             observe=True),
        # finer contours (64 nodes) with a soft repulsion
        dict(name="fine_n2304_f64", kind="run", model="fine", nx=48, ny=48, maxmode=10, ntheta=64, bits=64, steps=30),
        # compiled user terms: bending and adhesion
        dict(name="user_n1024_f64", kind="run", model="user", nx=32, ny=32, maxmode=8, ntheta=40, bits=64, steps=30),
        # every gradient buffer of a state, for analysis
        dict(name="gradients_n4096_f64", kind="gradients", model="poly", nx=64, ny=64, maxmode=10, ntheta=40, bits=64,
             steps=0),
        # a batch of uneven monolayers in one pool
        dict(name="pool_64_f32", kind="pool", model="poly", members=64, least=64, most=2048, maxmode=10, ntheta=40,
             bits=32, steps=50),
        # lists of positions alone, single precision
        dict(name="neighbors_n65536_f32", kind="neighbors", model="poly", nx=256, ny=256, maxmode=10, ntheta=40, bits=32,
             steps=0),
    ]


def _side(rng, least, most):
    """Lattice of about log-uniform size: any width, even height."""
    n = math.exp(rng.uniform(math.log(least), math.log(most)))
    nx = max(8, round(math.sqrt(n) * math.exp(rng.uniform(-0.3, 0.3))))
    return nx, max(8, 2 * round(n / nx / 2))


def draw(rng):
    kind = rng.choice(["run"] * 6 + ["step", "gradients", "pool", "neighbors"])
    bits = rng.choice([32, 32, 64])
    maxmode = rng.choice([6, 8, 10, 10])
    if kind == "pool":
        least, most = rng.choice([(64, 512), (64, 2048), (256, 1024), (64, 4096)])
        return dict(kind=kind, model="poly", members=rng.randint(8, 64), least=least, most=most, maxmode=maxmode,
                    ntheta=40, bits=bits, steps=rng.randint(10, 40))
    if kind == "step":
        nx, ny = _side(rng, 64, 4096)
        return dict(kind=kind, model="plain", nx=nx, ny=ny, maxmode=maxmode, ntheta=40, bits=bits, steps=rng.randint(1, 4))
    if kind == "neighbors":
        nx, ny = _side(rng, 512, 131072)
        return dict(kind=kind, model="poly", nx=nx, ny=ny, maxmode=maxmode, ntheta=40, bits=bits, steps=0)
    model = rng.choice(["plain", "poly", "poly", "poly", "nuclei", "fine", "user"])
    ntheta = rng.choice([48, 56, 64, 80]) if model == "fine" else rng.choice([24, 32, 37, 40, 40, 40, 40])
    if kind == "gradients":
        nx, ny = _side(rng, 64, 8192)
        return dict(kind=kind, model=model, nx=nx, ny=ny, maxmode=maxmode, ntheta=ntheta, bits=bits, steps=0)
    # a run's body-steps stay below the largest listed case's
    most = 262144 if bits == 32 and model in ("plain", "poly") else 32768
    nx, ny = _side(rng, 64, most)
    room = (4_000_000 if most > 32768 else 800_000) / (nx * ny)
    steps = max(2, min(round(math.exp(rng.uniform(math.log(10), math.log(200)))), int(room)))
    return dict(kind=kind, model=model, nx=nx, ny=ny, maxmode=maxmode, ntheta=ntheta, bits=bits, steps=steps,
                observe=rng.random() < 0.3)


# ----------------------------------------------------------------- models
DT = 0.005
# rms amplitude of modes 2..10 in a monolayer that has run for some hundred steps
AMPLITUDE = np.array([0.044, 0.035, 0.027, 0.015, 0.036, 0.011, 0.013, 0.0125, 0.013])
SHAPE_BOUND = math.sqrt(2.0 / 3.0)


def _deform(bodies, rng, jitter, scale=1.0):
    """Random shapes and displacements of a lattice of circles, in place."""
    n, K = bodies.n, (bodies.ncoef - 1) // 2
    amp = scale * AMPLITUDE[:K, None] / math.sqrt(2)
    bodies.coef[1:1 + K] = amp * rng.standard_normal((K, n))
    bodies.coef[1 + K:] = amp * rng.standard_normal((K, n))
    total = np.hypot(bodies.coef[1:1 + K], bodies.coef[1 + K:]).sum(0)
    bodies.coef[1:] *= np.minimum(1.0, 0.6 / total)
    bodies.coef[0] = np.sqrt(1 - 0.5 * np.sum(bodies.coef[1:] ** 2, axis=0))
    bodies.x += jitter * bodies.R0 * rng.standard_normal(n)
    bodies.y += jitter * bodies.R0 * rng.standard_normal(n)


def _single(bodies):
    """Round the state to single precision values (held as doubles)."""
    for f in ("x", "y", "θ", "coef", "R0"):
        getattr(bodies, f)[...] = np.asarray(getattr(bodies, f), np.float32)


def _system(case, seed, nx=None, ny=None):
    """(bodies, box, arguments of Simulation) of a case."""
    fcc = package()
    nx, ny = nx or case["nx"], ny or case["ny"]
    rng = np.random.default_rng([seed, nx, ny])
    model, maxmode = case["model"], case["maxmode"]
    mobile = fcc.BodyType(v0=0.06, Dr=0.01, μab=0.1)
    types, bonds = (mobile,), ()
    if model == "plain":
        bodies, box = fcc.hexagonal_monolayer(nx, ny, packing=0.95, maxmode=maxmode, rng=rng)
        energies = (fcc.Tension(0.01), fcc.Overlap(1.0))
    elif model == "nuclei":
        bodies, box = fcc.hexagonal_monolayer(nx, ny, packing=0.9, maxmode=maxmode, rng=rng)
        energies = (fcc.OnTypes(fcc.Tension(0.01), 1), fcc.OnTypes(fcc.Tension(0.05), 2),
                    fcc.Overlap([[1.0, 1.0], [1.0, 1.0]], related=[[1.0, -2.0], [-2.0, 1.0]]), fcc.HarmonicBond(0.2))
        types = (mobile, fcc.BodyType(v0=0.0, Dr=0.01, drag="parent", μab=0.1))
    else:
        bodies, box = fcc.polydisperse_monolayer(nx, ny, maxmode=maxmode, seed=int(rng.integers(1 << 31)))
        energies = {"poly": (fcc.Tension(0.01), fcc.PerimeterElasticity(0.1, 3.7), fcc.Overlap(1.0)),
                    "fine": (fcc.Tension(0.02), fcc.PerimeterElasticity(0.1, 3.7), fcc.LinearRepulsion(4.0)),
                    "user": (fcc.Tension(0.1), fcc.Bending(0.02), fcc.Overlap(1.0), fcc.Adhesion(0.3, 0.1))}[model]
    _deform(bodies, rng, 0.02)
    if model == "nuclei":
        cells = bodies.n
        bodies = fcc.with_nuclei(bodies, rng=rng)
        inner = fcc.Bodies(*(getattr(bodies, f)[..., cells:] for f in
                             ("x", "y", "θ", "imgx", "imgy", "coef", "R0", "type", "parent")))
        _deform(inner, rng, 0.1, 0.5)
        bonds = fcc.parent_bonds(bodies)
    bodies.x %= box.Lx
    bodies.y %= box.Ly
    if case["bits"] == 32:
        _single(bodies)
    kw = dict(types=types, energies=energies, bonds=bonds, dt=DT, seed=int(rng.integers(1 << 62)))
    return bodies, box, kw


def _members(case):
    """Lattices of a pool: sizes spread over the case's range on a log scale."""
    spread = np.random.default_rng([case["members"], case["least"], case["most"]])
    got = []
    for n in np.exp(spread.uniform(math.log(case["least"]), math.log(case["most"]), case["members"])):
        nx = max(8, round(math.sqrt(n)))
        got.append((nx, max(8, 2 * round(n / nx / 2))))
    return got


def _neighbor_inputs(case, seed):
    """Positions, contour bounds, box, cutoff and range of a list build."""
    bodies, box, _ = _system(case, seed)
    K = (bodies.ncoef - 1) // 2
    rmax = bodies.R0 * (bodies.coef[0] + np.hypot(bodies.coef[1:1 + K], bodies.coef[1 + K:]).sum(0))
    if case["bits"] == 32:
        rmax = np.asarray(rmax, np.float32).astype(np.float64)
    return bodies.x, bodies.y, rmax, box, 2 * bodies.R0.max() * (1 + SHAPE_BOUND) + 0.3, 0.3


# ---------------------------------------------------------- prepare and run
def prepare(case, seed):
    fcc = package()
    T = np.float32 if case["bits"] == 32 else np.float64
    kind = case["kind"]
    if kind == "neighbors":
        x, y, rmax, box, cutoff, reach = _neighbor_inputs(case, seed)
        return dict(kind=kind, args=(x, y, rmax, box.Lx, box.Ly, cutoff, reach), T=T)
    if kind == "pool":
        systems = [_system(case, seed + 7919 * k, nx, ny) for k, (nx, ny) in enumerate(_members(case))]
        pool = fcc.Pool(T=T, nθ=case["ntheta"], max_bodies=sum(b.n + 8 for b, _, _ in systems),
                        max_cells=sum(b.n for b, _, _ in systems), max_sims=len(systems))
        slots = [pool.add(b, box, horizon=1 << 40, **kw) for b, box, kw in systems]
        return dict(kind=kind, pool=pool, slots=slots, steps=case["steps"])
    bodies, box, kw = _system(case, seed)
    sim = fcc.Simulation(bodies, box, nθ=case["ntheta"], T=T, **kw)
    return dict(kind=kind, sim=sim, steps=case["steps"], observe=bool(case.get("observe")),
                host=fcc.pinned_copy(bodies), out=fcc.pinned_bodies(bodies.n, bodies.ncoef))


def _read(b):
    return dict(x=b.x, y=b.y, theta=b.θ, coef=b.coef, imgx=b.imgx, imgy=b.imgy)


def run(state):
    fcc = package()
    kind = state["kind"]
    if kind == "neighbors":
        return dict(zip(("cellid", "perm", "start", "stop", "idx", "count"),
                        fcc.build_neighbors(*state["args"], T=state["T"])))
    if kind == "pool":
        pool = state["pool"]
        pool.run(state["steps"])
        states = [pool.bodies(s) for s in state["slots"]]
        return {f: np.concatenate([_read(b)[f].ravel(order="F") for b in states])
                for f in ("x", "y", "theta", "coef", "imgx", "imgy")}
    sim = state["sim"]
    if kind == "step":
        sim.step(state["steps"])
        return _read(sim.get_state(out=state["out"]))
    sim.set_state(state["host"], clock=0)
    if kind == "gradients":
        sim.refresh()
        return dict(sim.grad._asdict())
    sim.run(state["steps"])
    got = _read(sim.get_state(out=state["out"]))
    if state["observe"]:
        got["shape_index"] = sim.shape_index()
    return got


def _bodies_of(case):
    if case["kind"] == "pool":
        return sum(nx * ny for nx, ny in _members(case))
    return case["nx"] * case["ny"] * (2 if case["model"] == "nuclei" else 1)


def work(case):
    """Bytes of the inputs and outputs, and the model's arithmetic per body and
    step: synthesis of R, R' and the pullback of their gradients (2 K + 1
    coefficients at every node), body terms, node tests against some 6 listed
    neighbours, some 40 nodes inside a neighbour's bounding circle, update."""
    n, K, nodes = _bodies_of(case), case["maxmode"] - 1, case["ntheta"]
    w = case["bits"] // 8
    nc = 2 * K + 1
    state = n * (8 * (3 + nc) + 8)  # x, y, theta, coef as doubles, image counters
    per_step = 8 * nodes * nc + 24 * nodes + 10 * 6 * nodes + (8 * K + 8) * nodes + 30 * K + 60
    if case["kind"] == "neighbors":
        return {"bytes": n * (24 + 12 + 32 * 4), "flops": n * 9 * 3 * 12}
    if case["kind"] == "gradients":
        return {"bytes": state + n * 8 * (4 * nodes + 4 + 2 * nc), "flops": n * per_step}
    record = n * w * (nc + 5)  # what a pool or a stepped simulation holds on the device
    both = record + state if case["kind"] in ("pool", "step") else 2 * state
    return {"bytes": both + (8 * n if case.get("observe") else 0), "flops": n * per_step * case["steps"]}


# ------------------------------------------------- the same in plain numpy
def _philox(body, draw, block, key):
    """Philox4x32-10 words of counter (body, draw, draw >> 32, block)."""
    low = np.uint64(0xFFFFFFFF)
    c = [np.asarray(body, np.uint64), np.full(len(body), draw & 0xFFFFFFFF, np.uint64),
         np.full(len(body), draw >> 32, np.uint64), np.full(len(body), block, np.uint64)]
    k0, k1 = key & 0xFFFFFFFF, key >> 32
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & low, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & low]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def _normals(n, draw, block, key, bits):
    c = _philox(np.arange(1, n + 1), draw, block, key)
    if bits == 32:
        u1, u2 = (((c[k] >> np.uint64(9)).astype(np.float64) + 0.5) * 2.0**-23 for k in (0, 2))
    else:
        u1, u2 = ((((c[k] << np.uint64(32) | c[k + 1]) >> np.uint64(12)).astype(np.float64) + 0.5) * 2.0**-52
                  for k in (0, 2))
    r = np.sqrt(-2 * np.log(u1))
    return r * np.cos(2 * np.pi * u2), r * np.sin(2 * np.pi * u2)


class _Model:
    """One simulation in 64-bit numpy: forces, gradients and time steps."""

    def __init__(self, case, bodies, box, kw):
        fcc = package()
        self.b, self.box, self.bits, self.key = bodies, box, case["bits"], kw["seed"]
        self.types, self.energies, self.bonds = kw["types"], kw["energies"], np.array(kw["bonds"]).reshape(-1, 2) - 1
        self.x, self.y, self.th = bodies.x.copy(), bodies.y.copy(), bodies.θ.copy()
        self.R0, self.t, self.parent = bodies.R0, bodies.type - 1, bodies.parent - 1
        self.K, self.nodes = (bodies.ncoef - 1) // 2, case["ntheta"]
        self.n = np.arange(2, self.K + 2)[:, None]
        self.phi = 2 * np.pi * np.arange(self.nodes) / self.nodes
        self.a, self.bb = bodies.coef[1:1 + self.K].copy(), bodies.coef[1 + self.K:].copy()
        self.imgx, self.imgy = bodies.imgx.copy(), bodies.imgy.copy()
        self.of = lambda name: [getattr(t, name) for t in self.types]
        self.reach = max([t.b for t in self.energies if isinstance(t, fcc.Adhesion)], default=0.0)
        self._bound_shape()
        self._candidates(0.4)

    def _bound_shape(self):
        total = np.hypot(self.a, self.bb).sum(0)
        f = np.where(total > SHAPE_BOUND, SHAPE_BOUND / np.maximum(total, 1e-300), 1.0)
        self.a, self.bb = self.a * f, self.bb * f
        self.a0 = np.sqrt(1 - 0.5 * (self.a**2 + self.bb**2).sum(0))
        self.rmax = self.R0 * (self.a0 + np.hypot(self.a, self.bb).sum(0))

    def _image(self, dx, dy):
        return dx - self.box.Lx * np.rint(dx / self.box.Lx), dy - self.box.Ly * np.rint(dy / self.box.Ly)

    def _candidates(self, margin):
        """Pairs (i, j) that may touch while nothing moves by half the margin."""
        L = np.array([self.box.Lx, self.box.Ly])
        far = 2 * self.rmax.max() + self.reach + margin
        m = np.maximum(1, (L / far).astype(int))
        at = np.minimum((np.stack([self.x, self.y], 1) / L * m).astype(int), m - 1)
        cell = at[:, 0] + m[0] * at[:, 1]
        order = np.argsort(cell, kind="stable")
        first = np.searchsorted(cell[order], np.arange(m[0] * m[1] + 1))
        I, J = [], []
        around = {(ox % m[0], oy % m[1]) for ox in (-1, 0, 1) for oy in (-1, 0, 1)}
        for ox, oy in sorted(around):
            other = (at[:, 0] + ox) % m[0] + m[0] * ((at[:, 1] + oy) % m[1])
            count = first[other + 1] - first[other]
            i = np.repeat(np.arange(len(self.x)), count)
            within = np.arange(len(i)) - np.repeat(np.cumsum(count) - count, count)
            I.append(i)
            J.append(order[first[other][i] + within])
        i, j = np.concatenate(I), np.concatenate(J)
        dx, dy = self._image(self.x[i] - self.x[j], self.y[i] - self.y[j])
        near = (i != j) & (np.hypot(dx, dy) <= self.rmax[i] + self.rmax[j] + self.reach + margin)
        self.i, self.j = i[near], j[near]

    def forces(self):
        fcc = package()
        n, phi, R0 = self.n, self.phi, self.R0
        c, s = np.cos(n * self.th), np.sin(n * self.th)
        al, be = R0 * (self.a * c - self.bb * s), R0 * (self.a * s + self.bb * c)
        C, S = np.cos(n * phi), np.sin(n * phi)
        R = (R0 * self.a0)[:, None] + al.T @ C + be.T @ S
        R1 = be.T @ (n * C) - al.T @ (n * S)
        R2 = -(al.T @ (n**2 * C) + be.T @ (n**2 * S))
        q = np.sqrt(R**2 + R1**2)
        dphi = 2 * np.pi / self.nodes
        Q = q.sum(1) * dphi
        E, W = np.zeros(len(R0)), np.zeros(len(R0))
        GR, GD, GDD = np.zeros_like(R), np.zeros_like(R), np.zeros_like(R)
        J = Jr = np.zeros((len(self.types), len(self.types)))
        k = eps = 0.0
        for term in self.energies:
            on = np.ones(len(R0), bool)
            if isinstance(term, fcc.OnTypes):
                on, term = np.isin(self.t + 1, term.types), term.term
            if isinstance(term, fcc.Tension):
                E, W = E + on * term.eta * Q, W + on * term.eta
            elif isinstance(term, fcc.PerimeterElasticity):
                d = Q - term.p0 * math.sqrt(math.pi) * R0
                E, W = E + on * term.lam * d**2, W + on * 2 * term.lam * d
            elif isinstance(term, fcc.Bending):
                N, V, w = R**2 + 2 * R1**2 - R * R2, R**2 + R1**2, on[:, None] * dphi
                E = E + on * (term.a * N**2 * V**-2.5).sum(1) * dphi
                f = term.a * N * V**-3.5
                GR += w * f * (2 * V * (2 * R - R2) - 5 * N * R)
                GD += w * f * (8 * V * R1 - 5 * N * R1)
                GDD += w * f * (-2 * V * R)
            elif isinstance(term, fcc.Overlap):
                J, Jr = np.broadcast_to(term.J, J.shape), np.broadcast_to(term.Jrelated, J.shape)
            elif isinstance(term, fcc.LinearRepulsion):
                k = term.k
            elif isinstance(term, fcc.Adhesion):
                eps = term.a
        # contact pressure of every node against the neighbours around it
        i, j = self.i, self.j
        dx, dy = self._image(self.x[i] - self.x[j], self.y[i] - self.y[j])
        near = np.hypot(dx, dy) <= self.rmax[i] + self.rmax[j] + self.reach
        i, j, dx, dy = i[near], j[near], dx[near], dy[near]
        X, Y = R * np.cos(phi), R * np.sin(phi)
        P = np.zeros_like(R)
        for lo in range(0, len(i), 1 << 17):
            ii, jj = i[lo:lo + (1 << 17)], j[lo:lo + (1 << 17)]
            ux, uy = dx[lo:lo + (1 << 17), None] + X[ii], dy[lo:lo + (1 << 17), None] + Y[ii]
            d2 = ux**2 + uy**2
            pair, node = np.nonzero(d2 <= ((self.rmax[jj] + self.reach) ** 2)[:, None])
            ux, uy, dist = ux[pair, node], uy[pair, node], np.sqrt(d2[pair, node])
            bi, bj = ii[pair], jj[pair]
            z1 = (ux + 1j * uy) / np.maximum(dist, 1e-300)
            z, rj = z1 * z1, (R0 * self.a0)[bj]
            for m in range(self.K):
                rj = rj + al[m, bj] * z.real + be[m, bj] * z.imag
                z = z * z1
            depth = rj - dist
            related = self.parent[bi] == self.parent[bj]
            g = np.where(depth >= 0, np.where(related, Jr[self.t[bi], self.t[bj]], J[self.t[bi], self.t[bj]]), 0.0)
            g = g + k * np.maximum(depth, 0) - eps * ((depth < 0) & (depth > -self.reach))
            np.add.at(P, (bi, node), g)
        W = W[:, None] * dphi
        p = P * dphi
        GR, GD = GR + W * R / q + p * R, GD + W * R1 / q
        gx = (p * (R * np.cos(phi) + R1 * np.sin(phi))).sum(1)
        gy = (p * (R * np.sin(phi) - R1 * np.cos(phi))).sum(1)
        gth = (-p * R * R1).sum(1)
        for term in self.energies:
            if isinstance(term, fcc.HarmonicBond):
                p0, p1 = self.bonds[:, 0], self.bonds[:, 1]
                ex, ey = self._image(self.x[p0] - self.x[p1], self.y[p0] - self.y[p1])
                for grad, e in ((gx, ex), (gy, ey)):  # rest length 0: k times the separation
                    np.add.at(grad, p0, term.k * e)
                    np.add.at(grad, p1, -term.k * e)
        g0 = GR.sum(1)
        ga = (C @ GR.T) - (n * S) @ GD.T - (n**2 * C) @ GDD.T
        gb = (S @ GR.T) + (n * C) @ GD.T - (n**2 * S) @ GDD.T
        h0 = R0 * g0 / (2 * self.a0)
        gca = R0 * (ga * c + gb * s) - h0 * self.a
        gcb = R0 * (gb * c - ga * s) - h0 * self.bb
        return dict(GR=GR.T, GD=GD.T, GDD=GDD.T, P=P.T, gx=gx, gy=gy, gθ=gth, glab=np.vstack([g0, ga, gb]),
                    gcoef=np.vstack([R0 * g0, gca, gcb]), Ebody=E)

    def step(self, clock):
        f = self.forces()
        per = lambda name: np.array(self.of(name))[self.t]
        drag = np.array([t.parent_drag for t in self.types])[self.t]
        N = len(self.x)
        own = per("mu_r") * f["gx"], per("mu_r") * f["gy"]
        fx, fy = f["gx"].copy(), f["gy"].copy()
        np.add.at(fx, self.parent[drag], f["gx"][drag])
        np.add.at(fy, self.parent[drag], f["gy"][drag])
        moves = []
        for total, mine, head in ((fx, own[0], np.cos), (fy, own[1], np.sin)):
            swim = per("v0") * head(self.th)
            base = DT * (swim - per("mu_r") * total)  # substrate drag carries the children's forces
            moves.append(np.where(drag, base[self.parent] + DT * (swim - mine), base))
        if any(self.of("Dt")):
            raise NotImplementedError
        z3, _ = _normals(N, clock, 1, self.key, self.bits)
        self.th = self.th - DT * per("mu_theta") * f["gθ"] + np.sqrt(2 * per("Dr") * DT) * z3
        K = self.K
        self.a = self.a - DT * per("mu_ab") * f["gcoef"][1:1 + K]
        self.bb = self.bb - DT * per("mu_ab") * f["gcoef"][1 + K:]
        self._bound_shape()
        for name, img, L, d in (("x", "imgx", self.box.Lx, moves[0]), ("y", "imgy", self.box.Ly, moves[1])):
            v = getattr(self, name) + d
            w = np.floor(v / L)
            setattr(self, name, v - w * L)
            setattr(self, img, getattr(self, img) + w.astype(np.int32))

    def state(self):
        return dict(x=self.x, y=self.y, theta=self.th, coef=np.vstack([self.a0, self.a, self.bb]), imgx=None, imgy=None)

    def shape_index(self):
        n, c = self.n, np.cos(self.n * self.th)
        s = np.sin(n * self.th)
        al, be = self.a * c - self.bb * s, self.a * s + self.bb * c
        C, S = np.cos(n * self.phi), np.sin(n * self.phi)
        R = self.a0[:, None] + al.T @ C + be.T @ S
        R1 = be.T @ (n * C) - al.T @ (n * S)
        dphi = 2 * np.pi / self.nodes
        return np.sqrt(R**2 + R1**2).sum(1) * dphi / np.sqrt((R**2).sum(1) * dphi / 2)


def exact(case, seed):
    kind = case["kind"]
    if kind == "neighbors" or _bodies_of(case) * max(1, case["steps"]) > 340_000:
        return None
    if kind == "gradients":
        return _Model(case, *_system(case, seed)).forces()
    if kind == "pool":
        systems = [_system(case, seed + 7919 * k, nx, ny) for k, (nx, ny) in enumerate(_members(case))]
    else:
        systems = [_system(case, seed)]
    models = [_Model(case, *s) for s in systems]
    for m in models:
        for clock in range(case["steps"]):
            m.step(clock)
    if kind == "pool":
        states = [m.state() for m in models]
        got = {f: np.concatenate([s[f].ravel(order="F") for s in states]) for f in ("x", "y", "theta", "coef")}
        return dict(got, imgx=None, imgy=None)
    got = models[0].state()
    if case.get("observe"):
        got["shape_index"] = models[0].shape_index()
    return got
