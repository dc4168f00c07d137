"""The page-locked memory of query results, on the CPU: a stand-in library
whose allocations are ordinary memory."""

import ctypes as C
import gc
import sys

import numpy as np

from conftest import fcc

simulation = fcc.simulation


class Library:
    """fcc_host_alloc and fcc_host_free, with a count of the bytes locked."""

    def __init__(self):
        self.blocks, self.locked, self.calls = {}, 0, 0

    def fcc_host_alloc(self, size, out):
        buf = np.zeros(size, np.uint8)
        self.blocks[buf.ctypes.data] = buf
        C.cast(out, C.POINTER(C.c_void_p))[0] = buf.ctypes.data
        self.locked += size
        self.calls += 1
        return 0

    def fcc_host_free(self, ptr):
        self.locked -= len(self.blocks.pop(ptr))
        return 0


def test_a_collection_during_an_eviction(monkeypatch):
    """A block held by a reference cycle comes back when a collection runs,
    which may be at any step of a request that is making room (here one at
    every line): the request goes on, and the blocks serve later ones."""
    monkeypatch.setattr(simulation._ResultBlocks, "LIMIT", 5 << 20)
    blocks, lib = simulation._ResultBlocks(), Library()
    idle = [blocks.take(lib, 600_000) for _ in range(2)]
    cycles = []
    for k in range(40):  # sizes that no earlier block had
        cycles.append([blocks.take(lib, 4096 * (k + 2))])
        cycles[-1].append(cycles[-1])
    assert all(c[0] is not None for c in cycles)
    del idle

    def collect(frame, event, arg):
        if frame.f_code.co_filename != simulation.__file__:
            return None
        if cycles:
            cycles.pop()
            gc.collect()
        return collect
    before = sys.gettrace()
    sys.settrace(collect)
    try:
        big = blocks.take(lib, 1_000_000)
    finally:
        sys.settrace(before)
    assert len(cycles) < 35 and big is not None and big.nbytes >= 1_000_000
    assert lib.locked <= 5 << 20
    cycles.clear()
    del big
    gc.collect()
    calls = lib.calls
    assert blocks.take(lib, 1_000_000) is not None and lib.calls == calls


def query(lib, n=4096, rows=40):
    """Results of about 2 rows n doubles, as a gradients query asks for them."""
    return simulation.result_arrays(lib, ((n, rows), np.float64), ((n, rows), np.float64), ((n,), np.float64))


def in_place(lib, array):
    return any(a <= array.ctypes.data < a + len(b) for a, b in lib.blocks.items())


def test_results_that_are_kept_are_never_page_locked(monkeypatch):
    """A recorder keeps what it asked for: no query pays for page-locked memory
    that could serve only once."""
    monkeypatch.setattr(simulation, "_BLOCKS", simulation._ResultBlocks())
    lib = Library()
    kept = [query(lib, n) for n in (64, 4096, 3000) for _ in range(60)]
    states = [simulation.result_bodies(lib, n, 19)[0] for n in (64, 16384) for _ in range(60)]
    assert lib.calls == 0
    for a in kept:
        a[0][...], a[2][...] = 1.0, 2.0
    assert all((a[0] == 1).all() and (a[2] == 2).all() for a in kept)
    assert states[0].coef.shape == (19, 64) and states[0].coef.flags.f_contiguous


def test_results_that_come_back_are_page_locked_once(monkeypatch):
    """Dropped results turn into page-locked ones, a first result does not, and
    the price (twice, by the rule) is never above what they have saved."""
    monkeypatch.setattr(simulation, "_BLOCKS", simulation._ResultBlocks())
    blocks, lib = simulation._BLOCKS, Library()
    spent = saved = 0.0
    for k in range(30):
        calls = lib.calls
        got = query(lib)
        if lib.calls > calls:
            spent += blocks.price(lib.locked)
            assert 2 * spent <= saved
        elif not in_place(lib, got[0]):
            saved += blocks.saving(blocks.size_of(sum(a.nbytes for a in got)))
        del got
    assert lib.calls == 1 and in_place(lib, query(lib)[0])
    first = query(lib, 100_000)  # another size, too large for what is locked
    assert lib.calls == 1 and not in_place(lib, first[0])


def test_small_results_share_a_slab(monkeypatch):
    """The states of a pool's members, dropped between passes: in place after
    some passes, in one slab."""
    monkeypatch.setattr(simulation, "_BLOCKS", simulation._ResultBlocks())
    lib = Library()
    for _ in range(30):
        states = [simulation.result_bodies(lib, 64 + 8 * k, 19) for k in range(32)]
        for k, (b, h) in enumerate(states):
            for f in ("x", "y", "θ", "R0", "imgx", "imgy", "type", "parent"):
                getattr(b, f)[...] = k
            b.coef[...] = k
        for k, (b, h) in enumerate(states):  # no two overlap
            assert all((getattr(b, f) == k).all() for f in ("x", "y", "θ", "R0", "imgx", "imgy", "type", "parent", "coef"))
        where = [in_place(lib, b.x) for b, h in states]
        del states, b, h
    assert all(where) and lib.calls == 1


def test_slabs_hand_out_memory_once_and_get_all_of_it_back(monkeypatch):
    """Random requests and returns: blocks in use are disjoint and inside their
    slabs, the limit holds, and at the end every slab is whole again."""
    monkeypatch.setattr(simulation._ResultBlocks, "LIMIT", 6 << 20)
    monkeypatch.setattr(simulation._ResultBlocks, "SLAB", 1 << 20)
    blocks, lib = simulation._ResultBlocks(), Library()
    rng = np.random.default_rng(3)
    used = []
    for _ in range(3000):
        if used and rng.random() < 0.5:
            used.pop(rng.integers(len(used)))
        else:
            b = blocks.take(lib, int(np.exp(rng.uniform(0, np.log(2 << 20)))))
            if b is not None:
                used.append(b)
        spans = sorted((b.ctypes.data, b.ctypes.data + b.nbytes) for b in used)
        assert all(a[1] <= b[0] for a, b in zip(spans, spans[1:]))
        assert all(any(at <= lo and hi <= at + len(m) for at, m in lib.blocks.items()) for lo, hi in spans)
        assert blocks._total == lib.locked <= 6 << 20
    used.clear()
    del b
    blocks._sort_in()
    assert blocks._find(1 << 40) is None
    assert all(s.holes == [[0, s.size]] for s in blocks._slabs)
