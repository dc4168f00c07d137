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
        if frame.f_code.co_filename != simulation.__file__ or frame.f_code.co_name == "_give":
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
