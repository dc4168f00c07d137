"""Device helpers on their own (marked ``gpu``): device_units.cu, compiled with
the library's flags, calls them at the arguments that whole simulations reach
rarely or not at all."""

import ctypes as C
import os
import re
import shlex
import subprocess

import numpy as np
import pytest

from conftest import PKG_DIR

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def unit(tmp_path_factory):
    """unit(name, *arguments): arrays go as pointers, the returned CUDA error
    must be 0."""
    make = open(os.path.join(PKG_DIR, "csrc", "Makefile")).read().replace("\\\n", " ")
    flags = re.search(r"^NVFLAGS\s*:=(.*)$", make, re.M)[1]
    flags = [f for f in shlex.split(flags.replace("$(HOSTCXX)", "g++")) if f not in ("-Xptxas", "-v")]
    so = str(tmp_path_factory.mktemp("units") / "units.so")
    nvcc = "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc if os.path.exists(nvcc) else "nvcc", *flags, "-shared", "-o", so,
                    os.path.join(HERE, "device_units.cu")], check=True)
    lib = C.CDLL(so)

    def call(name, *args):
        c = {int: C.c_int, float: C.c_double}
        got = getattr(lib, name)(*(c[type(a)](a) if type(a) in c else C.c_void_p(a.ctypes.data) for a in args))
        assert got == 0, (name, got)
    return call


@pytest.mark.parametrize("nθ", [5, 24, 37, 40])
def test_user_term_that_is_singular_on_a_circle(unit, nθ):
    """A term whose derivative does not exist where R' = R'' = 0, on deformed
    contours: the slots beyond a contour add nothing, the others w dq (the same
    IEEE operations in numpy; R' / s to one rounding of each: 4 ulp)."""
    rng = np.random.default_rng(nθ)
    R, R1, R2 = (v + rng.standard_normal((32, 5)) * 0.2 for v in (1.0, 0.0, 0.0))
    out = [np.zeros((32, 5)) for _ in range(3)]
    w = 0.7
    unit("unit_user_gradients", nθ, R, R1, R2, w, *out)
    node = np.arange(32)[:, None] % 8 + 8 * np.arange(5)
    s = np.sqrt(R1 ** 2 + R2 ** 2)
    for got, want in zip(out, (0 * R, w * R1 / s, w * R2 / s)):
        assert np.array_equal(got[node >= nθ], np.zeros((node >= nθ).sum()))
        assert np.allclose(got[node < nθ], want[node < nθ], rtol=4 * 2.0 ** -52, atol=0)


def test_fp64_roots_over_the_exponents(unit):
    """rsqrt_normal and sqrt_normal against 80-bit roots.  Bounds in units in
    the last place: the final rounding (1/2), for the reciprocal the rounding of
    x y in the residual (half of 2^-53, at most 1/2 ulp) and the cubic's
    remainder (5/16 (2^-19)^3, 0.02 ulp), for the root the rounding of a residual
    that is subnormal for the smallest x (1/4): 1.1 and 1."""
    rng = np.random.default_rng(1)
    tiny, huge = np.finfo(np.float64).tiny, np.finfo(np.float64).max
    edge = np.ldexp(1.0, np.arange(-1021, 1024))
    x = np.concatenate([np.ldexp(1 + rng.random(400_000), rng.integers(-1022, 1024, 400_000)),
                        np.nextafter(edge, 0), edge, np.nextafter(edge, np.inf), 1 + rng.random(100_000) * 3,
                        [tiny, huge]])
    inv, root = np.zeros_like(x), np.zeros_like(x)
    unit("unit_roots", x, len(x), inv, root)
    exact = np.sqrt(x.astype(np.longdouble))
    for got, want, bound in ((inv, 1 / exact, 1.1), (root, exact, 1.0)):
        ulp = np.spacing(want.astype(np.float64)).astype(np.longdouble)
        assert (np.abs(got - want) / ulp).max() <= bound
    x = np.array([0.0, 5e-324, 1e-320, 1e-310, np.nextafter(tiny, 0), np.inf, np.nan])
    inv, root = np.zeros_like(x), np.zeros_like(x)
    unit("unit_roots", x, len(x), inv, root)
    assert root[0] == 0 and root[5] == np.inf and np.isnan(root[6])
    # below the smallest normal number: within that number's root of the value
    assert (np.abs(root[1:5] - np.sqrt(x[1:5])) <= np.sqrt(tiny)).all()


@pytest.mark.parametrize("n,cells", [(1, 1), (5, 512), (70, 1300), (1000, 513)])
def test_loading_a_state_clears_the_counts_of_an_abandoned_rebuild(unit, n, cells):
    """A launch that gave up at a barrier between the count and the scatter of a
    rebuild leaves bodies counted; added to by the next rebuild they would put
    bodies beyond the sorted list's end.  Loading a state (which also renews the
    barriers) starts from zero."""
    count = np.full(cells, 7, np.int32)
    total = np.full(-(-cells // 512), 9, np.int32)
    unit("unit_init_counts", n, cells, count, total)
    assert not count.any() and not total.any()
