"""The normalisation sum of the initial states in loop order, without its
chain of additions: grids whose cell count is below, at and beyond a
sub-tile (256 terms), a tile (8192) and several tiles, and a grid with many
empty cells.  The norms follow every rounding of the sums, and equal the
oracle's sequential ones bit for bit.  The kernel alone (compiled here) is
given terms at which its whole-number sums have to step aside: ties, negative
and non-finite terms, binade crossings."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import pyoracle as P
from vhlle_b200 import build
from vhlle_b200 import capi
from vhlle_b200 import ic_files as F
from vhlle_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz,xmax", [(9, 9, 3, 8.), (15, 17, 4, 8.), (32, 32, 8, 9.), (33, 31, 9, 9.),
                                           (41, 40, 16, 24.)])
@pytest.mark.parametrize("name", ["RHIC62", "LHC276"])
def test_norms_equal_the_sequential_sums(nx, ny, nz, xmax, name, tmp_path):
    s = W.glauber3d_setup(nx=nx, ny=ny, nz=nz, xmax=xmax, etamax=5.0)
    path = str(tmp_path / "sources.txt")
    F.write_glissando(path, F.synthetic_glissando_events(2, seed=nx))
    ev = F.read_glissando(path)
    su = capi.ic_setup(capi.IC_GLISSANDO, name)
    o, on = P.oracle_ic(s, 5, ev, su, crmath=True)
    h = capi.GpuHydro(s, upload=False)
    assert h.init_glissando(ev, su) == on
    assert np.array_equal(h.get_state(("Q",))["Q"], o["Q"], equal_nan=True)
    h.close()


# the sources' Gaussians: a reach narrower than the grid, of its side, and
# beyond it in one direction or both; more sources than one launch takes
@pytest.mark.parametrize("nx,ny,xmax,events", [(33, 35, 9., 2), (17, 17, 2.4, 2), (15, 33, 2., 2),
                                               (33, 9, 2., 2), (9, 9, 1., 2), (9, 9, 0.5, 2), (33, 33, 1.3, 5)])
@pytest.mark.parametrize("name", ["RHIC62", "LHC276"])
def test_source_reach_equals_the_oracle(nx, ny, xmax, events, name, tmp_path):
    s = W.glauber3d_setup(nx=nx, ny=ny, nz=9, xmax=xmax, etamax=5.0)
    s.dt = 0.02
    path = str(tmp_path / "sources.txt")
    F.write_glissando(path, F.synthetic_glissando_events(events, seed=ny))
    ev = F.read_glissando(path)
    su = capi.ic_setup(capi.IC_GLISSANDO, name)
    o, on = P.oracle_ic(s, 5, ev, su, crmath=True)
    h = capi.GpuHydro(s, upload=False)
    assert h.init_glissando(ev, su) == on
    assert np.array_equal(h.get_state(("Q",))["Q"], o["Q"], equal_nan=True)
    h.close()


@pytest.fixture(scope="module")
def seq_sum(tmp_path_factory):
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cpp", "seq_sum.cu")
    so = str(tmp_path_factory.mktemp("seq_sum") / "seq_sum.so")
    subprocess.run([build.nvcc_path(), *build.nvcc_flags(), "-I", build.CSRC, "-shared", src, "-o", so], check=True,
                   capture_output=True)
    f = ctypes.CDLL(so).seq_sum
    f.argtypes = [ctypes.c_void_p, ctypes.c_long, ctypes.POINTER(ctypes.c_double)]

    def run(t):
        t = np.ascontiguousarray(t, dtype=np.float64)
        out = ctypes.c_double(7.)
        assert f(t.ctypes.data, len(t), ctypes.byref(out)) == 0
        return out.value
    return run


def _ordered(t):
    s = 0.0
    for x in np.asarray(t, dtype=np.float64).tolist():
        s += x
    return s


def _same(a, b):
    return a == b or (np.isnan(a) and np.isnan(b))


@pytest.mark.parametrize("n", [0, 1, 2, 31, 255, 256, 257, 8191, 8192, 8193, 20000])
@pytest.mark.parametrize("form", ["zeros", "ones", "uniform", "decades", "sparse", "signs", "tiny", "huge"])
def test_sum_in_order_of_any_terms(seq_sum, n, form):
    rng = np.random.default_rng(n)
    t = {"zeros": np.zeros(n), "ones": np.ones(n), "uniform": rng.random(n), "decades": 10. ** rng.uniform(-20, 5, n),
         "sparse": np.where(rng.random(n) < 0.01, rng.random(n), 0.), "signs": rng.normal(size=n),
         "tiny": 5e-324 * rng.integers(0, 9, n), "huge": 1e305 * rng.random(n)}[form]
    assert seq_sum(t) == _ordered(t)


@pytest.mark.parametrize("at", [0, 1, 100, 254, 255, 256, 257, 511, 8190, 8191, 8192, 9000])
@pytest.mark.parametrize("first", [2. ** 52, 2. ** 52 + 1., 2. ** 53 - 1., 2. ** 53 - 3., 1.])
def test_sum_steps_aside(seq_sum, at, first):
    """One special term at a lane's, a run's (256 terms) and a tile's (8192)
    first and last places, after a sum with an even and an odd last bit and
    just below the next binade."""
    u = first * 2. ** -52 if first == 1. else 1.
    for x in (0.5 * u, 1.5 * u, 2.5 * u, 0.25 * u, 0.75 * u, -u, -0.5 * u, -0., np.inf, -np.inf, np.nan, first, 3. * first,
              1e308, 5e-324):
        for fill in (0., u, 2. * u):
            t = np.full(9500, fill)
            t[0] = first
            if at == 0:
                t[0] = x
                t[1] = first
            else:
                t[at] = x
            assert _same(seq_sum(t), _ordered(t)), (x, fill)
    # ties all the way: half a unit of the last place in every term
    t = np.full(9500, 0.5 * u)
    t[at] = first
    assert seq_sum(t) == _ordered(t)


@pytest.mark.parametrize("k", [1, 255, 256, 257, 2048, 8192])
def test_sum_crosses_binades(seq_sum, k):
    """The sum reaches a power of two exactly, one unit below and one above, at
    term k."""
    for e in (0, 10, 52):
        for off in (-1, 0, 1):
            t = np.empty(9000)
            t[1:k + 1] = 2. ** (e - 20)
            t[0] = 2. ** (e + 1) - k * 2. ** (e - 20) + off * 2. ** (e - 52)
            t[k + 1:] = 2. ** (e - 30) * 1.37
            assert seq_sum(t) == _ordered(t), (e, off)
