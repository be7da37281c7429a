"""The normalisation sum of the initial states in loop order, without its
chain of additions: grids whose cell count is below, at and beyond a
sub-tile (256 terms), a tile (8192) and several tiles, and a grid with many
empty cells.  The norms follow every rounding of the sums, and equal the
oracle's sequential ones bit for bit."""
import numpy as np
import pytest

import pyoracle as P
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
