"""The face and con2prim kernels at the sizes and states where their splits
end: grids whose sides and cell counts leave remainders of a block's faces,
the smallest sides, and the root find and the table's nb = 0 row over states
and energies at their borders.  Everything is compared bit for bit."""
import ctypes

import numpy as np
import pytest

import pyoracle as P
from helpers import compare_states, gpu_state_as_oracle
from vhlle_b200 import capi
from vhlle_b200 import workloads as W

pytestmark = pytest.mark.gpu


# (2, 2): one face per direction; 64 and 65 cells: a block's faces, one more
@pytest.mark.parametrize("nx,ny,nz", [(2, 2, 1), (3, 2, 2), (4, 4, 4), (5, 13, 1), (8, 8, 1), (16, 5, 3),
                                      (33, 7, 2), (64, 3, 5), (65, 31, 1)])
@pytest.mark.parametrize("nb", [0.0, 0.3])
def test_steps_on_ragged_grids_equal_oracle(nx, ny, nz, nb):
    if nz > 1:
        s = W.glauber3d_setup(nx=nx, ny=ny, nz=nz, xmax=6.0, etamax=4.0, b=2.0, nb_peak=nb)
    else:
        s = W.batch_event(0, nz=1)
        g = W.Grid(nx, ny, 1, -6., 6., -6., 6., -0.5, 0.5)
        x, y, _ = g.coords()
        prof, _ = W.glauber_profile(3, 2.0, x, y)
        e = np.where(prof < 1e-3, 0., 40. * prof)[None]
        z = np.zeros_like(e)
        s.grid, s.m = g, (e.reshape(-1) > 0).astype(float)
        s.Q = W.conserved_from_primitive(s.tau0, e, z, nb * prof[None] * (e > 0), z, z, z).reshape(7, -1)
        s.zetaSparam = 0
    h, o = capi.GpuHydro(s), P.OracleRun(s)
    for _ in range(3):
        h.step(1)
        assert o.step(1) == 0
        bad = compare_states(gpu_state_as_oracle(h.get_state()), o.get_state())
        assert not bad, bad
    h.close()


def _axis(kind, n):
    if kind == "log":
        return np.exp(np.linspace(np.log(1e-4), np.log(1e3), n))
    if kind == "linear":
        return np.linspace(0.01, 50., n)
    if kind == "from_zero":
        return np.linspace(0., 50., n)
    return np.sort(np.random.default_rng(5).uniform(1e-3, 80., n))  # searched, not guessed


@pytest.mark.parametrize("kind", ["log", "linear", "from_zero", "irregular"])
@pytest.mark.parametrize("nbaxis", ["two", "many", "symmetric", "above_zero", "off_zero"])
def test_pressure_at_zero_charge(kind, nbaxis):
    """EoS::p (which the root find calls) at nb = 0 equals EoS::eos's p, which
    always takes the table's four corners, and the oracle's."""
    eg = _axis(kind, 301)
    ng = {"two": np.array([0., 1.]), "many": np.linspace(0., 1., 40), "symmetric": np.linspace(-1., 1., 41),
          "above_zero": np.linspace(0.1, 1., 7), "off_zero": np.linspace(-0.95, 1., 40)}[nbaxis]
    E, B = np.meshgrid(eg, ng)  # [in][ie]
    p = (0.3 * E - 0.01 + 0.02 * B * B).reshape(-1)
    eos = W.EosTable(kind=1, egrid=eg, ngrid=ng, p=p, T=(0.1 + 0.05 * E ** 0.25).reshape(-1), mub=B.reshape(-1))
    s = W.small_glauber3d(5, 5)
    s.eos = eos
    rng = np.random.default_rng(2)
    e = np.concatenate([eg, np.nextafter(eg, 0), np.nextafter(eg, 1e9), rng.uniform(-1e-3, 100., 2000),
                        10. ** rng.uniform(-300, 9, 2000), [0., -0., 1e-308, 5e-324, 1e12, 1e300]])
    h, o = capi.GpuHydro(s), P.OracleRun(s)
    for nb in (0., -0.):
        nbs = np.full_like(e, nb)
        got = h.eos6(e, nbs)
        assert np.array_equal(got[:, 4], got[:, 0], equal_nan=True)
        ok = e >= 0  # (EoS1f's eos does not return for e < 0)
        assert np.array_equal(got[ok, 4], o.eos6(e, nbs)[ok, 4], equal_nan=True)
    h.close()


@pytest.mark.parametrize("kind", ["log", "linear", "from_zero", "irregular"])
@pytest.mark.parametrize("nbaxis", ["two", "many", "symmetric", "above_zero", "off_zero"])
def test_lookup_with_charge(kind, nbaxis):
    """The table at nb != 0 (its packed axis, its last cells, outside it)
    equals the oracle's in every output."""
    eg = _axis(kind, 301)
    ng = {"two": np.array([0., 1.]), "many": np.linspace(0., 1., 40), "symmetric": np.linspace(-1., 1., 41),
          "above_zero": np.linspace(0.1, 1., 7), "off_zero": np.linspace(-0.95, 1., 40)}[nbaxis]
    E, B = np.meshgrid(eg, ng)
    s = W.small_glauber3d(5, 5)
    s.eos = W.EosTable(kind=1, egrid=eg, ngrid=ng, p=(0.3 * E - 0.01 + 0.02 * B * B).reshape(-1),
                       T=(0.1 + 0.05 * E ** 0.25 + 0.01 * B).reshape(-1), mub=(B * (1. + 0.01 * E)).reshape(-1))
    rng = np.random.default_rng(3)
    axis = np.concatenate([ng, np.nextafter(ng, -9), np.nextafter(ng, 9), [-3., 3., -0., 1e-300, -1e-300, 1e9]])
    ends = np.concatenate([eg[:3], eg[-3:], np.nextafter(eg[:3], 1e9), np.nextafter(eg[-3:], 0), [0., 5e-324, 1e9]])
    e, nb = (a.reshape(-1) for a in np.meshgrid(ends, axis))
    e = np.concatenate([e, rng.uniform(0., 100., 3000), 10. ** rng.uniform(-9, 4, 3000), rng.choice(eg, 500)])
    nb = np.concatenate([nb, rng.uniform(-1.5, 1.5, 6000), rng.choice(axis, 500)])
    h, o = capi.GpuHydro(s), P.OracleRun(s)
    assert np.array_equal(h.eos6(e, nb), o.eos6(e, nb), equal_nan=True)
    h.close()


@pytest.mark.parametrize("eos", ["table", "nb_table", "conformal", "chiral"])
def test_root_find_equals_oracle(eos):
    """transformPV from vacuum and rest to |M| > Q_t, over 24 decades, with and
    without charge."""
    torch = pytest.importorskip("torch")
    s = W.small_glauber3d(5, 5)
    s.eos = {"table": W.make_cs2_table, "nb_table": lambda: W.nb_table(400, 21), "chiral": W.chiral_eos,
             "conformal": lambda: W.EosTable(kind=0)}[eos]()
    rng = np.random.default_rng(11)
    n = 20000
    T = 10. ** rng.uniform(-20, 4, n)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    M = T * np.where(rng.random(n) < 0.5, rng.uniform(0., 1.2, n), 1. - 10. ** rng.uniform(-16, 0, n))
    Q = np.zeros((n, 7))
    Q[:, 0] = T
    Q[:, 1:4] = M[:, None] * d
    Q[n // 2:, 4] = T[n // 2:] * 10. ** rng.uniform(-6, 0, n - n // 2)
    Q[n // 2:, 5] = 0.4 * Q[n // 2:, 4]
    Q[::11, 1:4] = 0.           # at rest
    Q[::13, 3] = 0.
    Q[::17, 0] = 0.             # vacuum
    Q[::19, 0] *= -1.
    Q[::23, 4] = -0.
    h, o = capi.GpuHydro(s), P.OracleRun(s)
    dQ = torch.from_numpy(np.ascontiguousarray(Q.T)).cuda()
    out = torch.empty((8, n), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    h._check(h.L.vh_transform_pv(h.h, ctypes.c_void_p(dQ.data_ptr()), n, ctypes.c_void_p(out.data_ptr())))
    h.sync()
    assert np.array_equal(out.cpu().numpy().T, o.transform_pv(Q), equal_nan=True)
    h.close()


# the faces that can carry a flux are listed where they fill the chip (more
# than 1184 blocks of 64 faces, 1776 in 2+1D, and there with a table only):
# sizes on both sides of the line, mostly vacuum, with a filled event and with
# cells not filled yet (m < 1)
@pytest.mark.parametrize("nx,ny,nz", [(29, 29, 29), (29, 30, 29), (31, 29, 29), (33, 64, 32), (197, 191, 1),
                                      (200, 199, 1)])
@pytest.mark.parametrize("nb", [0.0, 0.3])
def test_listed_faces_equal_oracle(nx, ny, nz, nb):
    if nz > 1:
        s = W.glauber3d_setup(nx=nx, ny=ny, nz=nz, xmax=14.0, etamax=7.0, b=9.0, nb_peak=nb)
    else:
        s = W.gubser_setup(nx, ny)
        if nb:  # the conformal flow's state under a table
            s.eos = W.nb_table(400, 40)
        s.dt = 0.2 * min(s.grid.dx, s.grid.dy)
        x, y, _ = s.grid.coords()
        far = (np.hypot(*np.meshgrid(x, y)) > 2.5).reshape(-1)
        s.Q = s.Q.reshape(7, -1).copy()
        s.Q[:, far] = 0.
        s.m = np.where(far, 0., s.m.reshape(-1))
    rng = np.random.default_rng(4)
    s.m = np.where((s.m > 0) & (rng.random(s.m.shape) < 0.02), 0.4, s.m)  # matter in cells not filled
    h, o = capi.GpuHydro(s), P.OracleRun(s)
    for _ in range(3):
        h.step(1)
        assert o.step(1) == 0
        bad = compare_states(gpu_state_as_oracle(h.get_state()), o.get_state())
        assert not bad, bad
    h.close()


# the ideal update runs on a list above 1184 blocks of 128 cells: sizes on both
# sides of the line, the last block with and without a remainder, and the
# temperatures that the vorticity takes from it
@pytest.mark.parametrize("nx,ny,nz", [(48, 48, 49), (49, 49, 48), (64, 64, 28), (337, 339, 1), (64, 64, 37),
                                      (54, 53, 53), (64, 64, 38), (390, 391, 1)])
def test_listed_updates_equal_oracle(nx, ny, nz):
    test_listed_faces_equal_oracle(nx, ny, nz, 0.0)


@pytest.mark.parametrize("nx,ny", [(238, 238), (239, 238), (337, 339), (390, 391)])
def test_listed_faces_and_updates_in_2d_equal_oracle(nx, ny):
    test_listed_faces_equal_oracle(nx, ny, 1, 0.3)


@pytest.mark.parametrize("nx,ny,nz", [(49, 49, 48), (54, 53, 54)])
def test_listed_update_with_vorticity_equals_oracle(nx, ny, nz):
    s = W.glauber3d_setup(nx=nx, ny=ny, nz=nz, xmax=14.0, etamax=7.0, b=9.0, nb_peak=0.3)
    h, o = capi.GpuHydro(s), P.OracleRun(s, vorticity=True)
    h.enable_vorticity()
    for _ in range(2):
        h.step(1)
        assert o.step(1) == 0
        assert np.array_equal(h.get_dbeta(), o.dbeta, equal_nan=True)
    bad = compare_states(gpu_state_as_oracle(h.get_state()), o.get_state())
    assert not bad, bad
    h.close()


@pytest.mark.parametrize("viscous", [False, True])
@pytest.mark.parametrize("nb", [0.0, 0.02])
def test_full_listed_grid_equals_oracle(viscous, nb):
    """Matter in every cell of a grid whose faces and cells are listed."""
    s = W.glauber3d_setup(nx=54, ny=53, nz=55, xmax=9.0, etamax=5.0, eos=W.nb_table(400, 40) if nb else None)
    N = s.grid.ncells
    rng = np.random.default_rng(6)
    e = 1. + rng.random(N)
    s.Q = W.conserved_from_primitive(s.tau0, e, e / 4, nb * e, 0.2 + 0. * e, -0.1 + 0. * e, 0. * e).reshape(7, -1)
    s.m = np.ones(N)
    s.tr = dict(s.tr, etaS0=0.08 if viscous else 0.0, zetaS0=0.0)
    h, o = capi.GpuHydro(s), P.OracleRun(s)
    h.step(2)
    assert o.step(2) == 0
    bad = compare_states(gpu_state_as_oracle(h.get_state()), o.get_state())
    assert not bad, bad
    h.close()


@pytest.mark.parametrize("form", ["ordinary", "tiny", "mixed", "zero", "no_shear", "bump", "large_dt"])
def test_relaxation_ranges_equal_oracle(form):
    """Shear and bulk stresses inside and outside the ranges in which the
    relaxation divides without tests (2^+-140), exact zeros, eta/s = 0 and a
    zeta/s that falls off to 1e-200."""
    s = W.glauber3d_setup(nx=17, ny=15, nz=9, xmax=7.0, etamax=4.0, b=2.0, dt=0.2 if form == "large_dt" else 0.05)
    rng = np.random.default_rng(8)
    N = s.grid.ncells
    e = s.Q.reshape(7, N)[0] / s.tau0
    mag = {"ordinary": 0., "tiny": -60., "mixed": None, "zero": 0.}.get(form, 0.)
    ex = rng.uniform(-220., 0., (10, N)) if mag is None else np.full((10, N), mag)
    s.pi = 0.05 * e * rng.normal(size=(10, N)) * 10. ** ex
    s.Pi = 0.02 * e * rng.normal(size=N) * 10. ** ex[0]
    if form == "zero":
        s.pi[rng.random((10, N)) < 0.7] = 0.
        s.Pi[:] = 0.
    if form == "no_shear":
        s.tr = dict(s.tr, etaS0=0.0, zetaS0=0.1)
    if form == "bump":
        s = W.with_zeta_bump(s, width_T=0.008)
    h, o = capi.GpuHydro(s), P.OracleRun(s, crmath=form == "bump")
    for _ in range(3):
        h.step(1)
        assert o.step(1) == 0
        bad = compare_states(gpu_state_as_oracle(h.get_state()), o.get_state())
        assert not bad, bad
    h.close()


def _torn(nx, ny, nz, seed, viscous):
    """Random matter and flow, at a tau so small beside the step that the
    predictor's source makes Qh_t < 0 in some cells."""
    s = W.gubser_setup(nx, ny) if nz == 1 else W.glauber3d_setup(nx=nx, ny=ny, nz=nz, xmax=5.0, etamax=1.0)
    s.dt = 0.45 * min(s.grid.dx, s.grid.dy)
    s.tau0 = 0.6 * s.dt
    rng = np.random.default_rng(seed)
    N = s.grid.ncells
    e, v, c, ph = (10. ** rng.uniform(-3, 1, N), 0.98 * rng.random(N), rng.uniform(-1, 1, N),
                   rng.uniform(0, 2 * np.pi, N))
    r = v * np.sqrt(1. - c * c)
    s.Q = W.conserved_from_primitive(s.tau0, e, e / 3, 0. * e, r * np.cos(ph), r * np.sin(ph), v * c).reshape(7, -1)
    s.m = np.ones(N)
    s.tr = dict(s.tr, etaS0=0.2 if viscous else 0.0, zetaS0=0.0)
    return s


@pytest.mark.parametrize("nx,ny,nz", [(6, 5, 1), (4, 11, 1), (21, 21, 1), (47, 33, 1), (9, 8, 3), (4, 4, 4), (9, 3, 8)])
@pytest.mark.parametrize("viscous", [False, True])
def test_negative_rows_beside_the_edge_equal_oracle(nx, ny, nz, viscous):
    """Sides of 4 or fewer: the cells that the ghost copy reads are copied into
    too.  A row with Qh_t < 0 there is zeroed while the edge's threads read it;
    they must store zeros, not a part of the row."""
    def sources(n):
        return sorted({min(2, n - 1), max(n - 3, 0)} if n > 4 else {min(2, n - 1)})
    found = 0
    for seed in range(400):
        s = _torn(nx, ny, nz, seed, viscous)
        o = P.OracleRun(s)
        if o.step(1):
            continue
        st = o.get_state()
        q, before = (st[k].reshape(7, nz, ny, nx)[0] for k in ("Qh", "Qprev"))
        zeroed = (q == 0) & (before > 0)
        if not (zeroed[:, sources(ny), :].any() or zeroed[:, :, sources(nx)].any()):
            continue
        h = capi.GpuHydro(s)
        h.step(1)
        bad = compare_states(gpu_state_as_oracle(h.get_state()), st)
        h.close()
        assert not bad, (seed, bad)
        found += 1
        if found == 8:
            break
    assert found


@pytest.mark.parametrize("nx,ny,nz", [(9, 8, 1), (21, 20, 1), (9, 8, 7), (5, 6, 4), (12, 11, 10)])
def test_root_finds_of_a_step(nx, ny, nz):
    """Matter everywhere, moving, at a clock without rounding: a viscous step
    solves two states per face and one per cell in each pass, then D and C of
    every cell, and A of the cells that the ghost copy writes only, once."""
    s = W.glauber3d_setup(nx=nx, ny=ny, nz=nz, xmax=5.0, etamax=3.0) if nz > 1 else W.gubser_setup(nx, ny)
    s.tau0, s.dt = 1.0, 0.0625
    s.eos = W.EosTable(kind=0)
    N = s.grid.ncells
    one = np.ones(N)
    s.Q = W.conserved_from_primitive(s.tau0, 10. * one, 10. / 3 * one, 0. * one, 0.3 * one, 0.2 * one,
                                     0.1 * one).reshape(7, -1)
    s.m = one
    s.tr = dict(s.tr, etaS0=0.1, zetaS0=0.0)
    h = capi.GpuHydro(s)
    h.con2prim_stats(True)
    h.step(1)
    calls = h.con2prim_stats(False)[0]
    h.close()
    faces = (nx - 1) * ny * nz + nx * (ny - 1) * nz + nx * ny * (nz - 1)
    inner = max(nx - 4, 0) * max(ny - 4, 0) * max(nz - 4, 0)
    assert calls == 2 * (2 * faces + N) + 2 * N + (N - inner)
