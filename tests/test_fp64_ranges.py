"""FP64 step at the ends of its range, against the oracle."""
import ctypes

import numpy as np
import pytest

from mhd3d_mpi_fortran_gb300 import MHDSolver, abi, ics
from mhd3d_mpi_fortran_gb300.abi import DT_CFL, Params

RECONS = [1, 2, 3, 4, 5]


def flow(nx, ny, nz, seed=0):
    """Smooth rho and p, velocities of 0.5 to 0.6 along every axis, a weak random face field."""
    s = ics.empty_state(ics.grid(nx, ny, nz))
    r = np.random.default_rng(seed)
    x, y, z = [c.reshape(sh) for c, sh in zip(s.grid.centres(), ((-1, 1, 1), (1, -1, 1), (1, 1, -1)))]
    s.rho[...] = 1.0 + 0.2 * np.sin(2 * np.pi * (x + y)) + 0.0 * z
    s.p[...] = 0.6 + 0.1 * np.cos(2 * np.pi * (y + z)) + 0.0 * x
    for v in (s.vx, s.vy, s.vz):
        v[...] = 0.5 + 0.1 * r.random(v.shape)
    for b in (s.bi, s.bj, s.bk):
        b[...] = 0.05 * r.standard_normal(b.shape)
    return s


def same(a, b, tol):
    """Finite in the same places, and equal there to tol of the largest value."""
    ok = np.isfinite(b)
    return np.array_equal(np.isfinite(a), ok) and np.abs(a - b)[ok].max() <= tol * np.abs(b[ok]).max()


def fluxes_match(prm, s, tol=1e-13):
    from oracle.oracle import OracleSolver
    with MHDSolver(prm, s) as g:
        fg = g.debug_fluxes()
    fo = OracleSolver(prm, s).fluxes()
    for d in range(3):
        for q in range(8):
            assert same(fg[d][q], fo[d][q], tol), (d, q)
    return fo


@pytest.mark.gpu
@pytest.mark.parametrize("where", [(slice(7, 8),) * 3, (slice(7, 8), slice(None), slice(None)),
                                   (slice(7, 9), slice(None), slice(None))])
@pytest.mark.parametrize("recon", RECONS)
def test_zero_pressure(recon, where):
    """A cell, a layer and two layers of p = 0 in moving gas: fluxes of every reconstruction, and
    steps of those whose limiter keeps face pressures from going below zero."""
    from oracle.oracle import OracleSolver
    s = flow(12, 9, 10)
    s.p[where] = 0.0
    prm = Params(12, 9, 10, reconop=recon, tau=1e-3)
    fluxes_match(prm, s)
    if recon in (1, 2, 5):
        with MHDSolver(prm, s) as g:
            g.step(4)
            a = g.fetch()
        o = OracleSolver(prm, s)
        o.step(4)
        for k, b in o.fetch().items():
            assert np.isfinite(b).all() and same(a[k], b, 1e-11), k


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1e-160, 1e160])
def test_pressure_times_density_beyond_the_range(scale):
    """rho and p whose quotient is ordinary and whose product is zero or infinite."""
    s = flow(12, 9, 10)
    s.rho *= scale
    s.p *= scale
    for b in (s.bi, s.bj, s.bk):
        b *= np.sqrt(scale)
    fo = fluxes_match(Params(12, 9, 10, tau=1e-3), s)
    assert np.isfinite(fo[0][0]).all()


@pytest.mark.gpu
def test_tails_of_the_moments():
    """Two streams that leave a face: only the tails of the moments cross it.  Constant states on
    either side (so that the face states are the cells'), one argument z = sqrt(rho / 2p) |v| per
    row from 0.3 to 25; mass flux and magnetic stress relative to 40 digits.  The bound: z is off by
    5 half units of rounding, which a tail takes 2 z^2 times, and v v0 and b cancel to 1 / 2z^2."""
    mp = pytest.importorskip("mpmath")
    n = 64
    s = ics.empty_state(ics.grid(16, n, 8))
    z = np.geomspace(0.3, 25.0, n)
    row = np.ones(s.vx.shape[1])
    row[4:-4] = z
    left = (np.arange(s.vx.shape[0]) < 12).reshape(-1, 1, 1)
    s.rho[...] = np.where(left, 1.0, 2.0 ** -10)
    s.p[...] = np.where(left, 0.7, 1.3 * 2.0 ** -10)
    s.vx[...] = np.where(left, -1.0, 1.0) * np.sqrt(2 * s.p / s.rho) * row.reshape(1, -1, 1)
    s.bj[...] = 0.4
    with MHDSolver(Params(16, n, 8, tau=1e-3), s) as g:
        f = g.debug_fluxes()[0]
    mp.mp.dps = 40
    for j in range(n):
        mass = stress = 0
        for side, i in ((1, 11), (-1, 12)):
            rho, p, v, b2 = (mp.mpf(float(a)) for a in (s.rho[i, 4 + j, 4], s.p[i, 4 + j, 4], s.vx[i, 4 + j, 4], 0.4 ** 2))
            a, am = mp.sqrt(rho / (2 * p)), mp.sqrt(rho / (2 * p + b2))
            mass += rho * (v * mp.erfc(-side * a * v) / 2 + side * mp.exp(-(a * v) ** 2) / (2 * a * mp.sqrt(mp.pi)))
            stress += b2 / 2 * mp.erfc(-side * am * v) / 2
        for got, ref, k in ((f[0], mass, 0), (f[5], stress, 5)):
            err = abs(float((mp.mpf(float(got[8, j, 3])) - ref) / ref))
            assert err <= 4e-15 * (1 + z[j] ** 2), (z[j], k, err)


def test_table_rows_of_the_library():
    """The rows that the library uploads, as the kernels evaluate them: relative errors of the
    polynomials, the last row's outer edge included (1.1e-16: first terms left out and coefficients;
    as much again for the roundings of the evaluation)."""
    mp = pytest.importorskip("mpmath")
    lib = abi.load()
    fill = lib._ZN3mhd11gauss_tableEPd
    fill.argtypes, fill.restype = [ctypes.c_void_p], None
    out = np.zeros((209, 20))
    fill(out.ctypes.data)
    mp.mp.dps = 30
    r = np.random.default_rng(1)
    for i in range(0, 209, 3):
        c = i / 32.0
        for d in np.concatenate([[-1 / 64, 1 / 64, 0.0], r.uniform(-1 / 64, 1 / 64, 5)]):
            h = e = 0.0
            for k in range(9, -1, -1):
                h, e = h * d + out[i, k], e * d + out[i, 10 + k]
            x = mp.mpf(c) + mp.mpf(d)
            assert abs(h / (mp.erfc(x) / 2) - 1) <= 3.3e-16, (c, d)
            assert abs(e / (mp.exp(-x * x) / (2 * mp.sqrt(mp.pi))) - 1) <= 3.3e-16, (c, d)


@pytest.mark.gpu
@pytest.mark.parametrize("vals", [dict(p=-0.5), dict(rho=-0.5), dict(rho=-0.5, p=-0.5), dict(rho=0.0), dict(p=0.0),
                                  dict(rho=0.0, p=0.0)])
def test_cfl_dt_of_unphysical_cells(vals):
    """A cell of negative or zero density or pressure in a strong field, where its dt would be the
    smallest: the speed is NaN where get_dt's three roots give NaN, and drops out."""
    from oracle.oracle import OracleSolver
    s = flow(12, 9, 10)
    s.bi[7:9, 6, 6] = 8.0
    for k, x in vals.items():
        getattr(s, k)[7, 6, 6] = x
    prm = Params(12, 9, 10, dt_mode=DT_CFL, tau=1e-3)
    with MHDSolver(prm, s) as g:
        got = g.diagnostics()["dt_cfl"]
    ref = OracleSolver(prm, s).diagnostics()["dt_cfl"]
    assert np.isfinite(ref) and got == pytest.approx(ref, rel=1e-14)


@pytest.mark.gpu
@pytest.mark.parametrize("recon", [3, 4])
def test_weno_weights_beside_a_huge_jump(recon):
    """Smoothness indicators 1e166 apart: the smooth candidates keep their weights."""
    s = flow(16, 9, 10)
    s.vz[8:] = 1e80
    s.vz[:8] = 0.3
    fo = fluxes_match(Params(16, 9, 10, reconop=recon, tau=1e-3), s)
    assert all(np.isfinite(q).all() for q in fo[0])


@pytest.mark.gpu
@pytest.mark.parametrize("recon", RECONS)
def test_subnormal_density(recon):
    """Density and pressure of 1e-309, whose reciprocals are infinite: v = (rho v) / rho is still a
    number.  They hold 47 bits, so a quotient of two is good to 2^-46 and the bound is that of other steps."""
    from oracle.oracle import OracleSolver
    s = flow(12, 9, 10)
    s.rho *= 1e-309
    s.p *= 1e-309
    for b in (s.bi, s.bj, s.bk):
        b[...] = 0.0
    prm = Params(12, 9, 10, reconop=recon, tau=1e-3)
    with MHDSolver(prm, s) as g:
        g.step(2)
        a = g.fetch()
    o = OracleSolver(prm, s)
    o.step(2)
    for k, b in o.fetch().items():
        assert np.isfinite(b).all(), k
        assert not b.any() if k[0] == "b" else same(a[k], b, 1e-11), k
