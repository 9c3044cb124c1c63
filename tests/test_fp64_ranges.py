"""FP64 step at the ends of its range, against the oracle."""
import numpy as np
import pytest

from mhd3d_mpi_fortran_gb300 import MHDSolver, ics
from mhd3d_mpi_fortran_gb300.abi import Params

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
