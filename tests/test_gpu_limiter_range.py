"""Limiter constants whose double is not finite, in the GPU's forms of the PDM limiter."""
import numpy as np
import pytest

from mhd3d_mpi_fortran_gb300 import MHDSolver, ensemble_step, ics
from mhd3d_mpi_fortran_gb300.abi import FP32, FP64, Params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,pdmb", [(FP64, 1.5e308), (FP32, 3e38)])
def test_constants_whose_double_is_infinite(precision, pdmb):
    """A finite constant of which twice the value is not: equal cells still give a zero slope (the
    fluxes and steps of a constant that limits as little; FP64 faces to rounding)."""
    n = (16, 12, 10)
    s = ics.empty_state(ics.grid(*n))
    s.rho[...] = 1.0
    s.rho[10:] = 0.5
    s.p[...] = 1.0
    s.vx[...] = 0.2
    with MHDSolver(Params(*n, precision=precision, pdmb=pdmb, tau=1e-3), s) as g, \
         MHDSolver(Params(*n, precision=precision, pdmb=1e6, tau=1e-3), s) as h:
        for d in range(3):
            for q in range(8):
                x, y = g.debug_fluxes()[d][q], h.debug_fluxes()[d][q]
                assert np.isfinite(x).all() and np.abs(x - y).max() <= 1e-14 * np.abs(y).max(), (d, q)
            assert np.array_equal(g.debug_emf()[d], h.debug_emf()[d])
        ensemble_step([g], 2)
        ensemble_step([h], 2)
        a, b = g.fetch(), h.fetch()
        for k in a:
            assert np.isfinite(a[k]).all() and np.abs(a[k] - b[k]).max() <= 1e-14, k
