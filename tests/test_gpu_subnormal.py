"""FP32 face fluxes of states whose reciprocals or roots have subnormal operands."""
import numpy as np
import pytest

from mhd3d_mpi_fortran_gb300 import MHDSolver, ics
from mhd3d_mpi_fortran_gb300.abi import FP32, FP64, Params

pytestmark = pytest.mark.gpu


# (the fluxes of rho = 3e-39 through the areas of a mapped grid, 2e-41, have 14 bits left: Cartesian only)
@pytest.mark.parametrize("rho,p,mapped", [(r, p, m) for r, p in ((1e-30, 4e-39), (1e-37, 10.0), (2e-39, 1.0))
                                          for m in (False, True)] + [(3e-39, 4e-39, False)])
def test_subnormal_pressure_and_lambda(rho, p, mapped):
    """2p or rho / 2p below 1.2e-38 with its reciprocal or root in range: mass fluxes against the
    FP64 step (2e-5: the operands hold 20 of 24 bits)."""
    n = (12, 10, 9)
    s = ics.empty_state(*ics.mapped_grid(*n)) if mapped else ics.empty_state(ics.grid(*n))
    r = np.random.default_rng(1)
    c = np.sqrt(p / rho)
    s.rho[...] = rho * (1.0 + 0.1 * r.random(s.rho.shape))
    s.p[...] = p * (1.0 + 0.1 * r.random(s.p.shape))
    for v in (s.vx, s.vy, s.vz):
        v[...] = c * (0.3 + 0.1 * r.random(v.shape))
    with MHDSolver(Params(*n, precision=FP64, tau=1e-3), s) as h:
        ref = h.debug_fluxes()
    with MHDSolver(Params(*n, precision=FP32, tau=1e-3), s) as g:
        got = g.debug_fluxes()
    for d in range(3):
        assert np.abs(got[d][0] - ref[d][0]).max() <= 2e-5 * np.abs(ref[d][0]).max(), d
