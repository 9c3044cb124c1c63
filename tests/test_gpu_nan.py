"""Reconstructions beside NaN cells, against the oracle."""
import numpy as np
import pytest

from mhd3d_mpi_fortran_gb300 import MHDSolver
from mhd3d_mpi_fortran_gb300.abi import EMF_LFM, EMF_YEE, FP32, FP64, Params
from test_fp64_ranges import flow, same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("field", ["rho", "vx", "vy", "vz", "p", "bi"])
@pytest.mark.parametrize("emf,precision", [(EMF_LFM, FP64), (EMF_YEE, FP64), (EMF_YEE, FP32)])
def test_pdm_beside_a_nan(emf, precision, field, sign):
    """Fluxes and edge EMFs of PDM with one NaN in a field, of either sign: NaN in the same places as in
    the oracle, and the same values beside them (a clamped NaN interpolant leaves the larger near cell).
    The corner velocities of the LFM EMF take one of two estimates, where the oracle multiplies the
    other by zero: an edge is NaN for a velocity of its four cells, or of the estimate taken."""
    from oracle.oracle import OracleSolver
    s = flow(14, 11, 10)
    getattr(s, field)[9, 8, 8] = np.copysign(np.nan, sign)
    prm = Params(14, 11, 10, tau=1e-3, emf=emf, precision=precision)
    with MHDSolver(prm, s) as g:
        fg, eg = g.debug_fluxes(), g.debug_emf()
    o = OracleSolver(Params(14, 11, 10, tau=1e-3, emf=emf), s)
    fo, eo = o.fluxes(), o.emf()
    tol = 1e-13 if precision == FP64 else 1e-5
    for d in range(3):
        for q in range(8):
            assert same(fg[d][q], fo[d][q], tol), ("flux", d, q)
        got, ref = eg[d], eo[d]
        if emf == EMF_LFM and field[0] == "v":
            bad = np.isnan(got)
            assert bad.sum() == (4 if "xyz".index(field[1]) == d else 8) and np.isnan(ref[bad]).all(), ("emf", d)
            got, ref = np.where(np.isnan(ref), 0.0, got), np.where(np.isnan(ref), 0.0, ref)
        assert same(got, ref, tol), ("emf", d)
