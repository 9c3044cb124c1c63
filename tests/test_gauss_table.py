"""The FP64 Gaussian moments' Taylor table (gauss_table) against scipy and, on the GPU, the moments through the fluxes."""
import numpy as np
import pytest
from scipy.special import erfc


def rows():
    """gauss_table's recurrence (csrc/mhd_api.cu) in FP64."""
    out = np.zeros((209, 16))
    for i in range(209):
        c = i / 32.0
        a = [np.exp(-c * c) / (2.0 * np.sqrt(np.pi))]
        prev = 0.0
        for n in range(7):
            a.append(-2.0 * (c * a[n] + prev) / (n + 1))
            prev = a[n]
        out[i, 0] = 0.5 * erfc(c)
        out[i, 1:8] = [-2.0 * a[n] / (n + 1) for n in range(7)]
        out[i, 8:] = a
    return out


def test_taylor_rows_reach_double_precision():
    t = rows()
    z = np.concatenate([np.linspace(0.0, 6.5, 200001)[:-1], (np.arange(208) + 0.5) / 32.0])  # row edges included
    i = np.rint(z * 32).astype(int)
    d = z - i / 32.0
    h = np.polynomial.polynomial.polyval(d, t[i, :8].T, tensor=False)
    e = np.polynomial.polynomial.polyval(d, t[i, 8:].T, tensor=False)
    # first omitted terms (4e-17 and 4e-17) plus the roundings of a value below 0.5
    assert np.abs(h - 0.5 * erfc(z)).max() <= 2.5e-16
    assert np.abs(e - np.exp(-z * z) / (2 * np.sqrt(np.pi))).max() <= 2.5e-16


@pytest.mark.gpu
@pytest.mark.parametrize("mach", [0.0, 0.3, 3.0, 30.0])  # |z| around 0, inside the table, across its end, beyond it
def test_fluxes_across_the_table_match_oracle(mach):
    from mhd3d_mpi_fortran_gb300 import MHDSolver
    from mhd3d_mpi_fortran_gb300.abi import Params
    from oracle.oracle import OracleSolver
    from tests.test_gpu_parity import rand_state
    s = rand_state(17, 8, 9, seed=11)
    rng = np.random.default_rng(2)
    for v in (s.vx, s.vy, s.vz):
        v[...] = mach * rng.standard_normal(v.shape)
    prm = Params(17, 8, 9, tau=1e-5)
    with MHDSolver(prm, s) as g:
        fg = g.debug_fluxes()
    fo = OracleSolver(prm, s).fluxes()
    for d in range(3):
        for q in range(8):
            assert np.abs(fg[d][q] - fo[d][q]).max() <= 1e-13 * np.abs(fo[d][q]).max(), (d, q)
