"""Device memory of double-precision handles."""
import numpy as np
import pytest

from mhd3d_mpi_fortran_gb300 import MHDSolver, ics
from mhd3d_mpi_fortran_gb300.abi import FP32, FP64, STEP_AB2, STEP_RK3, Params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stepop", [STEP_AB2, STEP_RK3])
def test_a_double_handle_takes_twice_the_memory_of_a_single_one(stepop):
    """The arrays of a handle are those of its scheme, twice the bytes in FP64, before and after
    steps (allocations are rounded to 2 MB, and a captured step takes a little)."""
    import torch
    n = 96
    s = ics.empty_state(ics.grid(n, n, n))
    s.rho[...] = 1.0
    s.p[...] = 1.0
    take = {}
    for precision in (FP32, FP64):
        prm = Params(n, n, n, precision=precision, stepop=stepop, tau=1e-4)
        for _ in range(2):  # the first handle also loads the kernels
            torch.cuda.synchronize()
            free = torch.cuda.mem_get_info()[0]
            with MHDSolver(prm, s) as g:
                g.step(1)
                torch.cuda.synchronize()
                take[precision] = free - torch.cuda.mem_get_info()[0]
    assert np.isfinite(take[FP32]) and take[FP64] <= 2 * take[FP32] + (8 << 20)
