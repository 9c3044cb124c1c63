"""The PDM limiter without its signs (pdm_states, within and corner_quad of the kernels).

CPU: the soft threshold (FP32 kernels) bit for bit and the nested intervals
(FP64 face fluxes) to rounding against the reference's sign form (PDM2,
mhd3d3.f90:1069-1172) for positive pdmb, ties, jumps and values across the
exponent range included.  GPU: fluxes and EMFs for limiter constants on both
sides of the rule (pdmb > 0 takes these forms, anything else the reference's)
against the oracle, in every launch shape that reads the limiter.
"""
import numpy as np
import pytest

from mhd3d_mpi_fortran_gb300.abi import FP32, FP64, BC_OUTFLOW, BC_EVEN, Params


def within(c, far, out, x):
    lo = np.maximum(np.minimum(c, far), np.minimum(c, out))
    return np.maximum(lo, np.minimum(np.minimum(np.maximum(c, far), np.maximum(c, out)), x))


def reference(fm2, fm1, f0, fp1, fi, pdmb):
    sg = lambda v: np.where(v >= 0, 1.0, -1.0)
    fii = np.maximum(np.minimum(fm1, f0), np.minimum(fi, np.maximum(fm1, f0)))
    dm, d0, dp = pdmb * (fm1 - fm2), pdmb * (f0 - fm1), pdmb * (fp1 - f0)
    qm, qp = np.abs(sg(dm) + sg(d0)), np.abs(sg(d0) + sg(dp))
    left = fii - sg(d0) * np.maximum(0.0, np.abs(fii - fm1) - qm * np.abs(dm))
    right = fii + sg(d0) * np.maximum(0.0, np.abs(f0 - fii) - qp * np.abs(dp))
    return left, right


def threshold(near, x, D):
    """shrink() and its use: the excess of x - near over D, with the kernels' operations."""
    d = x - near
    m = np.minimum(np.abs(d), np.abs(D)) * np.where(np.signbit(d) == np.signbit(D), 1, -1).astype(d.dtype)
    return x - (d - np.copysign(np.maximum(m, 0), d))


def cells(kind):
    rng = np.random.default_rng(3)
    n = 20000
    f = rng.standard_normal((5, n))
    if kind == "ties":  # equal neighbours, zero and signed-zero slopes
        f = rng.integers(-2, 3, size=(5, n)).astype(float) * rng.choice([1.0, -0.0, 0.0], size=(5, n))
    if kind == "wide":
        f *= 10.0 ** rng.uniform(-15, 15, size=(1, n))
    return f


@pytest.mark.parametrize("pdmb", [0.25, 0.3, 4.0])
@pytest.mark.parametrize("kind", ["random", "ties", "wide"])
def test_threshold_has_the_reference_bits_in_fp32(kind, pdmb):
    f = cells(kind).astype(np.float32)
    p = np.float32(pdmb)
    sg = lambda v: np.where(v >= 0, np.float32(1), np.float32(-1))
    x = np.maximum(np.minimum(f[1], f[2]), np.minimum(f[4], np.maximum(f[1], f[2])))
    dm, d0, dp = p * (f[1] - f[0]), p * (f[2] - f[1]), p * (f[3] - f[2])
    zero = np.float32(0)
    l = x - sg(d0) * np.maximum(zero, np.abs(x - f[1]) - np.abs(sg(dm) + sg(d0)) * np.abs(dm))
    r = x + sg(d0) * np.maximum(zero, np.abs(f[2] - x) - np.abs(sg(d0) + sg(dp)) * np.abs(dp))
    k = p + p
    assert np.array_equal(threshold(f[1], x, k * (f[1] - f[0])), l)
    assert np.array_equal(threshold(f[2], x, k * (f[2] - f[3])), r)


@pytest.mark.parametrize("pdmb", [1e-6, 0.25, 1.0, 4.0, 1e6])
@pytest.mark.parametrize("kind", ["random", "ties", "wide"])
def test_interval_form_is_the_reference_limiter(kind, pdmb):
    f = cells(kind)
    l, r = reference(*f, pdmb)
    a, b = within(f[1], f[2], f[1] + 2 * pdmb * (f[1] - f[0]), f[4]), within(f[2], f[1], f[2] + 2 * pdmb * (f[2] - f[3]), f[4])
    # a few roundings of the largest term: the cells and the slopes times 2 pdmb
    tol = 8 * np.finfo(float).eps * np.abs(f).max(axis=0) * max(1.0, 2 * pdmb)
    assert np.all(np.abs(a - l) <= tol) and np.all(np.abs(b - r) <= tol)


def _state():
    from tests.test_gpu_parity import rand_state
    return rand_state(33, 9, 10, seed=5)


@pytest.mark.gpu
@pytest.mark.parametrize("pdmb", [4.0, 0.3, 0.0, -1.0])
def test_limiter_constant_fp64_matches_oracle(pdmb):
    from mhd3d_mpi_fortran_gb300 import MHDSolver
    from oracle.oracle import OracleSolver
    s = _state()
    prm = Params(33, 9, 10, pdmb=pdmb, bc=(0, BC_EVEN, BC_OUTFLOW), tau=1e-4)
    with MHDSolver(prm, s) as g:
        fg, eg = g.debug_fluxes(), g.debug_emf()
        g.step(2)
        sg = g.fetch()
    o = OracleSolver(prm, s)
    fo, eo = o.fluxes(), o.emf()
    o.step(2)
    so = o.fetch()
    for d in range(3):
        for q in range(8):
            assert np.abs(fg[d][q] - fo[d][q]).max() <= 1e-13 * np.abs(fo[d][q]).max()
        assert np.abs(eg[d] - eo[d]).max() <= 1e-13 * np.abs(eo[d]).max()
    for k in so:
        assert np.abs(sg[k] - so[k]).max() <= 1e-11 * np.abs(so[k]).max(), k


@pytest.mark.gpu
@pytest.mark.parametrize("pdmb", [4.0, 0.3, 0.0, -1.0])
@pytest.mark.parametrize("tiles", [(32, 1), (32, 8), (8, 4), (4, 8), (16, 1)])
def test_limiter_constant_fp32_shapes_agree(pdmb, tiles):
    from mhd3d_mpi_fortran_gb300 import MHDSolver, ensemble_step
    s = _state()
    prm = Params(33, 9, 10, pdmb=pdmb, precision=FP32, tau=1e-4)
    with MHDSolver(prm, s) as g, MHDSolver(prm, s) as h, MHDSolver(prm, s) as e:
        g.set_tiles(*tiles)
        g.step(2)
        h.step(2)
        e.set_tiles(*tiles)
        ensemble_step([e], 2)
        a, b, c = g.fetch(), h.fetch(), e.fetch()
    for k in a:
        assert np.array_equal(a[k], b[k]) and np.array_equal(a[k], c[k]), k
