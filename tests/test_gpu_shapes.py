"""Launch shapes that follow the grid: segments and flattened columns of the
FP32 column sweeps, and the batched step with its dt folded into the last stage."""
import ctypes

import numpy as np
import pytest

from mhd3d_mpi_fortran_gb300 import MHDSolver, ensemble_step, ics
from mhd3d_mpi_fortran_gb300.abi import DT_CFL, FP32, FP64, STEP_RK2, STEP_RK3, Params

pytestmark = pytest.mark.gpu
FIELDS = ("rho", "vx", "vy", "vz", "p", "bx", "by", "bz", "bi", "bj", "bk")


def state(nx, ny, nz, nord, seed):
    """Smooth waves with seeded noise and a random face field."""
    g = ics.grid(nx, ny, nz, nord=nord)
    s = ics.empty_state(g)
    r = np.random.default_rng(seed)
    x, y, z = [c.reshape(sh) for c, sh in zip(g.centres(), ((-1, 1, 1), (1, -1, 1), (1, 1, -1)))]
    s.rho[...] = 1.0 + 0.3 * np.sin(2 * np.pi * (x + y)) + 0.0 * z
    s.p[...] = 1.0 + 0.2 * np.cos(2 * np.pi * (y + z)) + 0.0 * x
    for v in (s.vx, s.vy, s.vz, s.bi, s.bj, s.bk):
        v[...] = 0.2 * r.standard_normal(v.shape)
    return s


@pytest.mark.parametrize("recon,nord", [(1, 8), (3, 6), (5, 4)])
@pytest.mark.parametrize("shape", [(9, 37, 10), (31, 5, 66), (33, 34, 4), (40, 65, 9), (65, 16, 21)])
def test_sweeps_equal_face_tiles(shape, recon, nord):
    """Columns flattened over (x, remaining axis) with rows that end inside a
    warp, and segments from 4 cells to a ragged last one: the bits of the face tiles."""
    s = state(*shape, nord, sum(shape))
    prm = Params(*shape, nord=nord, reconop=recon, stepop=STEP_RK3, precision=FP32, tau=2e-4)
    out = {}
    for td in (8, 32):
        with MHDSolver(prm, s) as g:
            g.set_tiles(td, 8)
            g.step(2)
            out[td] = g.fetch()
    for k in FIELDS:
        assert np.array_equal(out[8][k], out[32][k]), k


@pytest.mark.parametrize("precision,stepop", [(FP32, STEP_RK2), (FP32, STEP_RK3), (FP64, STEP_RK2)])
def test_batched_steps_fold_dt_as_single_steps(precision, stepop):
    """CFL-driven batches, in calls of 1, 2 and 1 steps with single steps of one
    grid between them (prepared and unprepared starts), against each grid alone."""
    shapes = [(16, 24, 9), (40, 16, 16), (33, 12, 20), (24, 24, 24)]
    ss = [state(*n, 8, 3 + m) for m, n in enumerate(shapes)]
    ps = [Params(*n, precision=precision, stepop=stepop, dt_mode=DT_CFL, tau=1e-4) for n in shapes]
    batch = [MHDSolver(p, s) for p, s in zip(ps, ss)]
    alone = [MHDSolver(p, s) for p, s in zip(ps, ss)]
    for n in (1, 2, 1):
        ensemble_step(batch, n)
        for g in alone:
            g.step(n)
        assert batch[1].step(1) == alone[1].step(1)  # (tau, status)
    for a, b in zip(batch, alone):
        fa, fb = a.fetch(), b.fetch()
        for k in FIELDS:
            assert np.array_equal(fa[k], fb[k]), k
        a.close()
        b.close()


@pytest.mark.parametrize("precision", [FP32, FP64])
@pytest.mark.parametrize("shape", [(16, 16, 5), (33, 9, 260), (70, 50, 35), (96, 96, 63)])
def test_cells_up_z_leave_consistent_faces(shape, precision):
    """CT passes of 1 to 8 cells a thread, with a ragged last walk: the cell B they
    leave is the mean of the stored faces bit for bit (a face computed as one
    cell's high side and the next one's low side is the same value)."""
    s = state(*shape, 8, 7)
    with MHDSolver(Params(*shape, stepop=STEP_RK3, precision=precision, tau=1e-4), s) as g:
        g.step(2)
        f = g.fetch()
    t = np.float32 if precision == FP32 else np.float64
    f = {k: v.astype(t) for k, v in f.items()}
    half = t(0.5)
    assert np.array_equal(f["bx"], half * (f["bi"][1:] + f["bi"][:-1]))
    assert np.array_equal(f["by"], half * (f["bj"][:, 1:] + f["bj"][:, :-1]))
    assert np.array_equal(f["bz"], half * (f["bk"][:, :, 1:] + f["bk"][:, :, :-1]))


@pytest.mark.parametrize("shape,nord,precision", [((8, 8, 8), 8, FP64), ((16, 16, 16), 8, FP32), ((40, 70, 31), 8, FP32),
                                                  ((56, 120, 64), 4, FP32), ((40, 21, 33), 6, FP64)])
def test_fetch_paths_agree(shape, nord, precision):
    """Frames by way of the staging buffer (small grids), straight into fresh pageable
    arrays, into pinned arrays, and a part of the fields only: the values mhd_init got."""
    import torch
    s = state(*shape, nord, 11)
    f = np.float32 if precision == FP32 else np.float64
    with MHDSolver(Params(*shape, nord=nord, reconop={8: 1, 6: 3, 4: 5}[nord], precision=precision, tau=1e-4), s) as g:
        got = g.fetch()
        pin = g.output_arrays()
        pin = {k: torch.empty(a.size, dtype=torch.float64, pin_memory=True).numpy().reshape(a.shape, order="F")
               for k, a in pin.items()}
        g.fetch(out=pin)
        some = [None] * 11
        part = {k: np.zeros_like(got[k]) for k in ("p", "bi", "bk")}
        for k, a in part.items():
            some[FIELDS.index(k)] = a.ctypes.data
        assert g.lib.mhd_fetch(g.h, *[None if q is None else ctypes.cast(q, ctypes.POINTER(ctypes.c_double))
                                      for q in some]) == 0
    c = slice(nord // 2, -(nord // 2))
    for k in ("rho", "vx", "vy", "vz", "p"):
        assert np.array_equal(got[k][c, c, c], getattr(s, k).astype(f)[c, c, c]), k
    for k in FIELDS:
        assert np.array_equal(got[k], pin[k]), k
    for k, a in part.items():
        assert np.array_equal(a, got[k]), k


@pytest.mark.parametrize("precision,stepop,dt_mode", [(FP32, 1, 0), (FP32, STEP_RK2, DT_CFL), (FP32, STEP_RK3, 0),
                                                      (FP64, STEP_RK3, DT_CFL), (FP64, 1, 0)])
def test_replayed_steps_equal_launched_ones(precision, stepop, dt_mode):
    """A handle's later steps replay a captured step: 13 steps in calls of 1, 9
    and 3 (with a tile change between, which drops the captures in FP32) against
    a handle that runs them as one graph, bit for bit."""
    shape = (24, 18, 21)
    s = state(*shape, 8, 5)
    prm = Params(*shape, precision=precision, stepop=stepop, dt_mode=dt_mode, tau=1e-4)
    with MHDSolver(prm, s) as g, MHDSolver(prm, s) as h:
        tg = g.step(1)
        tg = g.step(9)
        if precision == FP32:
            g.set_tiles(8, 8)
        tg = g.step(3)
        th = h.step(13, graph=True)  # one capture of all 13
        fg, fh = g.fetch(), h.fetch()
    assert tg == th
    for k in FIELDS:
        assert np.array_equal(fg[k], fh[k]), k
