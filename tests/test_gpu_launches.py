"""Which kernels and runtime calls an entry point makes (CUPTI, through torch's profiler).

The traced program is this file run as a child process that leaves by os._exit: the profiler's
libraries corrupt the heap when a process that has used them ends the usual way.
"""
import collections
import json
import os
import re
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

ROOT = str(Path(__file__).resolve().parent.parent)
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

from mhd3d_mpi_fortran_gb300 import MHDSolver, ensemble_step, ics  # noqa: E402
from mhd3d_mpi_fortran_gb300.abi import FP32, FP64, Params  # noqa: E402

pytestmark = pytest.mark.gpu


def child(*args):
    """What `PROGRAMS[args[0]](*args[1:])` returns in a process of its own."""
    r = subprocess.run([sys.executable, __file__, json.dumps(args)], capture_output=True, text=True, timeout=240, cwd=ROOT)
    assert r.returncode == 0, r.stderr[-2000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


def traced(fn):
    """(kernel base names with their launches, runtime calls) of fn()."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    for f in (lambda: torch.zeros(1, device="cuda"), fn):  # the first trace of a process may come back empty
        with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
            f()
            torch.cuda.synchronize()
    kernels, calls = collections.Counter(), collections.Counter()
    for e in p.events():
        if e.device_type.name == "CUDA":
            m = re.search(r"(k_\w+)", e.name)
            if m:
                kernels[m.group(1)] += 1
        else:
            calls[e.name] += 1
    return dict(kernels), dict(calls)


def state(n, seed=3):
    s = ics.empty_state(ics.grid(*n))
    r = np.random.default_rng(seed)
    s.rho[...] = 1.0
    s.p[...] = 1.0
    for v in (s.vx, s.vy, s.vz, s.bi, s.bj, s.bk):
        v[...] = 0.1 * r.standard_normal(v.shape)
    return s


def limited(precision, n, pdmb):
    """A grid alone, a batch of two and (FP32) the smaller tiles."""
    prm = Params(*n, precision=precision, pdmb=pdmb, tau=1e-5)
    gs = [MHDSolver(prm, state(n)) for _ in range(3)]
    gs[2].step(1)
    ensemble_step(gs[:2], 1)
    out = [traced(lambda: gs[2].time_steps(2))[0], traced(lambda: ensemble_step(gs[:2], 2))[0]]
    if precision == FP32:
        gs[2].set_tiles(4, 4)
        out.append(traced(lambda: gs[2].time_steps(2))[0])
    return out


@pytest.mark.parametrize("precision,n", [(FP32, (24, 16, 12)), (FP32, (96, 96, 64)), (FP64, (24, 16, 12))])
def test_every_limiter_constant_takes_the_same_kernels(precision, n):
    """Sweeps, streams, tiles and batched launches do not depend on pdmb's sign."""
    some = child("limited", precision, n, 0.3)
    assert all(some)
    for pdmb in (0.0, -1.0):
        assert child("limited", precision, n, pdmb) == some, pdmb


def timed(precision):
    """Two timings of three steps without a graph, the second after more steps."""
    with MHDSolver(Params(24, 16, 12, precision=precision, tau=1e-4), state((24, 16, 12))) as g:
        g.time_steps(2)
        one = traced(lambda: g.time_steps(3))
        g.step(9)
        return one, traced(lambda: g.time_steps(3))


@pytest.mark.parametrize("precision", [FP32, FP64])
def test_time_steps_without_a_graph_launches_the_kernels(precision):
    """Steps timed without a graph are launched one by one, however many the handle has run."""
    one, many = child("timed", precision)
    assert sum(one[0].values()) > 0 and one[0] == many[0]
    for k in ("cudaGraphLaunch", "cudaGraphInstantiate", "cudaStreamBeginCapture"):
        assert not any(c.startswith(k) for c in many[1]), k


PROGRAMS = {f.__name__: f for f in (limited, timed)}

if __name__ == "__main__":
    name, *args = json.loads(sys.argv[1])
    print(json.dumps(PROGRAMS[name](*args)), flush=True)
    os._exit(0)
