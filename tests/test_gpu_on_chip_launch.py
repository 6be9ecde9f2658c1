"""Launching the on-chip sweeps (k_resident.cu): several solvers at once, launches
that are refused, the tuner's table, errors that are reported and values that
are not finite.  Where the sweeps' result matters it is the segment kernel's
(sweep variant 0), bit for bit."""
import threading

import numpy as np
import pytest

from blaze_b200 import FluidSolver, SceneSettings, Timer
from blaze_b200._abi import BLZ_BC_FREE_SURFACE, BLZ_BC_REF_COMPAT

pytestmark = pytest.mark.gpu

ON_CHIP = 11


def make(dims, variant=ON_CHIP, bc=BLZ_BC_FREE_SURFACE, seed=0, **kw):
    """A solver of a random system."""
    W, H, D = dims
    s = FluidSolver(Timer(), SceneSettings(gridRes=dims, dx=1.0 / W, domainBboxMax=(1.0, H / W, D / W), bc_mode=bc,
                                           closedBounds=(1, 0, 1, 0, 0, 1), sweep_variant=variant, **kw))
    rng = np.random.default_rng(seed + W + 10 * H + 100 * D)
    s.set("RHS", rng.standard_normal((D, H, W)).astype(np.float32))
    s.set("P", rng.standard_normal((D, H, W)).astype(np.float32))
    return s


def in_threads(jobs):
    """Runs the callables side by side; returns their results or raises the first error."""
    out, err = [None] * len(jobs), []
    start = threading.Barrier(len(jobs))

    def call(i):
        try:
            start.wait()
            out[i] = jobs[i]()
        except Exception as e:               # noqa: BLE001 (handed to the caller)
            err.append(e)

    ts = [threading.Thread(target=call, args=(i,)) for i in range(len(jobs))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    if err:
        raise err[0]
    return out


def test_two_threads_sweep_grids_of_different_sizes():
    """Grids that share a kernel but need different amounts of shared memory,
    swept from two threads: every launch is taken, and the pressures are those
    of each grid alone."""
    dims, calls = [(96, 96, 96), (120, 100, 84)], 4000

    def sweeps(d):
        def job():
            with make(d) as s:
                for _ in range(calls):
                    s.sweeps(1)
                return s.get("P")
        return job

    got = in_threads([sweeps(d) for d in dims])
    for d, p in zip(dims, got):
        with make(d, variant=0) as s:
            s.sweeps(calls)
            np.testing.assert_array_equal(p, s.get("P"))
