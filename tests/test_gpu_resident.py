"""The on-chip sweeps (k_resident.cu): the grid stays in registers and shared
memory for a batch of sweeps, CTAs exchanging their borders.  They must give
the segment kernel's bits (sweep variant 0) at every split of the grid: one
CTA row or plane, ragged last CTAs, odd heights and depths, rows that straddle
warps, widths that are not whole quads, one sweep (no exchange otherwise) and
batches back to back."""
import numpy as np
import pytest

from blaze_b200 import FluidSolver, SceneSettings, Timer
from blaze_b200._abi import BLZ_BC_FREE_SURFACE, BLZ_BC_REF_COMPAT

pytestmark = pytest.mark.gpu

ON_CHIP = 11


def run(dims, variant, bc, batches):
    W, H, D = dims
    rng = np.random.default_rng(W + 10 * H + 100 * D)
    scn = SceneSettings(gridRes=dims, dx=1.0 / W, domainBboxMax=(1.0, H / W, D / W), bc_mode=bc,
                        closedBounds=(1, 0, 1, 0, 0, 1), sweep_variant=variant)
    with FluidSolver(Timer(), scn) as s:
        s.set("RHS", rng.standard_normal((D, H, W)).astype(np.float32))
        s.set("P", rng.standard_normal((D, H, W)).astype(np.float32))
        for n in batches:
            s.sweeps(n)
        return s.get("P")


@pytest.mark.parametrize("dims", [(8, 4, 4), (8, 5, 7), (16, 4, 300), (8, 301, 6), (24, 21, 74), (40, 66, 59),
                                  (64, 64, 64), (120, 100, 84), (104, 40, 48), (200, 100, 60), (128, 128, 127),
                                  (256, 40, 40), (384, 20, 61), (4, 4, 4), (6, 9, 5), (26, 151, 57),
                                  (84, 64, 33), (90, 22, 36), (222, 82, 48)])
@pytest.mark.parametrize("bc", [BLZ_BC_FREE_SURFACE, BLZ_BC_REF_COMPAT])
def test_on_chip_sweeps_equal_segment_kernel(dims, bc):
    for batches in ((1,), (2,), (1, 3, 6)):
        np.testing.assert_array_equal(run(dims, ON_CHIP, bc, batches), run(dims, 0, bc, batches))


def test_on_chip_solve_counts_and_reports():
    """A residual-controlled solve as a device loop picks the on-chip sweeps for
    a grid that fits and takes the sweeps the segment kernel takes."""
    out = []
    for variant in (-1, 0):
        rng = np.random.default_rng(3)
        scn = SceneSettings(gridRes=(48, 40, 36), dx=1.0 / 48, bc_mode=BLZ_BC_FREE_SURFACE, tol=1e-3,
                            closedBounds=(1, 1, 1, 0, 1, 1), maxIterSolve=2000, check_every=20, sweep_variant=variant)
        with FluidSolver(Timer(), scn) as s:
            s.set("RHS", rng.standard_normal((36, 40, 48)).astype(np.float32))
            st = s.solve()
            out.append((st["iterations"], st["residual"], s.get("P")))
            if variant < 0:
                assert st["sweep_variant"] == ON_CHIP and st["device_loop"] == 1
    assert out[0][:2] == out[1][:2]
    np.testing.assert_array_equal(out[0][2], out[1][2])


BATCHES = {
    "one wave": [(16, 16, 16), (64, 96, 40), (48, 40, 31), (8, 4, 5)],
    "several waves": [(128, 64, 64), (96, 96, 96), (384, 20, 61), (64, 64, 64), (8, 301, 6), (128, 128, 128), (48, 47, 48)],
    "many small": [(8 + 8 * (i % 3), 5 + i, 4 + (7 * i) % 11) for i in range(19)],
}


@pytest.mark.parametrize("name", BATCHES)
@pytest.mark.parametrize("check_every", [1, 10])
def test_on_chip_batch_equals_single_solves(name, check_every, monkeypatch):
    """Grids swept side by side, in one or several launches, while some have
    already stopped: each grid's sweep count, residual and pressure are those
    of its own solve with the segment kernel, bit for bit."""
    from blaze_b200 import FluidSolver, Timer
    from blaze_b200.batch import Batch
    from blaze_b200.scenes import SceneSettings
    monkeypatch.setenv("BLZ_SWEEP_VARIANT", "11")
    runs = []
    for batched in (False, True):
        sims = []
        for i, d in enumerate(BATCHES[name]):
            rng = np.random.default_rng(70 + i)
            W, H, D = d
            sims.append(FluidSolver(Timer(), SceneSettings(
                gridRes=d, dx=1 / 64, closedBounds=(1, 1, 1, 0, 1, 1), bc_mode=BLZ_BC_FREE_SURFACE, sweep_variant=0,
                maxIterSolve=60, tol=(0.2, 0.02, 1e-3)[i % 3], check_every=check_every)))
            sims[-1].set("RHS", rng.standard_normal((D, H, W)).astype(np.float32))
        if batched:
            batch = Batch(sims)
            stats = [batch.solve(), batch.solve()]
            assert all(st["sweep_variant"] == 11 for st in stats[0])
            batch.close()
        else:
            stats = [[s.solve() for s in sims] for _ in range(2)]
        runs.append((stats, [s.get("P") for s in sims]))
        for s in sims:
            s.close()
    (sa, pa), (sb, pb) = runs
    for f in range(2):
        for i in range(len(pa)):
            assert sa[f][i]["iterations"] == sb[f][i]["iterations"], (f, i)
            assert sa[f][i]["residual"] == sb[f][i]["residual"], (f, i)
    for i in range(len(pa)):
        assert np.array_equal(pa[i], pb[i]), i
