"""The on-chip sweeps (k_resident.cu): the grid stays in registers and shared
memory for a batch of sweeps, CTAs exchanging their borders.  They must give
the segment kernel's bits (sweep variant 0) at every split of the grid: one
CTA row or plane, ragged last CTAs, odd heights and depths, rows that straddle
warps, widths that are not whole quads, one sweep (no exchange otherwise) and batches back to back."""
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
