"""Stages whose kernels differ with the size of the grid, at sizes where the large
grids' kernels run and no axis is a multiple of their tiles, against the FP64
oracle.

Tolerance of the advection: the stage's (test_gpu_parity.py, sizes to 24) times 8.
Its error is that of a position in cells, whose rounding is half an ulp of the
position: an ulp at 133 cells is 8 times one at 24.  The gradient works cell by
cell and keeps the stage's."""
import numpy as np
import pytest

from blaze_b200 import BLZ_BC_FREE_SURFACE, BLZ_BC_REF_COMPAT
from test_gpu_parity import STAGE_ABS, STAGE_REL, assert_close, pair, scene

pytestmark = pytest.mark.gpu


def flow(kind, gpu, ref, seed):
    """Adds a flow, in cells a step, to the random velocities."""
    p = ref.p
    rng = np.random.default_rng(seed)
    k, j, i = (np.arange(n, dtype=np.float64) for n in (p.depth, p.height, p.width))
    cells = p.dx / p.dt
    if kind == "still":
        return
    for f in ("U", "V", "W"):
        a = getattr(ref, f)
        D, H, W = a.shape
        z, y, x = (np.arange(n) / n for n in a.shape)
        if kind == "uniform":                    # 25 cells a step: traces follow the shifted tile, and leave the domain
            a += cells * {"U": 25.0, "V": -13.0, "W": 7.0}[f]
        elif kind == "shear":                    # across a tile the displacement changes by more than its margin of 4
            a += cells * 120.0 * {"U": y[None, :, None] - 0.5, "V": z[:, None, None] - 0.5,
                                  "W": x[None, None, :] - 0.5}[f] * np.ones(a.shape)
        a[...] = a.astype(np.float32)
        gpu.set(f, a.astype(np.float32))


@pytest.mark.parametrize("scheme,kind,dens", [(0, "still", 0), (0, "uniform", 1), (0, "shear", 0), (1, "uniform", 0),
                                              (1, "shear", 1), (2, "uniform", 0), (2, "shear", 1)],
                         ids=lambda v: str(v))
def test_advect_large(scheme, kind, dens):
    """1445 tiles of 32 x 8 x 8 nodes with a remainder on every axis."""
    gpu, ref = pair(scene(dims=(130, 131, 133), advect_scheme=scheme, density_field=dens, buoyancy_alpha=0.05), 181)
    if dens:
        x = np.random.default_rng(182).uniform(0.0, 1.0, ref.DENSITY.shape).astype(np.float32)
        ref.DENSITY[...] = x
        gpu.set("DENSITY", x)
    flow(kind, gpu, ref, 183)
    gpu.advect()
    ref.advect()
    assert_close(gpu, ref, ("T", "U", "V", "W") + (("DENSITY",) if dens else ()), rel=8 * STAGE_REL, absol=8 * STAGE_ABS)
    gpu.close()


@pytest.mark.parametrize("dims", [(136, 131, 133), (66, 301, 300)])        # 2 and 8 planes per thread
@pytest.mark.parametrize("bc", [BLZ_BC_REF_COMPAT, BLZ_BC_FREE_SURFACE])
@pytest.mark.parametrize("bounds", [(1, 1, 1, 1, 1, 1), (1, 0, 1, 0, 1, 1), (0, 0, 0, 0, 0, 0)])
def test_gradient_of_several_planes(dims, bc, bounds):
    """Copied faces of the wall mode's open sides, ghosts of the free surface's."""
    gpu, ref = pair(scene(dims=dims, closedBounds=bounds, bc_mode=bc), 191, fields=("U", "V", "W", "P"))
    gpu.gradient()
    ref.gradient()
    assert_close(gpu, ref, ("U", "V", "W"))
    gpu.close()


@pytest.mark.parametrize("dims", [(136, 131, 133), (66, 301, 300)])
@pytest.mark.parametrize("bc", [BLZ_BC_REF_COMPAT, BLZ_BC_FREE_SURFACE])
def test_defect_gradient_of_several_planes(dims, bc):
    """The gradient of p + delta after a few sweeps of the correction: the oracle's
    of its own swept pressure, within the sweeps' tolerance (2e-5, 2e-4)."""
    gpu, ref = pair(scene(dims=dims, closedBounds=(1, 0, 0, 1, 1, 0), bc_mode=bc, defect_correction=1, maxIterSolve=8,
                          tol=0.0), 193)
    gpu.solve()
    gpu.gradient()
    ref.gs_sweeps(8)
    ref.gradient()
    assert_close(gpu, ref, ("P", "U", "V", "W"), rel=2e-5, absol=2e-4)
    gpu.close()


@pytest.mark.parametrize("dens", [0, 1])
def test_source_of_scattered_particles(dens):
    """A few particles in each of many bins: the kernel with one block per bin for all
    fields.  Particles on the domain's sides and outside, radii of up to 2.5 cells,
    several in some bins; the splat test's tolerance (test_gpu_parity.py)."""
    from blaze_b200 import FluidSolver, Timer
    from oracle import oracle
    scn = scene(dims=(82, 67, 91), density_field=dens, buoyancy_alpha=0.05)
    p = scn.to_params()
    rng = np.random.default_rng(31)
    rec = np.zeros((1500, 8), np.float32)
    rec[:, :3] = rng.uniform(np.array(scn.domainBboxMin) - 0.05, np.array(scn.domainBboxMax) + 0.05, (1500, 3))
    rec[:, 3:6] = rng.uniform(-1.0, 1.0, (1500, 3))
    rec[:, 6] = rng.uniform(0.0, 5.0, 1500) * p.dx
    rec[:, 7] = rng.uniform(-0.5, 2.0, 1500)
    rec[::9, 4] = 0.0                                     # a field skipped
    d = rng.uniform(0.0, 1.0, 1500).astype(np.float32) if dens else None
    with FluidSolver(Timer(), scn) as gpu:
        ref = oracle.State(p, np.float64)
        gpu.setParticles(rec, d)
        gpu.addSource()
        ref.add_source(rec, density=d)
        assert_close(gpu, ref, ("T", "U", "V", "W") + (("DENSITY",) if dens else ()), rel=1e-5, absol=1e-4)
