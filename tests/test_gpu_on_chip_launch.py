"""Launching the on-chip sweeps (k_resident.cu): several solvers at once, launches
that are refused, the tuner's table, errors that are reported and values that
are not finite.  Where the sweeps' result matters it is the segment kernel's
(sweep variant 0), bit for bit."""
import ctypes as C
import os
import subprocess
import sys
import threading

import numpy as np
import pytest
import torch
from cuda.bindings import runtime as cudart

from blaze_b200 import FluidSolver, SceneSettings, Timer, _abi, _lib
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


class Geom(C.Structure):
    _fields_ = [("W", C.c_int), ("H", C.c_int), ("D", C.c_int), ("dx", C.c_float), ("dt", C.c_float),
                ("inv_dx", C.c_float), ("dmin", C.c_float * 3), ("dsize", C.c_float * 3)]


class SolveParams(C.Structure):
    _fields_ = [("scale", C.c_float), ("scale_d", C.c_double), ("open", C.c_bool * 6), ("dirichlet", C.c_int)]


class ResidentWork(C.Structure):
    _fields_ = [("work", C.c_void_p), ("err", C.c_void_p)]


def internal(name, restype, argtypes):
    """A function of the library's own (C++ linkage) by its plain name."""
    out = subprocess.run(["nm", "-D", "--defined-only", _lib.load()._name], capture_output=True, text=True, check=True).stdout
    sym = [w[2] for w in map(str.split, out.splitlines()) if f"blz{len(name)}{name}E" in w[2]]
    assert len(sym) == 1, sym
    f = getattr(_lib.load(), sym[0])
    f.restype, f.argtypes = restype, argtypes
    return f


class System:
    """Device arrays of a small random system and the arguments that describe it."""

    def __init__(self, dims):
        W, H, D = dims
        self.g = Geom(W, H, D, 1.0 / W, 1.0 / 24, W, (C.c_float * 3)(), (C.c_float * 3)(1.0, H / W, D / W))
        self.sp = SolveParams(0.01, 0.01, (C.c_bool * 6)(0, 1, 0, 1, 1, 0), 1)
        gen = torch.Generator(device="cuda").manual_seed(W + H + D)
        self.rhs = [torch.randn(W // 2 * H * D, device="cuda", generator=gen) for _ in range(2)]
        self.p = [torch.randn(W // 2 * H * D, device="cuda", generator=gen) for _ in range(2)]
        self.bytes = internal("resident_bytes", C.c_size_t, [C.POINTER(Geom)])(C.byref(self.g))
        self.work = torch.zeros(self.bytes // 4, dtype=torch.int32, device="cuda")
        self.err = torch.zeros(1, dtype=torch.int32).pin_memory()

    def arrays(self):
        return [C.c_void_p(t.data_ptr()) for t in self.rhs + self.p]


def test_refused_launch_is_an_error_of_the_solve_graph():
    """A launch of the sweeps that is refused while the solve graph is built
    (here for want of an error flag) is an error: a graph without sweeps
    would be kept, and every later solve would only check the residual."""
    y = System((16, 16, 16))
    build = internal("build_solve_graph", C.c_int, [C.POINTER(Geom), C.POINTER(SolveParams)] + [C.c_void_p] * 5 +
                     [C.c_int, C.c_void_p, C.c_void_p, C.c_int, C.c_int, C.c_double, C.c_int] + [C.c_void_p] * 7 +
                     [C.POINTER(ResidentWork)])
    partials = torch.zeros(8192, dtype=torch.float64, device="cuda")
    norm2 = torch.zeros(2, dtype=torch.float64, device="cuda")
    ctl = torch.zeros(64, dtype=torch.int64, device="cuda")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    for err, taken in ((None, False), (y.err.data_ptr(), True)):
        graph, n = C.c_void_p(), [C.c_int(), C.c_int()]
        e = build(C.byref(y.g), C.byref(y.sp), *y.arrays(), partials.data_ptr(), 4096, norm2.data_ptr(), ctl.data_ptr(),
                  10, 20, 1e-3, ON_CHIP, stream.cuda_stream, C.byref(graph), C.byref(n[0]), C.byref(n[1]), None, None,
                  None, C.byref(ResidentWork(y.work.data_ptr(), err)))
        assert (e == 0) == taken and bool(graph.value) == taken, (err, e)


@pytest.mark.parametrize("dims,order", [((392, 16, 16), (0, 1)), ((400, 16, 16), (1, 0))])
def test_tuner_keeps_solvers_with_other_choices_apart(dims, order, monkeypatch):
    """Where the two-sweep passes do not apply (W > 384), a solver that may use
    the on-chip sweeps and one that may not (temporal_block) are offered the
    same number of launch shapes; each tunes its own choice."""
    monkeypatch.setenv("BLZ_TUNE_CACHE", "off")
    monkeypatch.delenv("BLZ_SWEEP_VARIANT", raising=False)
    for tb in order:
        with make(dims, variant=-1, temporal_block=tb, maxIterSolve=20) as s:
            st = s.solve()
            assert st["sweep_variant"] in ((0, 4, ON_CHIP) if tb == 0 else range(6)), (tb, st)
            assert s.kernel_launches() > 100, (tb, s.kernel_launches())      # 44 at most without tuning


def test_only_solvers_that_sweep_on_chip_hold_exchange_buffers():
    """A solver whose sweeps are forced to another kernel takes no more memory
    than one that may not use the on-chip sweeps (their buffers: 13 MB at
    128^3)."""
    def held(**kw):
        with make((128, 128, 128), **kw) as s:
            s.sweeps(1)
            torch.cuda.synchronize()
            return torch.cuda.mem_get_info()[0]

    held(variant=0)                                       # the allocator's first blocks
    without, forced = held(variant=0, temporal_block=1), held(variant=0)
    assert without - forced < 4 << 20, (without, forced)


@pytest.mark.parametrize("dims,variant", [((26, 30, 22), -1), ((32, 30, 22), ON_CHIP)])
def test_first_sweeps_of_a_solver_may_be_captured(dims, variant):
    """The first call that sweeps on chip, inside a capture of the caller's
    stream: taken, and each replay runs the sweeps."""
    with make(dims, variant=variant) as s, make(dims, variant=0) as ref:
        stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        _lib.check(_lib.load().blz_set_stream(s._h, C.c_void_p(stream.cuda_stream)), s._h)
        with torch.cuda.graph(graph, stream=stream):
            s.sweeps(3)
        for _ in range(2):
            graph.replay()
        torch.cuda.synchronize()
        ref.sweeps(6)
        np.testing.assert_array_equal(s.get("P"), ref.get("P"))
        _lib.check(_lib.load().blz_set_stream(s._h, None), s._h)


_FEW_SMS = r"""
import sys
sys.path[:0] = sys.argv[1:3]
import numpy as np
from cuda.bindings import driver as cu
import test_gpu_on_chip_launch as t
from blaze_b200.batch import Batch

def ok(r):
    assert r[0] == cu.CUresult.CUDA_SUCCESS, r[0]
    return r[1] if len(r) == 2 else r[1:]

ok(cu.cuInit(0))
dev = ok(cu.cuDeviceGet(0))
sms = ok(cu.cuDeviceGetDevResource(dev, cu.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
part = ok(cu.cuDevSmResourceSplitByCount(1, sms, 0, 16))[0]
green = ok(cu.cuGreenCtxCreate(ok(cu.cuDevResourceGenerateDesc(part, 1)), dev,
                               cu.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))

# a solver of the whole device, whose stream is then one of the context with few SMs
with t.make((64, 64, 64)) as s, t.make((64, 64, 64), variant=0) as ref:
    s.sweeps(3)
    stream = ok(cu.cuGreenCtxStreamCreate(green, cu.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    t._lib.check(t._lib.load().blz_set_stream(s._h, int(stream)), s._h)
    s.sweeps(3)
    ref.sweeps(6)
    np.testing.assert_array_equal(s.get("P"), ref.get("P"))
    t._lib.check(t._lib.load().blz_set_stream(s._h, None), s._h)

cu.cuCtxSetCurrent(ok(cu.cuCtxFromGreenCtx(green)))

def solve(dims, variant):
    with t.make(dims, variant=variant, maxIterSolve=20) as s:
        st = s.solve()
        return st["sweep_variant"], s.get("P")

for dims, variant in (((64, 64, 64), -1), ((26, 151, 57), -1), ((64, 64, 64), t.ON_CHIP)):
    v, p = solve(dims, variant)
    assert v != t.ON_CHIP, (dims, variant)
    np.testing.assert_array_equal(p, solve(dims, 0)[1])
dims = [(64, 64, 64), (48, 40, 36)]
sims = [t.make(d, variant=0, maxIterSolve=20, tol=1e-9, check_every=10) for d in dims]
b = Batch(sims)
b.solve()                                                # small grids may still fit the SMs there are
for d, s in zip(dims, sims):
    np.testing.assert_array_equal(s.get("P"), solve(d, 0)[1])
b.close()
print("done")
"""


def test_contexts_with_few_sms_sweep_with_the_other_kernels():
    """In a context that holds 16 of the SMs, where the blocks of an on-chip launch
    cannot all run at once, solvers use the other kernels, and batches either
    those or a plan for 16 SMs."""
    here = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, BLZ_TUNE_CACHE="off")
    env.pop("BLZ_SWEEP_VARIANT", None)
    r = subprocess.run([sys.executable, "-c", _FEW_SMS, os.path.dirname(here), here], env=env, capture_output=True,
                       text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.endswith("done\n"), r.stderr[-2000:]


def resident(s):
    """The solver's exchange buffers and error flag."""
    return internal("solver_resident", C.POINTER(ResidentWork), [C.c_void_p])(s._h).contents


def reports(call):
    """Whether the call ends with the report of a wait that gave up."""
    try:
        call()
    except _lib.BlazeError as e:
        assert e.code == _abi.BLZ_ERR_TIMEOUT, e
        return True
    return False


def test_a_wait_that_gave_up_is_reported_once_by_the_next_call_that_waits():
    with make((32, 16, 16), maxIterSolve=4) as s:
        s.sweeps(1)
        flag = C.cast(resident(s).err, C.POINTER(C.c_int))
        rhs = s.get("RHS")
        for call in (lambda: s.get("P"), s.residual, lambda: s.set("RHS", rhs), s.solve, s.project, s.step,
                     lambda: s.tight_solve(1e-2, 100, 1.5)):
            flag[0] = 1
            s.sweeps(1)                                   # does not wait: no report
            assert reports(call) and not reports(call)


def test_a_wait_that_gave_up_while_tuning_rules_the_candidate_out(monkeypatch):
    monkeypatch.setenv("BLZ_TUNE_CACHE", "off")
    monkeypatch.delenv("BLZ_SWEEP_VARIANT", raising=False)
    with make((56, 16, 16), variant=-1, maxIterSolve=4) as s:
        C.cast(resident(s).err, C.POINTER(C.c_int))[0] = 1
        assert s.solve()["sweep_variant"] in (0, 4)
        s.get("P")


def test_a_wait_that_runs_out_ends_the_launch():
    """One block's epoch is set off from the others': its waits and its
    neighbours' run out, the launch ends, the error is reported, and with the
    epoch put right the next sweeps are the segment kernel's."""
    dims = (64, 64, 64)
    with make(dims) as s, make(dims, variant=0) as ref:
        s.sweeps(1)
        p = s.get("P")
        last = resident(s).work + System(dims).bytes - 4          # the last block's epoch
        assert cudart.cudaMemset(last, 1, 4)[0] == 0
        s.sweeps(2)
        assert reports(lambda: s.get("P"))
        assert cudart.cudaMemcpy(last, last - 4, 4, cudart.cudaMemcpyKind.cudaMemcpyDeviceToDevice)[0] == 0
        s.set("P", p)
        s.sweeps(5)
        ref.sweeps(6)
        np.testing.assert_array_equal(s.get("P"), ref.get("P"))


@pytest.mark.parametrize("dims", [(128, 128, 112), (64, 192, 160), (126, 128, 128), (130, 128, 112)])
@pytest.mark.parametrize("bc", [BLZ_BC_FREE_SURFACE, BLZ_BC_REF_COMPAT])
def test_four_planes_per_thread(dims, bc):
    """Grids near the most that fit: four planes per thread, rows that fill whole
    warps and rows that are not whole quads."""
    for batches in ((1,), (2, 5)):
        out = []
        for variant in (ON_CHIP, 0):
            with make(dims, variant=variant, bc=bc) as s:
                for n in batches:
                    s.sweeps(n)
                out.append(s.get("P"))
        np.testing.assert_array_equal(*out)


def test_solves_at_once():
    """Device-loop solves of three solvers and a batch from four threads, each on its
    own stream: launches whose blocks must all run at once take turns, and sweep
    counts and pressures are those of each alone."""
    from blaze_b200.batch import Batch
    kw = dict(tol=1e-9, maxIterSolve=400, check_every=20)
    dims = [(128, 128, 128), (96, 96, 96), (130, 64, 64)]
    many = [(64, 64, 64), (48, 40, 36), (64, 96, 40)]

    def alone(d):
        def job():
            with make(d, **kw) as s:
                n = [s.solve()["iterations"] for _ in range(4)]
                return n, s.get("P")
        return job

    def batched():
        sims = [make(d, **kw) for d in many]
        b = Batch(sims)
        n = [[st["iterations"] for st in b.solve()] for _ in range(4)]
        out = [(list(k), s.get("P")) for k, s in zip(zip(*n), sims)]
        b.close()
        for s in sims:
            s.close()
        return out

    got = in_threads([alone(d) for d in dims] + [batched])
    for d, (n, p) in zip(dims + many, got[:3] + got[3]):
        with make(d, variant=0, **kw) as s:
            assert [s.solve()["iterations"] for _ in range(4)] == n, d
            np.testing.assert_array_equal(s.get("P"), p)


def test_solvers_are_made_and_solved_from_several_threads():
    """Solvers of different sizes, made, solved as device loops and closed in four
    threads over and over: every solve graph is captured while other threads
    allocate, launch and capture, and none of the captures ends early."""
    dims = [(128, 128, 128), (96, 96, 96), (130, 64, 64), (64, 64, 64)]

    def job(d):
        def rounds():
            n = set()
            for _ in range(25):
                with make(d, variant=-1, tol=1e-9, maxIterSolve=40, check_every=20) as s:
                    n.add((s.solve()["iterations"], s.solve()["iterations"]))
            return n
        return rounds

    assert in_threads([job(d) for d in dims]) == [{(40, 40)}] * 4


def test_tuned_solves_at_once_give_the_bits_of_one(monkeypatch):
    """Eight solves at once of solvers that tune their sweeps, some of which leave the
    on-chip sweeps to others: sweep counts and pressures are the segment kernel's."""
    monkeypatch.delenv("BLZ_SWEEP_VARIANT", raising=False)
    kw = dict(tol=1e-9, maxIterSolve=200, check_every=20)
    dims = [(64, 64, 64), (26, 60, 58), (120, 50, 44), (64, 40, 72)] * 2

    def job(d):
        def solve():
            with make(d, variant=-1, **kw) as s:
                st = [s.solve() for _ in range(6)]
                assert all(x["sweep_variant"] in (0, -1, 4, ON_CHIP) for x in st), st
                return [x["iterations"] for x in st], s.get("P")
        return solve

    for d, (n, p) in zip(dims, in_threads([job(d) for d in dims])):
        with make(d, variant=0, **kw) as s:
            assert [s.solve()["iterations"] for _ in range(6)] == n, d
            np.testing.assert_array_equal(s.get("P"), p)
