"""The work a user of this framework has it do, as timed cases.

Every case goes through the public Python API (FluidSolver, Batch,
WarmStartUNet, RenderEngine) the way a program uses it.  Kinds:

  frame    one simulation frame (addSource + step) of a scene whose fields the
           host application owns: it writes the frame's T, U, V, W (and the
           density scalar) through the solver's field pointers and reads the
           new fields there.  Small previews, production frames, fire with
           curl noise and wind.
  project  the projection alone (divergence, a fixed number of sweeps,
           gradient) on a host's velocity field: the drop-in for a code that
           has its own advection, with the reference's Neumann solve.
  solve    a pressure solve to a relative FP64 residual with a sweep cap, the
           frame's dominant cost; plain or in defect-correction form.
  warm     the same solve started by the learned warm start.
  batch    one frame of many small simulations of uneven sizes, stepped
           together (dataset generation).
  forward  the warm-start network's forward pass.
  train    one training sample's loss and parameter gradients.
  render   one image of a temperature field, read back to the host.

Sizes come from the repository's scenes (64^3 smoke plume, 128^3 fire, the
256^3 plume family, the 384^3 large fire, the batch's five grids, 128^3
training crops) and, in draw(), from the ranges around them.

exact() restates every computed output in FP64 torch.
"""
import math

import numpy as np
import torch

from blaze_b200 import _abi
from blaze_b200.batch import Batch
from blaze_b200.render import RenderEngine, default_render_params
from blaze_b200.scenes import BATCH_DIMS, SceneSettings, Timer
from blaze_b200.solver import FluidSolver
from blaze_b200.unet import WarmStartUNet, weights_path

DT = 1.0 / 24
TIME = 0.5                                   # scene time of the frames (drives the noise)


def listed():
    return [
        # an interactive preview: everything is latency and launches
        {"name": "frame_preview_32", "kind": "frame", "w": 32, "h": 32, "d": 32, "sweeps": 20, "tol": 0.0,
         "fire": False, "density": False, "particles": 500},
        # the smoke plume at 64^3 with the density scalar, 80 sweeps
        {"name": "frame_plume_64", "kind": "frame", "w": 64, "h": 64, "d": 64, "sweeps": 80, "tol": 0.0,
         "fire": False, "density": True, "particles": 2000},
        # fire and smoke at 128^3: curl noise, wind, 400 sweeps at most
        {"name": "frame_fire_128", "kind": "frame", "w": 128, "h": 128, "d": 128, "sweeps": 400, "tol": 1e-4,
         "fire": True, "density": False, "particles": 20000},
        # a 256^3 production frame with a fixed sweep budget
        {"name": "frame_plume_256", "kind": "frame", "w": 256, "h": 256, "d": 256, "sweeps": 80, "tol": 0.0,
         "fire": False, "density": False, "particles": 20000},
        # the projection alone on a ragged box, the reference's default 200 sweeps
        {"name": "project_120x100x84", "kind": "project", "w": 120, "h": 100, "d": 84, "sweeps": 200,
         "closed": True},
        # the 256^3 solve to 1e-4, capped at 2000 sweeps
        {"name": "solve_256", "kind": "solve", "w": 256, "h": 256, "d": 256, "sweeps": 2000, "check": 20,
         "defect": False},
        # the 384^3 large-fire solve in defect-correction form
        {"name": "solve_defect_384", "kind": "solve", "w": 384, "h": 384, "d": 384, "sweeps": 320, "check": 80,
         "defect": True},
        # the learned solve at the training crops' size
        {"name": "warm_128", "kind": "warm", "w": 128, "h": 128, "d": 128, "sweeps": 400, "check": 20},
        # dataset generation: uneven plumes stepped together
        {"name": "batch_16", "kind": "batch", "count": 16, "mix": 4, "sweeps": 400},
        # the network alone on the production grid
        {"name": "forward_256", "kind": "forward", "w": 256, "h": 256, "d": 256},
        # one training sample on a 128^3 crop
        {"name": "train_128", "kind": "train", "w": 128, "h": 128, "d": 128},
        # one 720p image of a 256^3 fire
        {"name": "render_256", "kind": "render", "w": 256, "h": 256, "d": 256, "width": 1280, "height": 720,
         "lights": 1},
    ]


def _log_int(rng, lo, hi, step=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(["frame", "frame", "project", "solve", "warm", "batch", "forward", "train", "render"])
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(3, 32), "mix": rng.randint(5, 10 ** 6),
                "sweeps": 20 * _log_int(rng, 2, 20)}
    if kind in ("warm", "forward", "train"):
        hi = 128 if kind == "train" else 192
        c = {"kind": kind, "w": _log_int(rng, 32, hi, 8), "h": _log_int(rng, 32, hi, 8),
             "d": _log_int(rng, 32, hi, 8)}
        if kind == "warm":
            c.update(sweeps=20 * _log_int(rng, 2, 20), check=20)
        return c
    # widths are mostly multiples of 8, any even width now and then; the other axes are free
    hi = 224 if kind != "solve" else 256
    c = {"kind": kind, "w": _log_int(rng, 24, hi, rng.choice([8, 8, 8, 2])), "h": _log_int(rng, 20, hi),
         "d": _log_int(rng, 20, hi)}
    if kind == "frame":
        fire = rng.random() < 0.5
        c.update(sweeps=20 * _log_int(rng, 1, 10), tol=0.0 if rng.random() < 0.5 else 1e-4, fire=fire,
                 density=not fire and rng.random() < 0.5, particles=_log_int(rng, 200, 20000))
    elif kind == "project":
        c.update(sweeps=_log_int(rng, 10, 300), closed=rng.random() < 0.5)
    elif kind == "solve":
        c.update(sweeps=80 * _log_int(rng, 1, 12), check=rng.choice([20, 40, 80]), defect=rng.random() < 0.4)
    else:
        c.update(width=_log_int(rng, 320, 1280), height=_log_int(rng, 180, 720), lights=rng.randint(1, 3))
    return c


# ---------------------------------------------------------------------------
# Scenes and inputs
# ---------------------------------------------------------------------------
def _batch_dims(case):
    r = np.random.default_rng(case["mix"])
    return [BATCH_DIMS[i] for i in r.integers(0, len(BATCH_DIMS), case["count"])]


def _scene(case, dims=None):
    W, H, D = dims or (case["w"], case["h"], case["d"])
    dx = 1.0 / W
    s = SceneSettings(gridRes=(W, H, D), dx=dx, dt=DT, domainBboxMax=(W * dx, H * dx, D * dx),
                      closedBounds=(1, 1, 1, 0, 1, 1), bc_mode=_abi.BLZ_BC_FREE_SURFACE, maxIterSolve=case.get("sweeps", 80),
                      tol=case.get("tol", 0.0), check_every=case.get("check", 20), buoyancy=1.0,
                      vorticityConf=0.3 * 64.0 / max(W, H, D, 64), reset_pressure=1)
    kind = case["kind"]
    if kind == "frame":
        s.windAmp = 0.2 * dx / DT
        s.coolingRate, s.drag = 0.1, 0.05
        if case["fire"]:
            s.turbulence_amp, s.turbulence_scale = 0.5 * 128 * dx, 4.0
            s.turbMaskTempRamp = (0.8, 1.6)
            s.bc_mode = _abi.BLZ_BC_REF_COMPAT
        if case["density"]:
            s.density_field, s.buoyancy_alpha = 1, 0.05
    elif kind == "project":
        s.bc_mode = _abi.BLZ_BC_REF_COMPAT
        if case["closed"]:
            s.closedBounds = (1,) * 6
    elif kind == "solve":
        s.tol, s.defect_correction = 1e-4, int(case["defect"])
    elif kind == "warm":
        s.tol, s.reset_pressure = 1e-4, 0
    elif kind == "batch":
        s.tol = 1e-4
    return s


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _modes(shape, gen, count, kmax):
    """A smooth random field: `count` separable waves of up to kmax half periods."""
    out = torch.zeros(shape, device="cuda")
    for _ in range(count):
        axes = []
        for n in shape:
            k, ph = torch.rand(2, device="cuda", generator=gen)
            axes.append(torch.sin(math.pi * (1 + k * (kmax - 1)) * torch.arange(n, device="cuda") / n + 6.28 * ph))
        out += axes[0][:, None, None] * axes[1][None, :, None] * axes[2][None, None, :]
    return out


def _plume_t(shape, gen, blobs=4):
    """A temperature field of warm blobs in still air (exact zeros outside)."""
    D, H, W = shape
    out = torch.zeros(shape, device="cuda")
    for _ in range(blobs):
        c = torch.rand(3, device="cuda", generator=gen) * 0.6 + 0.2
        r = 0.06 + 0.08 * torch.rand(1, device="cuda", generator=gen)
        g = [torch.exp(-((torch.arange(n, device="cuda") / n - c[a]) / r) ** 2) for a, n in enumerate((D, H, W))]
        out += 1.2 * g[0][:, None, None] * g[1][None, :, None] * g[2][None, None, :]
    out *= 1 + 0.3 * _modes(shape, gen, 3, 14).clamp(-1, 1)
    return torch.where(out > 0.02, out, torch.zeros_like(out))


def _fields(s, seed, density=False):
    """T, U, V, W (, DENSITY) of a developed flow: speeds up to about two cells per frame."""
    W, H, D = s.gridRes
    gen = _gen(seed)
    f = {"T": _plume_t((D, H, W), gen)}
    v = 0.6 * s.dx / s.dt
    f["U"] = v * _modes((D, H, W + 1), gen, 6, 10)
    f["V"] = v * _modes((D, H + 1, W), gen, 6, 10)
    f["W"] = v * _modes((D + 1, H, W), gen, 6, 10)
    if density:
        f["DENSITY"] = 0.8 * _plume_t((D, H, W), gen)
    return f


def _particles(s, seed, count):
    """Two balls of source particles in the lower half, 1.5 cells wide each."""
    r = np.random.default_rng(seed)
    W, H, D = s.gridRes
    rad = min(12.0, min(W, H, D) / 5.0)
    rec = np.zeros((count, 8), np.float32)
    d = r.standard_normal((count, 3))
    d *= (r.random((count, 1)) ** (1 / 3)) * rad / np.linalg.norm(d, axis=1, keepdims=True)
    lo = np.array([rad + 2, rad + 2, rad + 2])
    hi = np.array([W - rad - 2, max(0.5 * H, rad + 3), D - rad - 2])
    centres = r.uniform(np.minimum(lo, hi), np.maximum(lo, hi), (2, 3))
    rec[:, :3] = (centres[np.arange(count) % 2] + d) * s.dx + np.array(s.domainBboxMin)
    rec[:, 4] = 0.4 * s.dx / s.dt
    rec[:, 6], rec[:, 7] = 1.5 * s.dx, r.uniform(0.5, 1.5, count)
    s.sourceMaxParticleCount = count
    return rec


def _rhs(s, seed):
    """A right-hand side like a frame's: smooth buoyant sources plus cell-scale noise."""
    W, H, D = s.gridRes
    gen = _gen(seed)
    t = _plume_t((D, H, W), gen)
    r = (t - t.mean()) + 0.2 * _modes((D, H, W), gen, 4, 20) + 0.05 * torch.randn((D, H, W), device="cuda", generator=gen)
    return (r * (0.1 / (DT * s.dx))).contiguous()


class _View:
    """A solver's buffer as torch sees it; keeps the solver alive."""

    def __init__(self, solver, ptr, shape):
        self.solver = solver
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (ptr, False), "version": 3}


class _Fields:
    """Zero-copy tensors of a solver's front buffers (they alternate)."""

    def __init__(self, solver):
        self.solver, self.seen = solver, {}

    def __getitem__(self, name):
        ptr = self.solver.field_ptr(name)
        t = self.seen.get((name, ptr))
        if t is None:
            t = torch.as_tensor(_View(self.solver, ptr, self.solver.params.field_shape(name)), device="cuda")
            self.seen[name, ptr] = t
        return t


class State:
    pass


def _open_solver(st, s, particles=None, density=None):
    return FluidSolver(Timer(time=TIME), s, particles=particles, density=density, stream=st.stream.cuda_stream)


def prepare(case, seed):
    st = State()
    st.case, kind = case, case["kind"]
    st.stream = torch.cuda.Stream()
    if kind == "batch":
        st.sims, st.inputs = [], []
        for i, dims in enumerate(_batch_dims(case)):
            s = _scene(case, dims)
            parts = _particles(s, seed * 1000 + i, 2000)
            st.sims.append(FluidSolver(Timer(time=TIME), s, particles=parts))
            st.inputs.append(_fields(s, seed * 1000 + i))
        torch.cuda.synchronize()
        st.batch = Batch(st.sims)
        st.stream = torch.cuda.ExternalStream(st.batch.stream)
        st.views = [_Fields(x) for x in st.sims]
        return st
    s = st.scene = _scene(case)
    W, H, D = s.gridRes
    if kind == "frame":
        parts = _particles(s, seed, case["particles"])
        dens = np.linspace(0.2, 1.0, len(parts), dtype=np.float32) if case["density"] else None
        st.inputs = _fields(s, seed, case["density"])
        st.solver = _open_solver(st, s, parts, dens)
        st.views = _Fields(st.solver)
    elif kind == "project":
        st.inputs = {k: v for k, v in _fields(s, seed).items() if k != "T"}
        st.solver = _open_solver(st, s)
        st.views, st.p = _Fields(st.solver), torch.empty((D, H, W), device="cuda")
    elif kind in ("solve", "warm"):
        st.solver, st.p = _open_solver(st, s), torch.empty((D, H, W), device="cuda")
        rhs = _rhs(s, seed)
        torch.cuda.synchronize()
        st.solver.set_device("RHS", rhs.data_ptr())
        if kind == "warm":
            st.net = WarmStartUNet(s.gridRes).load(weights_path("plume256.npz"))
            st.solver.set_warm_start(st.net)
            st.p_prev = _p_prev(s, rhs, seed)
    elif kind in ("forward", "train"):
        st.net = WarmStartUNet(s.gridRes).load(weights_path("plume256.npz"))
        st.params, st.rhs = s.to_params(), _rhs(s, seed)
        st.p_prev = _p_prev(s, st.rhs, seed)
        if kind == "train":
            st.target = st.p_prev + 0.1 * st.p_prev.std() * _modes((D, H, W), _gen(seed + 7), 4, 6)
        else:
            st.out = torch.empty((D, H, W), device="cuda")
    else:
        st.t = _plume_t((D, H, W), _gen(seed), blobs=8)
        st.engine = RenderEngine(Timer(), s, default_render_params(s, case["width"], case["height"], case["lights"]))
    torch.cuda.synchronize()
    return st


def _p_prev(s, rhs, seed):
    """The previous frame's pressure: smooth, with the level a solve would give it."""
    W, H, D = s.gridRes
    scale = s.density * s.dx * s.dx / s.dt
    return (scale * rhs.std() * min(W, H, D) * 2.0 * _modes((D, H, W), _gen(seed + 3), 5, 5)).contiguous()


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(st):
    kind = st.case["kind"]
    if kind == "frame":
        with torch.cuda.stream(st.stream):
            for name, t in st.inputs.items():
                st.views[name].copy_(t)
            st.solver.addSource()
            stats = st.solver.step()
        out = {name: st.views[name] for name in st.inputs}
        out["sweeps"] = stats["iterations"]
        return out
    if kind == "project":
        with torch.cuda.stream(st.stream):
            for name, t in st.inputs.items():
                st.views[name].copy_(t)
            st.solver.project()
            st.solver.get_device("P", st.p.data_ptr())
        return dict({name: st.views[name] for name in st.inputs}, P=st.p)
    if kind in ("solve", "warm"):
        if kind == "warm":
            st.solver.set_device("P", st.p_prev.data_ptr())
        stats = st.solver.solve()
        st.solver.get_device("P", st.p.data_ptr())
        return {"P": st.p, "sweeps": stats["iterations"]}
    if kind == "batch":
        with torch.cuda.stream(st.stream):
            for v, f in zip(st.views, st.inputs):
                for name, t in f.items():
                    v[name].copy_(t)
            st.batch.add_source()
            stats = st.batch.step([TIME] * len(st.sims))
        return [dict({name: v[name] for name in ("T", "V")}, sweeps=q["iterations"])
                for v, q in zip(st.views, stats)]
    if kind == "forward":
        return st.net.forward(st.params, st.rhs, st.p_prev, out=st.out)
    if kind == "train":
        loss, _ = st.net.loss_grad(st.params, st.rhs, st.p_prev, st.target)
        return {"loss": loss, "grads": st.net.get_grads()}
    st.engine.render(st.t)
    return st.engine.image()


# ---------------------------------------------------------------------------
# What one pass cannot do without
# ---------------------------------------------------------------------------
NET_FLOPS = 120160.0                         # forward, per fine voxel
NET_PARAMS = 1.41e6
FRAME_FLOPS = 4 * (64 * 2 + 3 * 3 * 30) + 300


def work(case):
    kind = case["kind"]
    if kind == "batch":
        n = float(sum(w * h * d for w, h, d in _batch_dims(case)))
        return {"bytes": 8 * 4 * n, "flops": n * (FRAME_FLOPS + 9.0 * case["sweeps"])}
    n = float(case["w"]) * case["h"] * case["d"]
    if kind == "frame":
        fields = 5 if case["density"] else 4
        return {"bytes": 8 * fields * n + 32.0 * case["particles"], "flops": n * (FRAME_FLOPS + 9.0 * case["sweeps"])}
    if kind == "project":
        return {"bytes": 4 * 7 * n, "flops": n * (20 + 9.0 * case["sweeps"])}
    if kind == "solve":
        return {"bytes": 8 * n, "flops": 9.0 * case["sweeps"] * n}
    if kind == "warm":
        return {"bytes": 12 * n + 4 * NET_PARAMS, "flops": (9.0 * case["sweeps"] + NET_FLOPS) * n}
    if kind == "forward":
        return {"bytes": 12 * n + 4 * NET_PARAMS, "flops": NET_FLOPS * n}
    if kind == "train":
        return {"bytes": 12 * n + 8 * NET_PARAMS, "flops": 3 * NET_FLOPS * n}
    rays = float(case["width"]) * case["height"]
    steps = 0.5 * max(case["w"], case["h"], case["d"])
    return {"bytes": 4 * n + 12 * rays, "flops": rays * steps * (20 + case["lights"] * steps)}


# ---------------------------------------------------------------------------
# The same outputs in FP64 torch
# ---------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind == "render":
        return None                          # defined by the texture unit's 8-bit filter weights
    if kind == "batch":
        out = []
        for i, dims in enumerate(_batch_dims(case)):
            s = _scene(case, dims)
            f = _exact_frame(s, _fields(s, seed * 1000 + i), _particles(s, seed * 1000 + i, 2000), None)
            out.append({"T": f["T"], "V": f["V"], "sweeps": None})
        return out
    s = _scene(case)
    if kind == "frame":
        parts = _particles(s, seed, case["particles"])
        dens = np.linspace(0.2, 1.0, len(parts), dtype=np.float32) if case["density"] else None
        return dict(_exact_frame(s, _fields(s, seed, case["density"]), parts, dens), sweeps=None)
    if kind == "project":
        f = {k: v.double() for k, v in _fields(s, seed).items() if k != "T"}
        p = _Pressure(s, _divergence(s, f))
        p.sweep(s.maxIterSolve)
        _gradient(s, f, p.p)
        return dict(f, P=p.p)
    if kind == "solve":
        p = _Pressure(s, _rhs(s, seed).double())
        p.solve()
        return {"P": p.p, "sweeps": None}
    rhs = _rhs(s, seed)
    prev = _p_prev(s, rhs, seed)
    with np.load(weights_path("plume256.npz"), allow_pickle=False) as z:
        params, kappa = torch.from_numpy(z["params"]).double().cuda(), float(z["kappa"])
    pr = _Pressure(s, rhs.double(), prev.double())
    x, level = _net_input(s, pr, kappa)
    if kind == "train":
        D, H, W = rhs.shape
        target = prev + 0.1 * prev.std() * _modes((D, H, W), _gen(seed + 7), 4, 6)
        params.requires_grad_(True)
        loss = ((_net(params, x) - (target.double() - prev.double()) / level) ** 2).mean()
        loss.backward()
        return {"loss": float(loss), "grads": params.grad}
    with torch.no_grad():
        delta = _net(params, x)
    if kind == "forward":
        return delta
    d = level * delta
    r = pr.residual()
    ad = pr.apply(d)
    pr.set(pr.p + ((d * r).sum() / (d * ad).sum()) * d)
    pr.solve()
    return {"P": pr.p, "sweeps": None}


def _open(s):
    cb = s.closedBounds                      # grid y runs down: j = 0 is the world's yMax
    return [not cb[4], not cb[5], not cb[3], not cb[2], not cb[0], not cb[1]]      # z-, z+, y-, y+, x-, x+


class _Pressure:
    """Red-black Gauss-Seidel on the 7-point system, cells (z, y, x)."""

    SIDES = [(0, 0), (0, 2), (1, 0), (1, 2), (2, 0), (2, 2)]           # (axis, offset in the padded array)

    def __init__(self, s, rhs, p=None):
        D, H, W = rhs.shape
        self.s, self.b = s, (s.density * s.dx * s.dx / s.dt) * rhs
        self.pad = torch.zeros((D + 2, H + 2, W + 2), dtype=torch.float64, device="cuda")
        self.p = self.pad[1:-1, 1:-1, 1:-1]
        if p is not None:
            self.p.copy_(p)
        dirichlet = s.bc_mode == _abi.BLZ_BC_FREE_SURFACE
        self.count = torch.zeros((D, H, W), dtype=torch.float64, device="cuda")
        for (axis, off), op in zip(self.SIDES, _open(s)):
            c = torch.ones_like(self.count)
            edge = [slice(None)] * 3
            edge[axis] = 0 if off == 0 else rhs.shape[axis] - 1
            c[tuple(edge)] = 1.0 if dirichlet and op else 0.0
            self.count += c
        z, y, x = (torch.arange(n, device="cuda") for n in (D, H, W))
        self.red = ((z[:, None, None] + y[None, :, None] + x[None, None, :]) & 1) == 0

    def set(self, p):
        self.p.copy_(p)

    def _neighbour(self, pad, axis, off):
        sl = [slice(1, -1)] * 3
        sl[axis] = slice(off, off + pad.shape[axis] - 2)
        return pad[tuple(sl)]

    def _sum(self, pad, out):
        for axis, off in self.SIDES:
            out += self._neighbour(pad, axis, off)
        return out

    def sweep(self, n):
        for _ in range(n):
            for colour in (self.red, ~self.red):
                v = self._sum(self.pad, self.b.clone()).div_(self.count)
                self.p.copy_(torch.where(colour, v, self.p))

    def apply(self, x):
        pad = torch.zeros_like(self.pad)
        pad[1:-1, 1:-1, 1:-1] = x
        return self.count * x - self._sum(pad, torch.zeros_like(x))

    def residual(self):
        return self.b - self.apply(self.p)

    def solve(self):
        done = 0
        while float(self.residual().norm() / self.b.norm()) > self.s.tol and done < self.s.maxIterSolve:
            n = min(self.s.check_every, self.s.maxIterSolve - done)
            self.sweep(n)
            done += n


def _divergence(s, f):
    U, V, W = f["U"], f["V"], f["W"]
    ih = 1.0 / s.dx
    r = -ih * (U[:, :, 1:] - U[:, :, :-1] + V[:, 1:] - V[:, :-1] + W[1:] - W[:-1])
    o = _open(s)
    if not o[4]: r[:, :, 0] -= ih * U[:, :, 0]
    if not o[5]: r[:, :, -1] += ih * U[:, :, -1]
    if not o[2]: r[:, 0] -= ih * V[:, 0]
    if not o[3]: r[:, -1] += ih * V[:, -1]
    if not o[0]: r[0] -= ih * W[0]
    if not o[1]: r[-1] += ih * W[-1]
    return r


def _gradient(s, f, p):
    k = s.dt / (s.density * s.dx)
    o = _open(s)
    ghost = s.bc_mode == _abi.BLZ_BC_FREE_SURFACE
    for axis, name in ((0, "W"), (1, "V"), (2, "U")):
        a = f[name].movedim(axis, 0)
        q = p.movedim(axis, 0)
        a[1:-1] -= k * (q[1:] - q[:-1])
        for end, inner, sign, op in ((0, 1, 1.0, o[2 * axis]), (-1, -2, -1.0, o[2 * axis + 1])):
            if not op:
                a[end] = 0.0
            elif ghost:
                a[end] -= sign * k * q[end]
            else:
                a[end] = a[inner]


OFFSET = {"T": (0.5, 0.5, 0.5), "DENSITY": (0.5, 0.5, 0.5), "U": (0.5, 0.5, 0.0), "V": (0.5, 0.0, 0.5),
          "W": (0.0, 0.5, 0.5)}                                       # (z, y, x)


def _clamped(c, n):
    c = c.clamp(0.0, n - 1.001)
    i = c.long()
    return i, c - i


def _on_grid(a, name, zyx):
    """Trilinear samples of a field at the product grid of three coordinate vectors (in cells)."""
    for axis in range(3):
        i, w = _clamped(zyx[axis] - OFFSET[name][axis], a.shape[axis])
        w = w.reshape([-1 if q == axis else 1 for q in range(3)])
        a = a.index_select(axis, i) * (1 - w) + a.index_select(axis, i + 1) * w
    return a


def _points(shape, off):
    return [torch.arange(n, dtype=torch.float64, device="cuda") + o for n, o in zip(shape, off)]


def _trilinear(a, name, pos):
    sy, sz = a.shape[2], a.shape[1] * a.shape[2]
    (z, fz), (y, fy), (x, fx) = (_clamped(pos[q] - OFFSET[name][q], a.shape[q]) for q in range(3))
    q, a = z * sz + y * sy + x, a.reshape(-1)
    row = lambda o: a[q + o] * (1 - fx) + a[q + o + 1] * fx
    return (1 - fz) * ((1 - fy) * row(0) + fy * row(sy)) + fz * ((1 - fy) * row(sz) + fy * row(sz + sy))


def _cubic(t):
    t2, t3 = t * t, t * t * t
    return [-t / 3 + t2 / 2 - t3 / 6, 1 - t2 + (t3 - t) / 2, t + (t2 - t3) / 2, (t3 - t) / 6]


def _tricubic(a, name, pos, clamp):
    idx, wts = [], []
    for q in range(3):
        i, f = _clamped(pos[q] - OFFSET[name][q], a.shape[q])
        idx.append([(i - 1).clamp(min=0), i, i + 1, (i + 2).clamp(max=a.shape[q] - 1)])
        wts.append(_cubic(f))
    sy, sz, flat = a.shape[2], a.shape[1] * a.shape[2], a.reshape(-1)
    cut = (lambda v: v.clamp(min=0)) if clamp else (lambda v: v)
    zs = 0
    for kz in range(4):
        ys = 0
        for jy in range(4):
            base = idx[0][kz] * sz + idx[1][jy] * sy
            ys = ys + wts[1][jy] * cut(sum(wts[2][ix] * flat[base + idx[2][ix]] for ix in range(4)))
        zs = zs + wts[0][kz] * cut(ys)
    return cut(zs)


def _advect(s, f):
    r = s.dt / s.dx                          # positions in cells
    out = {}
    for name, a in f.items():
        new = torch.empty_like(a)
        for z0 in range(0, a.shape[0], 32):  # slabs bound the memory
            shape = (min(32, a.shape[0] - z0),) + tuple(a.shape[1:])
            o = OFFSET[name]
            pz, py, px = _points(shape, (o[0] + z0, o[1], o[2]))
            p = [t.expand(shape).reshape(-1) for t in (pz[:, None, None], py[None, :, None], px[None, None, :])]
            vel = lambda at: [_trilinear(f[n], n, at) for n in ("W", "V", "U")]
            k1 = vel(p)
            k2 = vel([c - 0.5 * r * k for c, k in zip(p, k1)])
            k3 = vel([c - 0.75 * r * k for c, k in zip(p, k2)])
            at = [c - r * (2 * a1 + 3 * a2 + 4 * a3) / 9 for c, a1, a2, a3 in zip(p, k1, k2, k3)]
            new[z0:z0 + shape[0]] = _tricubic(a, name, at, name in ("T", "DENSITY")).reshape(shape)
        out[name] = new
    return out


def _splat(s, f, rec, dens):
    W, H, D = s.gridRes
    rec = torch.from_numpy(rec).double().cuda()
    lo = torch.tensor(s.domainBboxMin, dtype=torch.float64, device="cuda")
    size_y = s.domainBboxMax[1] - s.domainBboxMin[1]
    pos = torch.stack([rec[:, 2] - lo[2], size_y - (rec[:, 1] - lo[1]), rec[:, 0] - lo[0]], 1)
    radius = rec[:, 6] / 2
    values = {"T": rec[:, 7], "U": rec[:, 3], "V": -rec[:, 4], "W": rec[:, 5]}
    if dens is not None:
        values["DENSITY"] = torch.from_numpy(dens).double().cuda()
    for name, val in values.items():
        a = f[name]
        acc = torch.zeros(a.numel(), dtype=torch.float64, device="cuda")
        off = torch.tensor(OFFSET[name], dtype=torch.float64, device="cuda")
        base = torch.floor(pos / s.dx - off).long()
        for o in range(64):
            c = base + torch.tensor([o // 16 - 1, o // 4 % 4 - 1, o % 4 - 1], device="cuda")
            ok = ((c >= 0) & (c < torch.tensor(a.shape, device="cuda"))).all(1)
            x = (pos - (c + off) * s.dx).norm(dim=1) / radius
            m = torch.where((x <= 1) & ok, 1 - x * x * (3 - 2 * x), torch.zeros_like(x))
            c = c.clamp(min=0)
            q = ((c[:, 0] * a.shape[1] + c[:, 1]) * a.shape[2] + c[:, 2]).clamp(max=a.numel() - 1)
            acc.index_add_(0, q, m * val)
        acc = acc.reshape(a.shape)
        f[name] = torch.where(acc.abs() > 1e-5, acc, a)


def _vorticity(s, f):
    W, H, D = s.gridRes
    dx, cells = s.dx, _points((D, H, W), (0.5, 0.5, 0.5))
    at = lambda n, axis, d: _on_grid(f[n], n, [c + (d if q == axis else 0) for q, c in enumerate(cells)])
    diff = lambda n, axis: (at(n, axis, 1.0) - at(n, axis, -1.0)) / (2 * dx)
    om = torch.stack([diff("W", 1) - diff("V", 0), diff("U", 0) - diff("W", 2), diff("V", 2) - diff("U", 1)])
    mag = om.norm(dim=0)
    g = torch.zeros_like(om)
    g[0][:, :, 1:-1] = (mag[:, :, 2:] - mag[:, :, :-2]) / (2 * dx)
    g[1][:, 1:-1] = (mag[:, 2:] - mag[:, :-2]) / (2 * dx)
    g[2][1:-1] = (mag[2:] - mag[:-2]) / (2 * dx)
    speed = torch.stack([_on_grid(f[n], n, cells) for n in ("U", "V", "W")]).norm(dim=0)
    norm = mag + 1e-20 / (dx * s.dt)
    om = torch.where(norm > speed, om * (speed / norm), om)
    force = 0.5 * s.dt * s.vorticityConf * dx * torch.cross(g, om, dim=0)
    inner = torch.zeros((D, H, W), dtype=torch.float64, device="cuda")
    inner[2:D - 2, 2:H - 2, 2:W - 2] = 1.0
    return force * inner


def _to_faces(f, cells):
    """Adds a cell vector field to both faces of each cell along each axis."""
    for name, c, axis in (("U", cells[0], 2), ("V", cells[1], 1), ("W", cells[2], 0)):
        a, n = f[name], c.shape[axis]
        a.narrow(axis, 0, n).add_(c)
        a.narrow(axis, 1, n).add_(c)


def _perlin(px, py, pz, scale, seed):
    """Gradient noise; the lattice hash reads an FP32 sum, so that sum is formed in FP32."""
    one = torch.float32
    p = [(c.to(one) * torch.tensor(scale, dtype=one)) for c in (px, py, pz)]
    base = [c.floor() for c in p]
    frac = [(c - b).double() for c, b in zip(p, base)]
    fma = lambda a, b, c: (a.double() * b + c.double()).to(one)
    grads = torch.tensor([[1, 1, 0], [-1, 1, 0], [1, -1, 0], [-1, -1, 0], [1, 0, 1], [-1, 0, 1], [1, 0, -1],
                          [-1, 0, -1], [0, 1, 1], [0, -1, 1], [0, 1, -1], [0, -1, -1], [1, 1, 0], [0, -1, 1],
                          [-1, 1, 0], [0, -1, -1]], dtype=torch.float64, device="cuda")

    def corner(dx, dy, dz):
        x, y, z = base[0] + dx, base[1] + dy, base[2] + dz
        acc = fma(z, 149812.0, fma(x, 1723.0, y * 93241.0)) + 3824.0 + float(seed)
        h = acc.double().clamp(0, 4294967295.0).long()
        m = 0xFFFFFFFF
        h = (h + 0x7ed55d16 + (h << 12)) & m
        h = (h ^ 0xc761c23c) ^ (h >> 19)
        h = (h + 0x165667b1 + (h << 5)) & m
        h = ((h + 0xd3a2646c) & m) ^ ((h << 9) & m)
        h = (h + 0xfd7046c5 + (h << 3)) & m
        h = (h ^ 0xb55a4f09) ^ (h >> 16)
        g = grads[h & 15]
        return g[..., 0] * (frac[0] - dx) + g[..., 1] * (frac[1] - dy) + g[..., 2] * (frac[2] - dz)

    u, v, w = (t * t * t * (t * (6 * t - 15) + 10) for t in frac)
    x = [corner(0, dy, dz) * (1 - u) + corner(1, dy, dz) * u for dz in (0, 1) for dy in (0, 1)]
    return (x[0] * (1 - v) + x[1] * v) * (1 - w) + (x[2] * (1 - v) + x[3] * v) * w


def _turbulence(s, f):
    W, H, D = s.gridRes
    offset = math.fmod(float(np.float32(TIME)) * ((W + H + D) / 3.0), 25000.0)
    offset = float(np.float32(offset))
    fit = lambda v, a, b: ((v - a) / (b - a)).clamp(0, 1)
    noise = {}
    for name in ("U", "V", "W"):
        pts = _points(f[name].shape, OFFSET[name])
        m = 1 - fit(_on_grid(f["T"], "T", pts), *s.turbMaskTempRamp)
        speed = torch.stack([_on_grid(f[n], n, pts) for n in ("U", "V", "W")]).norm(dim=0)
        m = m * fit(speed, *s.turbMaskVelRamp)
        z, y, x = (t.float() for t in _points(f[name].shape, (0.0, 0.0, 0.0)))
        sh = {"U": (x, 2), "V": (y, 1), "W": (z, 0)}[name][1]
        z, y, x = (t + offset if q == sh else t for q, t in enumerate((z, y, x)))
        shape = f[name].shape
        n = _perlin(x[None, None, :].expand(shape), y[None, :, None].expand(shape), z[:, None, None].expand(shape),
                    float(np.float32(1.0) / np.float32(s.turbulence_scale)), 123)
        noise[name] = m * s.turbulence_amp * n
    u0, u1 = noise["U"][:, :, :-1], noise["U"][:, :, 1:]
    v0, v1 = noise["V"][:, :-1], noise["V"][:, 1:]
    w0, w1 = noise["W"][:-1], noise["W"][1:]
    dudx, dvdy, dwdz = (u1 - v0) / s.dx, (v1 - v0) / s.dx, (w1 - v0) / s.dx
    c = torch.stack([dvdy - dwdz, dwdz - dudx, dudx - dvdy])
    mean = torch.stack([u0 + u1, v0 + v1, w0 + w1]).norm(dim=0) / 2
    _to_faces(f, 0.5 * s.dt * mean * c / (c.norm(dim=0) + 1e-20 / (s.dx * s.dt)))


def _wind(s, f):
    keep = 1 - s.dt
    W = s.gridRes[0]
    for name in ("U", "V", "W"):
        a = f[name]
        slab = torch.arange(a.shape[2], device="cuda")
        slab = ((slab < 2) | (slab >= W - 1))[None, None, :]
        f[name] = torch.where(slab, a * keep + (s.windAmp * s.dt if name == "U" else 0.0), a)


def _exact_frame(s, fields, rec, dens):
    f = {k: v.double() for k, v in fields.items()}
    _splat(s, f, rec, dens)
    f["T"] = f["T"] * (1 - s.dt * s.coolingRate)
    for n in ("U", "V", "W"):
        f[n] = f[n] * (1 - s.dt * s.drag)
    force = _vorticity(s, f)
    face = _points(f["V"].shape, OFFSET["V"])
    lift = s.buoyancy * _on_grid(f["T"], "T", face)
    if s.density_field:
        lift = lift - s.buoyancy_alpha * _on_grid(f["DENSITY"], "DENSITY", face)
    _to_faces(f, force)
    f["V"] += s.dt * s.gravity * lift
    if s.windAmp > 0:
        _wind(s, f)
    if s.turbulence_amp > 0:
        _turbulence(s, f)
    p = _Pressure(s, _divergence(s, f))
    if s.tol > 0:
        p.solve()
    else:
        p.sweep(s.maxIterSolve)
    _gradient(s, f, p.p)
    return _advect(s, f)


# (taps, cin, cout) of the network's layers in parameter order
LAYERS = [(27, 16, 16), (27, 16, 16), (27, 16, 32), (27, 32, 32), (27, 32, 64), (27, 64, 64), (27, 64, 128),
          (27, 128, 128), (27, 128, 64), (27, 64, 64), (27, 64, 32), (27, 32, 32), (27, 32, 16), (27, 16, 16),
          (8, 128, 64), (8, 64, 32), (8, 32, 16), (1, 16, 1)]


def _net_input(s, pr, kappa):
    """The padded 16-channel input and the correction's scale kappa rms(r)."""
    r = pr.residual()
    rms = [a.square().mean().sqrt() for a in (pr.b, pr.p, r)]
    D, H, W = r.shape
    x = torch.zeros((16, D + 2, H + 2, W + 2), dtype=torch.float64, device="cuda")
    for c, (a, m) in zip((0, 2, 3), zip((pr.b, pr.p, r), rms)):
        x[c, 1:-1, 1:-1, 1:-1] = a / m
    for (axis, off), op in zip(_Pressure.SIDES, _open(s)):
        if not (op and s.bc_mode == _abi.BLZ_BC_FREE_SURFACE):
            x[1].select(axis, 0 if off == 0 else -1).fill_(1.0)
    return x, kappa * rms[2]


def _net(params, x):
    """The U-Net in FP64: shifted products, channels first; x carries its halo."""
    w, b, at = [], [], 0
    for taps, cin, cout in LAYERS:
        n = taps * cin * cout
        w.append(params[at:at + n].reshape(taps, cout, cin))
        b.append(params[at + n:at + n + cout])
        at += n + cout

    def conv(i, a, padded=False):
        a = a if padded else torch.nn.functional.pad(a, (1,) * 6)
        D, H, W = (n - 2 for n in a.shape[1:])
        y = 0
        for t in range(27):
            z, yy, xx = t // 9, t // 3 % 3, t % 3
            v = a[:, z:z + D, yy:yy + H, xx:xx + W].reshape(a.shape[0], -1)
            y = y + w[i][t] @ v
        return torch.relu(y + b[i][:, None]).reshape(-1, D, H, W)

    def up(i, a):
        c, D, H, W = a.shape
        y = torch.einsum("toc,cn->otn", w[i], a.reshape(c, -1)) + b[i][:, None, None]
        y = y.reshape(-1, 2, 2, 2, D, H, W).permute(0, 4, 1, 5, 2, 6, 3)
        return y.reshape(-1, 2 * D, 2 * H, 2 * W)

    pool = lambda a: torch.nn.functional.avg_pool3d(a[None], 2)[0]
    e0 = conv(1, conv(0, x, padded=True))
    e1 = conv(3, conv(2, pool(e0)))
    e2 = conv(5, conv(4, pool(e1)))
    e3 = conv(7, conv(6, pool(e2)))
    d2 = conv(9, conv(8, torch.cat([up(14, e3), e2])))
    d1 = conv(11, conv(10, torch.cat([up(15, d2), e1])))
    d0 = conv(13, conv(12, torch.cat([up(16, d1), e0])))
    return (w[17][0] @ d0.reshape(16, -1) + b[17][:, None]).reshape(x.shape[1] - 2, x.shape[2] - 2, x.shape[3] - 2)
