"""The workloads this library is measured on, through its public entry points.

A case is a dict of plain values; `prepare` makes what a user's program holds
before the call (simulators with their terrain and state on the GPU), `run` is
one pass, `work` the bytes and operations a pass cannot do without, and `exact`
the same pass in 64 bits with plain torch. Kinds of case:

  step      `steps` calls of perform_step from the simulator's current state, as
            a script does that steps a simulation itself
  loop      one simulate_to_time over a time of about `steps` CFL steps, the
            device-resident time loop, from an initial state that the program
            keeps on the GPU and copies in before each run
  request   a whole call on host data: upload an initial state, run to an end
            time with a gauge callback, read the water volume and the final state
  ensemble  simulate_batch of `members` simulations from their current states,
            each to its own end time, at most `steps` steps
  gradient  the forward run with checkpoints and the reverse sweep of a gauge
            loss: dLoss/dB for every bottom corner and dLoss/dCz

Scenes: "dam" is the circular dam break on a flat bottom in the unit square,
"hills" a lake among Gaussian hills with moving water, thin films on dry land,
rain, infiltration and friction (cells of `dx` metres).
"""
import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "volumefluxes.jl_gb300"))

import volumefluxes_sm103 as vf  # noqa: E402
from volumefluxes_sm103.adjoint import GaugeAdjoint  # noqa: E402
from volumefluxes_sm103.ensemble import simulate_batch  # noqa: E402

G = 9.81
KAPPA = 1e-5
THETA = 1.2
WORDS_PER_STEP = 7   # state in (3), state out (3), bottom corners (1)
FLOPS_PER_STEP = {("linear", "rk2"): 760, ("linear", "fe"): 370, ("none", "rk2"): 640, ("none", "fe"): 310}


def _case(name, kind, nx, ny, real, scene, steps, **kw):
    c = dict(name=name, kind=kind, nx=nx, ny=ny, real=real, scene=scene, steps=steps, bc="wall", rec="linear",
             stepper="rk2", law="bsa2012", dynamic=False, faithful=False, cutoff=1e-5, dx=1.0, members=1)
    c.update(kw)
    return c


def listed():
    return [
        # A script that steps a small dam break by hand: the smallest call, one step.
        _case("step_dam_64_f64", "step", 64, 64, "f64", "dam", 1),
        # The 256^2 circular dam break of the parity and throughput runs, in the device loop.
        _case("loop_dam_256_f64", "loop", 256, 256, "f64", "dam", 16),
        # A small flood request on host buffers: upload, simulate with gauges, download.
        _case("request_200x120_f32", "request", 200, 120, "f32", "hills", 40, cutoff=8e-2),
        # An ordinary Float32 flood run on a ragged grid, in the device loop.
        _case("loop_hills_1021x511_f32", "loop", 1021, 511, "f32", "hills", 16, cutoff=8e-2),
        # A catchment run as the terrain example sets it up: NeumannBC, rain by a
        # table, Horton infiltration, friction_bh2021, cells whose size is no power of two.
        _case("loop_terrain_611x397_f64", "loop", 611, 397, "f64", "hills", 4, bc="neumann", law="bh2021",
              dynamic=True, cutoff=8e-2, dx=2.5),
        # PeriodicBC (CartesianGrid's default) with time-dependent sources in Float32.
        _case("loop_periodic_997x753_f32", "loop", 997, 753, "f32", "hills", 8, bc="periodic", dynamic=True,
              cutoff=8e-2),
        # The headline configuration, 4096^2 wet/dry hills, in Float32 and in Float64.
        _case("step_hills_4096_f32", "step", 4096, 4096, "f32", "hills", 4),
        _case("step_hills_4096_f64", "step", 4096, 4096, "f64", "hills", 1),
        # The Float64 tolerance mode on a medium grid.
        _case("step_hills_1500x1100_faithful", "step", 1500, 1100, "f64", "hills", 2, faithful=True),
        # An ensemble of floods of mixed sizes in one batch, Float32 and Float64.
        _case("ensemble_32_f32", "ensemble", 64, 448, "f32", "hills", 24, members=32, cutoff=8e-2),
        _case("ensemble_20_f64", "ensemble", 64, 224, "f64", "hills", 8, members=20, cutoff=8e-2),
        # The gradient of a gauge loss with respect to the terrain and Manning's n.
        _case("gradient_160x128_f64", "gradient", 160, 128, "f64", "hills", 9),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges (`rng`: a random.Random)."""
    kind = rng.choices(["step", "loop", "request", "ensemble", "gradient"], [20, 40, 12, 16, 12])[0]
    real = rng.choice(["f32", "f64"])
    opts = {}
    if kind in ("step", "loop"):
        opts["bc"] = rng.choices(["wall", "periodic", "neumann"], [70, 15, 15])[0]
        opts["rec"] = rng.choices(["linear", "none"], [85, 15])[0]
        opts["stepper"] = rng.choices(["rk2", "fe"], [85, 15])[0]
        opts["dynamic"] = rng.random() < 0.25
    if kind == "ensemble":
        lo = _log_uniform(rng, 64, 128)
        hi = _log_uniform(rng, 2 * lo, 512 if real == "f32" else 256)
        return {**_case("", kind, lo, hi, real, "hills", rng.randint(4, 32 if real == "f32" else 10),
                        members=rng.randint(8, 40), cutoff=8e-2), "salt": rng.randrange(1 << 20)}
    if kind == "gradient":
        c = _case("", kind, _log_uniform(rng, 48, 256), _log_uniform(rng, 48, 256), "f64", "hills", rng.randint(4, 12),
                  law=rng.choice(["bsa2012", "fcg2016", "bh2021"]))
        return {**c, "salt": rng.randrange(1 << 20)}
    top = 400 if kind == "request" else 4096
    nx, ny = _log_uniform(rng, 48, top), _log_uniform(rng, 48, top)
    scene = "dam" if opts.get("bc", "wall") == "wall" and not opts.get("dynamic") and rng.random() < 0.2 else "hills"
    if scene == "dam":
        ny = nx = min(nx, 1024)
        opts["cutoff"] = 1e-5
    else:
        opts["dx"] = rng.choice([1.0, 1.0, 2.5, 4.0])
        opts["law"] = rng.choice(["bsa2012", "bsa2012", "fcg2016", "bh2021"])
        opts["cutoff"] = 1e-5 if kind == "step" else 8e-2
    opts["faithful"] = real == "f64" and kind != "request" and rng.random() < 0.15
    most = (1 << 26) if real == "f32" else (1 << 24)  # cell-steps of a pass
    steps = max(1, min(most // (nx * ny), rng.choice([1, 2, 4]) if kind == "step" else rng.randint(4, 40)))
    return {**_case("", kind, nx, ny, real, scene, steps, **opts), "salt": rng.randrange(1 << 20)}


# ------------------------------------------------------------------ inputs
def _generator(seed):
    g = torch.Generator(device="cpu")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


class _Inputs:
    """Bottom corners (ny+5, nx+5) and interior state (3, ny, nx), Float64 on
    the GPU, with values that the case's real type holds exactly."""

    def __init__(self, case, seed, nx=None, ny=None, depth=None):
        nx, ny = nx or case["nx"], ny or case["ny"]
        self.nx, self.ny = nx, ny
        gen = _generator(seed)
        u = lambda n, lo=0.0, hi=1.0: (torch.rand(n, generator=gen, dtype=torch.float64) * (hi - lo) + lo).cuda()  # noqa: E731
        real = torch.float32 if case["real"] == "f32" else torch.float64
        f = dict(dtype=torch.float64, device="cuda")
        if case["scene"] == "dam":
            self.dx, self.dy = 1.0 / nx, 1.0 / ny
            self.extent = [[0.0, 1.0], [0.0, 1.0]]
            x = (torch.arange(nx, **f) + 0.5) / nx
            y = (torch.arange(ny, **f) + 0.5) / ny
            cx, cy = u(2, 0.4, 0.6)
            r = torch.sqrt((x[None, :] - cx) ** 2 + (y[:, None] - cy) ** 2)
            lo, hi = u(1, 0.8, 1.2), u(1, 1.8, 2.2)
            h = torch.where(r < u(1, 0.12, 0.25), hi, lo)
            speed = u(2, -0.3, 0.3)
            self.U = torch.stack([h, h * speed[0] * torch.sin(6 * y)[:, None], h * speed[1] * torch.cos(5 * x)[None, :]])
            self.U = self.U.to(real).double()
            self.B = None
            return
        dx = case["dx"]
        self.dx = self.dy = dx
        lx, ly = nx * dx, ny * dx
        self.extent = [[0.0, lx], [0.0, ly]]
        xc = (torch.arange(nx + 5, **f) - 2) * dx
        yc = (torch.arange(ny + 5, **f) - 2) * dx
        n_hills = 24
        cx, cy, a, s = u(n_hills, 0, lx), u(n_hills, 0, ly), u(n_hills, 0.5, 4.0), u(n_hills, 50, 400) * dx
        ex = torch.exp(-((xc[None, :] - cx[:, None]) ** 2) / (2 * s[:, None] ** 2))
        ey = torch.exp(-((yc[None, :] - cy[:, None]) ** 2) / (2 * s[:, None] ** 2)) * a[:, None]
        B = ey.T @ ex + 1e-3 * xc[None, :]
        self.B = B.to(real).double()
        Bc = 0.25 * (self.B[:-1, :-1] + self.B[:-1, 1:] + self.B[1:, :-1] + self.B[1:, 1:])[2:-2, 2:-2]
        x = (torch.arange(nx, **f) + 0.5) / nx
        y = (torch.arange(ny, **f) + 0.5) / ny
        ph, am = u(8, 0, 2 * math.pi), u(4, 0.3, 1.0)
        wave = 0.12 * (am[0] * torch.sin(5 * x + ph[0])[None, :] + am[1] * torch.sin(7 * y + ph[1])[:, None])
        if depth is not None:        # a sheet of water over the terrain
            h = depth + wave
        else:                        # a lake with islands: about half of the land dry under a film of rain
            level = torch.quantile(Bc.reshape(-1)[:: max(1, Bc.numel() // 100000)], 0.75)
            film = 1.5e-4 * (1 + torch.sin(40 * x + ph[2])[None, :] * torch.sin(37 * y + ph[3])[:, None])
            h = torch.maximum(level + wave - Bc, film)
        vx = 0.6 * am[2] * torch.sin(4 * x + ph[4])[None, :] * torch.cos(6 * y + ph[5])[:, None]
        vy = 0.6 * am[3] * torch.cos(6 * x + ph[6])[None, :] * torch.sin(4 * y + ph[7])[:, None]
        damp = torch.clamp(h, max=1.0)
        self.U = torch.stack([Bc + h, h * damp * vx, h * damp * vy]).to(real).double()

    def host(self, case):
        """The interior planes as (nx, ny) arrays, x fastest, in the real type."""
        dt = np.float32 if case["real"] == "f32" else np.float64
        return [p.cpu().numpy().astype(dt).T for p in self.U]


def _speed(case, depth):
    return math.sqrt(G * depth) + 0.6


def _params(case, seed):
    """Scalar parameters of a hills case."""
    r = random.Random(int(seed) * 7919 + 13)
    return dict(rain=r.uniform(2e-6, 3e-5), infil=r.uniform(5e-7, 3e-6), manning=r.uniform(0.02, 0.06),
                table=[r.uniform(0.02, 0.2) for _ in range(3)], factor=r.uniform(0.5, 1.5))


def _simulator(case, inp, par, *, manning=None):
    backend = vf.SM103Backend(np.float32 if case["real"] == "f32" else np.float64,
                              arithmetic="faithful" if case["faithful"] else "reference")
    bc = {"wall": vf.WallBC, "periodic": vf.PeriodicBC, "neumann": vf.NeumannBC}[case["bc"]]()
    grid = vf.CartesianGrid(inp.nx, inp.ny, gc=2, boundary=bc, extent=inp.extent)
    bottom = vf.ConstantBottomTopography() if inp.B is None else vf.BottomTopography2D(inp.B.cpu().numpy().T, backend, grid)
    eq = vf.ShallowWaterEquations(bottom, depth_cutoff=case["cutoff"], desingularizing_kappa=KAPPA)
    sources, friction = [], None
    if case["scene"] == "hills":
        sources.append(vf.SourceTermBottom())
        if case["dynamic"]:
            sources.append(vf.TimeDependentRain(par["table"], [0.0, 1.0, 60.0]))
            sources.append(vf.HortonInfiltration(grid, backend, factor=par["factor"]))
        else:
            sources.append(vf.ConstantRain(par["rain"] * 3600))
            sources.append(vf.ConstantInfiltration(par["infil"]))
        law = {"bsa2012": vf.friction_bsa2012, "fcg2016": vf.friction_fcg2016, "bh2021": vf.friction_bh2021}[case["law"]]
        friction = vf.ImplicitFriction(Cz=par["manning"] ** 2, friction_function=law)
    rec = vf.LinearReconstruction(THETA) if case["rec"] == "linear" else vf.NoReconstruction()
    system = vf.ConservedSystem(backend, rec, vf.CentralUpwind(eq), eq, grid, sources, friction)
    stepper = vf.RungeKutta2() if case["stepper"] == "rk2" else vf.ForwardEulerStepper()
    return vf.Simulator(backend, system, stepper, grid, cfl=_cfl(case))


def _cfl(case):
    return 0.2 if case["scene"] == "dam" else 0.25


def _time(case, inp, steps):
    """A time of about `steps` CFL steps, as the case's real type holds it."""
    h = 2.2 if inp.B is None else float((inp.U[0].max() - inp.B.min()).cpu())
    return float(np.float32(steps * _cfl(case) * min(inp.dx, inp.dy) / _speed(case, min(h, 6.0))))


def _members(case, seed):
    """(side, depth, end time in steps) of an ensemble's members: sides log-uniform
    in [case nx, case ny], each with its own depth and length of run."""
    sides = random.Random(int(case.get("salt", 0)) * 31 + 5)
    r = random.Random(int(seed) * 31 + 7)
    out = []
    for _ in range(case["members"]):
        side = _log_uniform(sides, case["nx"], case["ny"])
        out.append((side, r.uniform(0.4, 2.0), sides.uniform(0.6, 1.0) * case["steps"]))
    return out


def _gauges(case, seed, n=32):
    r = random.Random(int(seed) * 101 + 3)
    return np.array([[r.randrange(case["nx"]), r.randrange(case["ny"])] for _ in range(n)], dtype=np.int32)


class _DeviceArray:
    def __init__(self, ptr, shape, strides, typestr):
        self.__cuda_array_interface__ = dict(shape=shape, strides=strides, typestr=typestr, data=(ptr, False), version=3)


class _Views:
    """Tensors over the simulator's two state buffers, made once per buffer:
    what a program keeps that reads and writes the state on the GPU."""

    def __init__(self, sim):
        self.sim = sim
        self.base = ctypes.c_void_p()
        self.pitch, self.plane, self.first = ctypes.c_int64(), ctypes.c_int64(), ctypes.c_int64()
        self.refs = [ctypes.byref(v) for v in (self.base, self.pitch, self.plane, self.first)]
        self.made = {}
        stream = ctypes.c_void_p()
        sim._lib.vf_stream(sim.handle, ctypes.byref(stream))
        self.stream = torch.cuda.ExternalStream(stream.value)

    def _tensors(self):
        s = self.sim
        s._lib.vf_device_state(s.handle, *self.refs)
        ptr = self.base.value
        if ptr not in self.made:
            e = s.dtype.itemsize
            a = _DeviceArray(ptr + self.first.value * e, (3, s.grid.ny + 4, s.grid.nx + 4),
                             (self.plane.value * e, self.pitch.value * e, e), "<f%d" % e)
            volume = torch.as_tensor(a, device="cuda")
            self.made[ptr] = volume, volume[:, 2:-2, 2:-2]
        return self.made[ptr]

    def current(self):
        """The interior, (3, ny, nx)."""
        return self._tensors()[1]

    def keep(self):
        """A copy of the whole volume, ghost cells included."""
        with torch.cuda.stream(self.stream):
            self.kept = self._tensors()[0].clone()

    def restore(self):
        with torch.cuda.stream(self.stream):
            self._tensors()[0].copy_(self.kept)


# ------------------------------------------------------------------ a pass
def prepare(case, seed):
    seed = int(seed) + int(case.get("salt", 0))
    kind = case["kind"]
    if kind == "ensemble":
        sims, times = [], []
        for k, (side, depth, steps) in enumerate(_members(case, seed)):
            inp = _Inputs(case, seed * 64 + k, side, side, depth)
            sim = _simulator(case, inp, _params(case, seed * 64 + k))
            vf.set_current_state(sim, inp.host(case))
            sims.append(sim)
            times.append(_time(case, inp, steps))
        return dict(case=case, sims=sims, times=times, views=[_Views(s) for s in sims])
    inp = _Inputs(case, seed, depth=1.0 if kind == "gradient" else None)
    par = _params(case, seed)
    sim = _simulator(case, inp, par)
    state = dict(case=case, sim=sim, time=_time(case, inp, case["steps"]))
    if kind == "request":
        out = np.empty((3, inp.ny, inp.nx), dtype=sim.dtype)
        state.update(host=inp.host(case), gauges=_gauges(case, seed), out=out, planes=vf.StateView(*(p.T for p in out)))
        return state
    vf.set_current_state(sim, inp.host(case))
    if kind == "gradient":
        gauges = _gauges(case, seed)
        r = random.Random(seed + 17)
        w = inp.U[0].cpu().numpy()
        state.update(gauges=gauges, target=np.array([w[j, i] + r.uniform(-0.3, 0.3) for i, j in gauges]),
                     adjoint=GaugeAdjoint(sim, case["steps"]))
    state["views"] = _Views(sim)
    if kind == "loop":
        state["views"].keep()
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "ensemble":
        ends = [float(np.float32(s.t + t)) for s, t in zip(state["sims"], state["times"])]
        res = simulate_batch(state["sims"], ends, max_steps=case["steps"])
        return [v.current() for v in state["views"]], [r.t for r in res[:8]]
    sim = state["sim"]
    if kind == "step":
        for _ in range(case["steps"]):
            vf.perform_step(sim, math.inf)
            sim.t += sim.current_timestep
        return state["views"].current(), sim.current_timestep
    if kind == "loop":
        state["views"].restore()
        sim.t = 0.0
        vf.simulate_to_time(sim, state["time"])
        return state["views"].current(), sim.t
    if kind == "request":
        sim.t = 0.0
        vf.set_current_state(sim, state["host"])
        gauges = vf.GaugeRecorder(state["gauges"])
        vf.simulate_to_time(sim, state["time"], callback=vf.IntervalWriter(state["time"] / 4, gauges))
        volume = vf.water_volume(sim)
        vf.current_interior_state(sim, state["planes"])
        return state["out"], gauges.values[-1], volume
    dts = state["adjoint"].forward()
    loss, grad_B, grad_Cz = state["adjoint"].backward(state["gauges"], state["target"])
    return dts, loss, grad_B, grad_Cz, state["views"].current()


def work(case):
    per = FLOPS_PER_STEP[(case["rec"], case["stepper"])]
    e = 4 if case["real"] == "f32" else 8
    if case["kind"] == "ensemble":
        lo, hi = math.log(case["nx"]), math.log(case["ny"])
        mean_cells = (math.exp(2 * hi) - math.exp(2 * lo)) / (2 * (hi - lo))
        cell_steps = case["members"] * 0.8 * case["steps"] * mean_cells
    else:
        cell_steps = case["nx"] * case["ny"] * case["steps"]
    if case["kind"] == "gradient":  # forward, recomputation, and a reverse step of at least twice a forward one
        return dict(bytes=cell_steps * e * WORDS_PER_STEP * 4, flops=cell_steps * per * 4)
    extra = 6 * e * case["nx"] * case["ny"] if case["kind"] == "request" else 0
    return dict(bytes=cell_steps * e * WORDS_PER_STEP + extra, flops=cell_steps * per)


# ------------------------------------------------------------------ the same in 64 bits
class _Exact:
    """The scheme in Float64 torch operations on the GPU: state (3, ny+4, nx+4)."""

    def __init__(self, case, inp, par, B=None, Cz=None):
        self.case, self.nx, self.ny, self.dx, self.dy = case, inp.nx, inp.ny, inp.dx, inp.dy
        f = dict(dtype=torch.float64, device="cuda")
        self.B = B if B is not None else inp.B
        if self.B is None:
            self.B = torch.zeros(self.ny + 5, self.nx + 5, **f)
        b = self.B
        self.Bc = 0.25 * (b[:-1, :-1] + b[:-1, 1:] + b[1:, :-1] + b[1:, 1:])
        self.bx = 0.5 * (b[:-1, :] + b[1:, :])  # x faces (ny+4, nx+5)
        self.by = 0.5 * (b[:, :-1] + b[:, 1:])  # y faces (ny+5, nx+4)
        self.cutoff = case["cutoff"]
        self.hills = case["scene"] == "hills"
        self.par = par
        self.Cz = Cz if Cz is not None else par["manning"] ** 2
        U = torch.zeros(3, self.ny + 4, self.nx + 4, **f)
        U[:, 2:-2, 2:-2] = inp.U
        self.U = self.ghosts(U)
        self.t = 0.0
        self.dt = 0.0

    def ghosts(self, U):
        U = U.clone()
        bc, nx, ny = self.case["bc"], self.nx, self.ny
        I, J = slice(2, nx + 2), slice(2, ny + 2)
        if bc == "periodic":
            U[:, J, :2], U[:, J, nx + 2:] = U[:, J, nx:nx + 2].clone(), U[:, J, 2:4].clone()
            U[:, :2, I], U[:, ny + 2:, I] = U[:, ny:ny + 2, I].clone(), U[:, 2:4, I].clone()
            return U
        sx = torch.tensor([1.0, -1.0, 1.0], dtype=U.dtype, device=U.device)[:, None, None]
        sy = torch.tensor([1.0, 1.0, -1.0], dtype=U.dtype, device=U.device)[:, None, None]
        if bc == "neumann":  # right and top: the inner ghost takes the outer ghost's value
            U[:, J, :2] = U[:, J, 2:4].flip(2).clone()
            U[:, J, nx + 2] = U[:, J, nx + 3].clone()
            U[:, :2, I] = U[:, ny:ny + 2, I].clone()
            U[:, ny + 2, I] = U[:, ny + 3, I].clone()
            return U
        U[:, J, :2], U[:, J, nx + 2:] = (sx * U[:, J, 2:4].flip(2)).clone(), (sx * U[:, J, nx:nx + 2].flip(2)).clone()
        U[:, :2, I], U[:, ny + 2:, I] = (sy * U[:, 2:4, I].flip(1)).clone(), (sy * U[:, ny:ny + 2, I].flip(1)).clone()
        return U

    @staticmethod
    def desing(h):
        small = h.abs() < KAPPA
        m = torch.clamp(h * h / (2 * KAPPA) + KAPPA / 2, max=KAPPA)
        return torch.where(small, torch.sign(torch.where(h == 0, torch.ones_like(h), h)) * torch.maximum(h.abs(), m), h)

    @staticmethod
    def minmod(a, b, c):
        lo = torch.where(a < b, a, b)
        lo = torch.where(lo < c, lo, c)
        hi = torch.where(a > b, a, b)
        hi = torch.where(hi > c, hi, c)
        zero = torch.zeros_like(a)
        return torch.where((a > 0) & (b > 0) & (c > 0), lo, torch.where((a < 0) & (b < 0) & (c < 0), hi, zero))

    def direction(self, U, face, Bc, delta, x):
        """Along the last axis: U (3, n, m), face bottoms (n, m+1); the
        derivative of the inner cells (3, n, m-4), the maximum speed."""
        c = U[:, :, 1:-1]
        Bl, Br = face[:, 1:-2], face[:, 2:-1]
        if self.case["rec"] == "none":
            L = R = torch.stack([c[0] - Bc[:, 1:-1], c[1], c[2]])
        else:
            fwd, bwd = U[:, :, 2:] - c, c - U[:, :, :-2]
            s = self.minmod(THETA * fwd, 0.5 * (fwd + bwd), THETA * bwd)
            w = c[0]
            s0 = torch.where(w - 0.5 * s[0] < Bl, 2 * (w - Bl), torch.where(w + 0.5 * s[0] < Br, 2 * (Br - w), s[0]))
            s = torch.stack([s0, s[1], s[2]])
            L, R = c - 0.5 * s, c + 0.5 * s
            L = torch.stack([L[0] - Bl, L[1], L[2]])
            R = torch.stack([R[0] - Br, R[1], R[2]])
        n, k = (1, 2) if x else (2, 1)  # normal and transverse momentum

        def side(q):
            wet = q[0] > self.cutoff
            h = torch.where(wet, q[0], torch.ones_like(q[0]))
            hs = self.desing(h)
            un, ut = q[n] / hs, q[k] / hs
            f = h * un
            c = torch.sqrt(G * h)
            z = torch.zeros_like(h)
            w_ = lambda v: torch.where(wet, v, z)  # noqa: E731
            return [w_(f), w_(f * un + 0.5 * G * h * h), w_(f * ut)], w_(un + c), w_(un - c)

        m, p = R[:, :, :-1], L[:, :, 1:]
        (fm, em1, em2), (fp, ep1, ep2) = side(m), side(p)
        ap = torch.where(ep1 > em1, ep1, em1)
        ap = torch.where(ap > 0, ap, torch.zeros_like(ap))
        am = torch.where(ep2 < em2, ep2, em2)
        am = torch.where(am < 0, am, torch.zeros_like(am))
        d = ap - am
        dry = d < KAPPA
        ds = torch.where(dry, torch.ones_like(d), d)
        F = [torch.where(dry, torch.zeros_like(d), (ap * a - am * b) / ds + (ap * am) / ds * (p[i] - m[i]))
             for i, a, b in zip((0, n, k), fm, fp)]
        speed = torch.where(dry | ((m[0] < self.cutoff) & (p[0] < self.cutoff)), torch.zeros_like(d),
                            torch.maximum(ap.abs(), am.abs()))
        out = [None] * 3
        for i, f in zip((0, n, k), F):
            out[i] = -(f[:, 1:] - f[:, :-1]) / delta
        if self.hills:
            slope = (Br - Bl)[:, 1:-1] / delta
            out[n] = out[n] - G * slope * 0.5 * (R[0] + L[0])[:, 1:-1]
        return torch.stack(out), float(speed.detach().max())

    def derivative(self, U, t):
        dU = torch.zeros_like(U)
        gx, ax = self.direction(U[:, 2:-2, :], self.bx[2:-2], self.Bc[2:-2], self.dx, True)
        tr = lambda a: a.transpose(-1, -2)  # noqa: E731
        gy, ay = self.direction(tr(U[:, :, 2:-2]), tr(self.by[:, 2:-2]), tr(self.Bc[:, 2:-2]), self.dy, False)
        dU[:, 2:-2, 2:-2] = gx + tr(gy)
        if self.hills:
            p = self.par
            if self.case["dynamic"]:
                k = 2 if t >= 60.0 else 1 if t >= 1.0 else 0
                rate = p["table"][k] / 3600 - p["factor"] * (3.272e-5 + (1.977e-4 - 3.272e-5) * math.exp(-2.43e-3 * t))
            else:
                rate = p["rain"] - p["infil"]
            dU[0] = dU[0] + rate
        return dU, ax, ay

    def friction(self, U):
        hs = self.desing(U[0] - self.Bc)
        u, v = U[1] / hs, U[2] / hs
        q = u * u + v * v
        moving = q > 0
        speed = torch.sqrt(torch.where(moving, q, torch.ones_like(q)))
        cb = torch.sign(hs) * hs.abs() ** (1.0 / 3.0)
        den = {"bsa2012": cb * hs, "fcg2016": cb * hs * hs, "bh2021": hs * hs}[self.case["law"]]
        return torch.where(moving, -self.Cz * speed / den, torch.zeros_like(speed))

    def finish(self, V, S, dt):
        if self.hills:
            V = torch.stack([V[0], V[1] / (1 - dt * S), V[2] / (1 - dt * S)])
        dry = V[0] - self.Bc < self.cutoff
        z = torch.zeros_like(V[1])
        w = torch.where(dry & (V[0] < self.Bc), self.Bc, V[0])
        return self.ghosts(torch.stack([w, torch.where(dry, z, V[1]), torch.where(dry, z, V[2])]))

    def step(self, max_dt):
        U = self.U
        dU, ax, ay = self.derivative(U, self.t)
        dt = min(_cfl(self.case) * min(self.dx / ax if ax else math.inf, self.dy / ay if ay else math.inf), max_dt)
        V = self.finish(U + dt * dU, self.friction(U) if self.hills else None, dt)
        if self.case["stepper"] == "rk2":
            dV, _, _ = self.derivative(V, self.t)
            V = self.finish(0.5 * (U + V + dt * dV), self.friction(V) if self.hills else None, dt)
        self.U, self.dt = V, dt
        return dt

    def simulate(self, end, max_steps=1 << 30):
        for _ in range(max_steps):
            if self.t >= end:
                break
            left = end - self.t
            self.t += self.step(left)
            if end - self.t < 1e-6 * self.dt:
                self.t = end

    def interior(self):
        return self.U[:, 2:-2, 2:-2].contiguous()


def exact(case, seed):
    seed = int(seed) + int(case.get("salt", 0))
    kind = case["kind"]
    if kind == "ensemble":
        if case["members"] * case["steps"] > 1200:
            return None
        states, ends = [], []
        for k, (side, depth, steps) in enumerate(_members(case, seed)):
            inp = _Inputs(case, seed * 64 + k, side, side, depth)
            e = _Exact(case, inp, _params(case, seed * 64 + k))
            e.simulate(_time(case, inp, steps), case["steps"])
            states.append(e.interior())
            ends.append(e.t)
        return states, ends[:8]
    inp = _Inputs(case, seed, depth=1.0 if kind == "gradient" else None)
    par = _params(case, seed)
    if kind == "gradient":
        return _exact_gradient(case, seed, inp, par)
    e = _Exact(case, inp, par)
    if kind == "step":
        for _ in range(case["steps"]):
            e.t += e.step(math.inf)
        return e.interior(), e.dt
    e.simulate(_time(case, inp, case["steps"]))
    if kind == "loop":
        return e.interior(), e.t
    U = e.interior()
    volume = float(((U[0] - e.Bc[2:-2, 2:-2]) * e.dx * e.dy).sum())
    return U, None, volume


def _exact_gradient(case, seed, inp, par):
    B = inp.B.clone().requires_grad_(True)
    Cz = torch.tensor(par["manning"] ** 2, dtype=torch.float64, device="cuda", requires_grad=True)
    # the initial state stays as it is when the terrain changes
    e = _Exact(case, inp, par, B, Cz)
    dts = []
    for _ in range(case["steps"]):
        dts.append(e.step(math.inf))
    gauges = _gauges(case, seed)
    r = random.Random(seed + 17)
    w0 = inp.U[0].cpu().numpy()
    target = torch.tensor([w0[j, i] + r.uniform(-0.3, 0.3) for i, j in gauges], dtype=torch.float64, device="cuda")
    g = torch.tensor(gauges.astype(np.int64), device="cuda")
    w = e.U[0, 2:-2, 2:-2][g[:, 1], g[:, 0]]
    loss = ((w - target) ** 2).sum()
    gB, gC = torch.autograd.grad(loss, (B, Cz))
    return np.array(dts), float(loss.detach()), gB.T.contiguous(), float(gC), e.interior().detach()
