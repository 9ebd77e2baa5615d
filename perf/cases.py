"""What a user of this framework has it compute, as measurable cases.

A case is a dict of plain values with a `kind`:

  preset   one frame of a solver preset (MacSimulation3D(n, box, algorithm_params)):
           kick and stir emitter, a fixed budget of 600 SOR iterations
  plume    one step of the benchmark plume (Reflection + MacCormack, two profile
           sources), every projection solved to a relative residual with the
           mixed-precision SOR
  learned  the same step with the learned solver (flexible PCG around the
           shipped coarse-grid U-Net)
  batch    one step of several uneven plume scenes with one Batch.advance
  project  one staged pressure projection, on device fields (optionally around a
           solid sphere) or on host arrays as the Projection3D plugin is called
  advect   staged transport of the three velocity components and the smoke
  network  forward and backward of the U-Net (a training step's two halves)
  plume2d  one frame of the 2D reflection plume, read back for display

Tolerance-driven steps start every pass from the same snapshot, written into the
simulation's device fields on its own stream as a coupled program does, so that
every pass solves the same problem; fixed-budget frames simply go on. A pass is
ordered with the caller's stream on both sides, as a program that reads the
fields between steps needs it.
"""
import ctypes as C
import math

import numpy as np
import torch

import vapor_b200 as vb
from vapor_b200 import abi, mac2d
from vapor_b200.learned import COARSE_WEIGHTS, WarmStartNet
from vapor_b200.plume import DT, omega_for, scene_params

BATCH_SIZES = (32, 48, 64, 96, 128)
LAYERS = ((16, 16), (16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (96, 32), (32, 32), (48, 16), (16, 16))


def listed():
    return [
        # the default-constructed solver: 32^3, box 4.5, interactive frame rate; latency and launches count
        {"name": "preset_32", "kind": "preset", "algorithm": abi.REFLECTION_MACCORMACK, "n": 32},
        # the cheapest preset on a grid nobody tuned for: odd, rows that divide by nothing
        {"name": "preset_45", "kind": "preset", "algorithm": abi.SIMPLE_SEMI_LAGRANGIAN, "n": 45},
        # a small plume solved to 1e-6, as when a scene is set up or training pairs are made
        {"name": "plume_64", "kind": "plume", "n": 64, "rel": 1e-6},
        # the benchmark grid with the plain solver: the largest pass
        {"name": "plume_256", "kind": "plume", "n": 256, "rel": 1e-6},
        # the learned solver at the smaller grid it pays for, and at the benchmark grid
        {"name": "learned_128", "kind": "learned", "n": 128, "rel": 1e-6},
        {"name": "learned_256", "kind": "learned", "n": 256, "rel": 1e-6},
        # uneven scenes stepped together
        {"name": "batch_8", "kind": "batch", "sizes": "32,48,64,64,96,96,128,32", "rel": 1e-6},
        # the mixed-precision projection to 1e-8 around an obstacle, device fields
        {"name": "project_obstacle_96", "kind": "project", "n": 96, "rel": 1e-8, "solver": "mixed", "solid": True,
         "host": False},
        # the staged plugin inside a host program: numpy fields in and out, the reference's SOR
        {"name": "project_host_50", "kind": "project", "n": 50, "rel": 1e-5, "solver": "sor", "solid": False,
         "host": True},
        # transport alone, limiter on, a cell size that is no power of two
        {"name": "advect_160", "kind": "advect", "n": 160, "method": abi.MACCORMACK},
        # training: the coarse network at its resolution for a 256^3 solve
        {"name": "network_64", "kind": "network", "n": 64},
        # the 2D application scene with MacCormack smoke, read back every frame
        {"name": "plume2d_128", "kind": "plume2d", "n": 128, "method": mac2d.MACCORMACK},
    ]


def _spread(rng, lo, hi, step=1):
    """An integer multiple of `step` in lo..hi, spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi + step)))
    return max(lo, min(hi, int(v) // step * step))


def draw(rng):
    kind = rng.choice(["preset", "preset", "plume", "plume", "learned", "learned", "batch", "project", "project",
                       "advect", "network", "plume2d"])
    if kind == "preset":
        return {"kind": kind, "algorithm": rng.randrange(4), "n": _spread(rng, 16, 96)}
    if kind == "plume":
        return {"kind": kind, "n": _spread(rng, 24, 224), "rel": rng.choice([1e-5, 1e-6])}
    if kind == "learned":
        return {"kind": kind, "n": _spread(rng, 64, 240, 16), "rel": rng.choice([1e-5, 1e-6])}
    if kind == "batch":
        sizes = [rng.choice(BATCH_SIZES) for _ in range(rng.randint(3, 12))]
        return {"kind": kind, "sizes": ",".join(map(str, sizes)), "rel": 1e-6}
    if kind == "project":
        if rng.random() < 0.5:
            return {"kind": kind, "n": _spread(rng, 16, 96), "rel": 1e-5, "solver": "sor", "solid": False, "host": True}
        return {"kind": kind, "n": _spread(rng, 24, 160), "rel": rng.choice([1e-6, 1e-8]), "solver": "mixed",
                "solid": rng.random() < 0.5, "host": False}
    if kind == "advect":
        return {"kind": kind, "n": _spread(rng, 24, 224),
                "method": rng.choice([abi.SEMI_LAGRANGIAN, abi.MACCORMACK])}
    if kind == "network":
        return {"kind": kind, "n": _spread(rng, 16, 64, 4)}
    return {"kind": kind, "n": _spread(rng, 32, 256), "method": rng.choice([mac2d.SEMI_LAGRANGIAN, mac2d.MACCORMACK])}


# ---- inputs ---------------------------------------------------------------

def _shapes(n):
    return abi.field_shapes(n)


def _swirl(n, seed, amplitude, box=1.0):
    """u, v, w of eight Gaussian vortices with seeded centres and axes (the
    benchmark's initial state), normal velocity zero on the walls."""
    rng = np.random.default_rng(seed)
    centres = rng.uniform(0.2, 0.8, size=(8, 3)) * box
    axes = rng.normal(size=(8, 3))
    axes /= np.linalg.norm(axes, axis=1, keepdims=True)
    sigma, h = 0.08 * box, box / n
    out = []
    for c, shape in enumerate(_shapes(n)[1:]):
        z, y, x = [((torch.arange(s, device="cuda", dtype=torch.float32) + (0.0 if c == d else 0.5)) * h)
                   for d, s in zip((2, 1, 0), shape)]
        f = torch.zeros(shape, device="cuda")
        for (cx, cy, cz), a in zip(centres.tolist(), axes.tolist()):
            r = ((x - cx)[None, None, :], (y - cy)[None, :, None], (z - cz)[:, None, None])
            g = torch.exp(-(r[0] ** 2 + r[1] ** 2 + r[2] ** 2) / (2 * sigma * sigma)) * (amplitude / sigma)
            i, j = ((1, 2), (2, 0), (0, 1))[c]
            f += (a[i] * r[j] - a[j] * r[i]) * g
        wall = f.movedim(2 - c, 0)
        wall[0] = wall[-1] = 0
        out.append(f.contiguous())
    return out


def _smooth(shape, seed, slope):
    """A seeded random field with spectrum ~ k^slope, largest magnitude 1."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    f = torch.fft.rfftn(torch.randn(shape, generator=gen, device="cuda"))
    ks = [torch.fft.fftfreq(s, device="cuda") * s for s in shape[:2]] + [torch.fft.rfftfreq(shape[2], device="cuda") * shape[2]]
    k = torch.sqrt(ks[0][:, None, None] ** 2 + ks[1][None, :, None] ** 2 + ks[2][None, None, :] ** 2)
    k[0, 0, 0] = 1.0
    amp = k ** slope
    amp[0, 0, 0] = 0.0
    g = torch.fft.irfftn(f * amp, s=shape)
    return (g / g.abs().max()).contiguous()


def _velocity(n, seed):
    """A seeded velocity with a full spectrum and divergence, walls closed."""
    out = []
    for c, shape in enumerate(_shapes(n)[1:]):
        f = _smooth(shape, 3 * seed + c, -11.0 / 6.0)
        wall = f.movedim(2 - c, 0)
        wall[0] = wall[-1] = 0
        out.append(f)
    return out


def _smoke(n, seed):
    return _smooth(_shapes(n)[0], seed, -1.5).clamp(min=0.0).contiguous()


def _sphere(n, seed):
    rng = np.random.default_rng(seed)
    centre, radius = rng.uniform(0.3, 0.7, size=3), rng.uniform(0.1, 0.2)
    c = (np.arange(n) + 0.5) / n
    d2 = (c[None, None, :] - centre[0]) ** 2 + (c[None, :, None] - centre[1]) ** 2 + (c[:, None, None] - centre[2]) ** 2
    return (d2 < radius * radius).astype(np.uint8)


class _Memory:
    """Device memory of the library, as torch takes it without a copy; a tensor
    over it keeps this object, and so the simulation that owns the memory."""

    def __init__(self, owner, pointer, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (pointer, False), "shape": tuple(shape), "typestr": "<f4",
                                         "version": 3}


class _Resident:
    """A resident simulation in a program that works on its device fields."""

    def __init__(self, sim):
        self.sim = sim
        self.stream = torch.cuda.ExternalStream(sim.stream())
        self.views = {}
        self.snapshot = None

    def fields(self):
        out = []
        for p, shape in zip(self.sim.device_fields(), _shapes(self.sim.n)):
            if p not in self.views:
                self.views[p] = torch.as_tensor(_Memory(self.sim, p, shape), device="cuda")
            out.append(self.views[p])
        return out

    def load(self, fields):
        self.stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(self.stream):
            for dst, src in zip(self.fields(), fields):
                dst.copy_(src, non_blocking=True)

    def results(self):
        """The fields after the step, for work on the current stream."""
        torch.cuda.current_stream().wait_stream(self.stream)
        return self.fields()

    def develop(self, steps):
        """A developed state: the seeded start advanced a few steps."""
        for _ in range(steps):
            self.sim.advance(DT)
        self.sim.synchronize()
        self.snapshot = [f.clone() for f in self.fields()]


def _plume(n, seed, rel, learned=False, **scene):
    p = scene_params(vb.default_params(), n, rel=rel, max_iterations=20000, **scene)
    if learned:
        p.solver_kind = abi.SOLVER_FPCG
    state = _Resident(vb.MacSimulation3D(n, 1.0, p))
    if learned:
        state.net = WarmStartNet.load(COARSE_WEIGHTS)
        state.sim.set_preconditioner(state.net)
    torch.cuda.synchronize()
    state.load([torch.zeros(_shapes(n)[0], device="cuda")] + _swirl(n, seed, 0.5))
    return state


def prepare(case, seed):
    kind, n = case["kind"], case.get("n")
    if kind == "preset":
        p = vb.algorithm_params(case["algorithm"])
        p.random_seed = seed & 0xFFFFFFFF
        state = _Resident(vb.MacSimulation3D(n, 4.5, p))
        start = [torch.zeros(_shapes(n)[0], device="cuda")] + _swirl(n, seed, 0.5, 4.5)
        torch.cuda.synchronize()
        state.load(start)
        for _ in range(2):
            state.sim.advance(1 / 60)
        state.sim.synchronize()
        return state
    if kind in ("plume", "learned"):
        state = _plume(n, seed, case["rel"], kind == "learned")
        state.develop(2)
        return state
    if kind == "batch":
        rng = np.random.default_rng(seed)
        scenes = []
        for k, size in enumerate(int(s) for s in case["sizes"].split(",")):
            source = (float(rng.uniform(0.3, 0.7)), float(rng.uniform(0.3, 0.7)), float(rng.uniform(0.1, 0.25)))
            scenes.append(_plume(size, 101 * seed + k, case["rel"], sources=(source,),
                                 radius=float(rng.uniform(0.05, 0.12)), buoyancy=float(rng.uniform(0.5, 2.0))))
        batch = vb.Batch([s.sim for s in scenes])
        for _ in range(2):
            batch.advance(DT)
        batch.synchronize()
        for s in scenes:
            s.snapshot = [f.clone() for f in s.fields()]
        return {"batch": batch, "scenes": scenes}
    if kind == "project":
        stage = vb.StageBackend(n, 1.0)
        stage.set_solver_kind(abi.SOLVER_MIXED_REFINEMENT if case["solver"] == "mixed" else abi.SOLVER_RED_BLACK_SOR)
        if case["solid"]:
            stage.set_solid(_sphere(n, seed))
        options = vb.ProjectionOptions(DT, omega_for(n), vb.LinearSolveOptions.defaults(
            max_iterations=20000 if case["solver"] == "mixed" else 1000, relative_tolerance=case["rel"],
            absolute_tolerance=0.0))
        fields = _velocity(n, seed)
        if case["host"]:
            fields = [f.cpu().numpy() for f in fields]
        return {"stage": stage, "options": options, "fields": fields}
    if kind == "advect":
        stage = vb.StageBackend(n, 1.0)
        stream = C.c_void_p()
        vb.check(vb.library().vapor_stage_stream(stage._h, C.byref(stream)))
        return {"stage": stage, "method": case["method"], "stream": torch.cuda.ExternalStream(stream.value), "flow": _swirl(n, seed, 0.5),
                "source": _swirl(n, seed + 77, 0.5), "smoke": _smoke(n, seed),
                "out": [torch.empty(s, device="cuda") for s in (_shapes(n)[1:] + _shapes(n)[:1])]}
    if kind == "network":
        features = torch.zeros((n, n, n, 16), device="cuda", dtype=torch.bfloat16)
        rhs, g = _network_inputs(n, seed)
        features[..., 0] = rhs.to(torch.bfloat16)
        return {"net": WarmStartNet.load(COARSE_WEIGHTS), "features": features, "grad": g,
                "out": torch.empty((n, n, n), device="cuda")}
    sim = mac2d.ReflectionSimulation2D(n, mac2d.reflection_app_params(case["method"]))
    rng = np.random.default_rng(seed)
    shapes = abi.field_shapes_2d(n)
    grid = np.linspace(0, 2 * np.pi, n, dtype=np.float32)
    phase = rng.uniform(0, 2 * np.pi, size=4).astype(np.float32)
    smoke = np.clip(np.sin(grid + phase[0])[:, None] * np.sin(grid + phase[1])[None, :], 0, 1).astype(np.float32)
    u = np.zeros(shapes[1], np.float32)
    v = np.zeros(shapes[2], np.float32)
    u[:, 1:-1] = (0.2 * np.sin(grid[:, None] + phase[2]) * np.sin(grid[None, :-1] / 2)).astype(np.float32)
    v[1:-1, :] = (0.2 * np.sin(grid[:-1, None] / 2) * np.sin(grid[None, :] + phase[3])).astype(np.float32)
    sim.upload(smoke, u, v)
    return sim


def _network_inputs(n, seed):
    """A coarse residual's features (mean zero, rms 1) and an output gradient."""
    rhs = _smooth((n, n, n), seed, -1.0)
    g = _smooth((n, n, n), seed + 5, -1.0)
    return (rhs - rhs.mean()) / rhs.std(), (g / g.std()).contiguous()


# ---- one pass -------------------------------------------------------------

def run(state):
    if isinstance(state, mac2d.ReflectionSimulation2D):
        state.advance(1 / 60)
        return state.download()
    if isinstance(state, _Resident):
        if state.snapshot is None:
            state.stream.wait_stream(torch.cuda.current_stream())
            state.sim.advance(1 / 60)
        else:
            state.load(state.snapshot)
            state.sim.advance(DT)
        return state.results()
    if "batch" in state:
        for s in state["scenes"]:
            s.load(s.snapshot)
        state["batch"].advance(DT)
        return [s.results() for s in state["scenes"]]
    if "options" in state:
        stage, options = state["stage"], state["options"]
        if isinstance(state["fields"][0], np.ndarray):
            work = [f.copy() for f in state["fields"]]
            _, pressure = stage.project(*work, options, 6.0, want_pressure=True)
            return work + [pressure]
        work = [f.clone() for f in state["fields"]]
        pressure = torch.empty(_shapes(stage.n)[0], device="cuda")
        torch.cuda.current_stream().synchronize()  # the stage works on its own stream
        stage.project_device(*[f.data_ptr() for f in work], options, 6.0, pressure.data_ptr())
        return work + [pressure]
    if "flow" in state:
        lib, h = vb.library(), state["stage"]._h
        flow = [f.data_ptr() for f in state["flow"]]
        method = state["method"]
        for axis in range(3):
            vb.check(lib.vapor_stage_advect_face_device(h, axis, DT, 3.0, method, state["source"][axis].data_ptr(),
                                                        *flow, state["out"][axis].data_ptr()))
        with torch.cuda.stream(state["stream"]):
            state["out"][3].copy_(state["smoke"], non_blocking=True)  # the smoke is moved in place
        vb.check(lib.vapor_stage_advect_scalar_device(h, DT, 3.0, method, state["out"][3].data_ptr(), *flow))
        return state["out"]
    net, n = state["net"], state["out"].shape[0]
    lib = vb.library()
    grads = np.empty(net.count, np.float32)
    vb.check(lib.vapor_unet_forward_features(net.handle, n, state["features"].data_ptr(), state["out"].data_ptr()))
    vb.check(lib.vapor_unet_backward(net.handle, n, state["grad"].data_ptr(), grads.ctypes.data))
    return [state["out"], grads]


# ---- what a pass cannot do without ----------------------------------------

def _step_bytes(n):
    return 2 * 4 * (n ** 3 + 3 * n * n * (n + 1))  # the state read and written once


def _network_flops(n):
    levels = (n, n, n // 2, n // 2, n // 4, n // 4, n // 2, n // 2, n, n)
    return sum(2 * 27 * ci * co * m ** 3 for (ci, co), m in zip(LAYERS, levels))


def work(case):
    kind, n = case["kind"], case.get("n")
    if kind == "preset":  # the caller asks for its 600 SOR iterations: 10 operations a cell each
        return {"bytes": _step_bytes(n), "flops": 600 * 10 * n ** 3}
    if kind in ("plume", "learned"):  # how many iterations the tolerance takes is the solver's business
        return {"bytes": _step_bytes(n), "flops": 0}
    if kind == "batch":
        return {"bytes": sum(_step_bytes(int(s)) for s in case["sizes"].split(",")), "flops": 0}
    if kind == "project":
        return {"bytes": 4 * (6 * n * n * (n + 1) + n ** 3), "flops": 0}
    if kind == "advect":
        return {"bytes": 4 * (9 * n * n * (n + 1) + 2 * n ** 3), "flops": 0}
    if kind == "network":  # forward, input gradients and weight gradients
        return {"bytes": n ** 3 * (32 + 4 + 4) + 4 * 2 * 359761, "flops": 3 * _network_flops(n)}
    return {"bytes": 4 * 2 * (n * n + 2 * n * (n + 1)) + 4 * n * n, "flops": 120 * 8 * n * n}


# ---- the same in 64 bits ---------------------------------------------------

def exact(case, seed):
    """Projections, transport and the network in 64 bits. A whole step has no
    such value here: its limiter and iteration counts branch on rounding."""
    with torch.no_grad():
        if case["kind"] == "project":
            return _exact_project(case, seed)
        if case["kind"] == "advect":
            return _exact_advect(case, seed)
    return _exact_network(case, seed) if case["kind"] == "network" else None


def _along_axes(m, t):
    """Matrix `m` applied along each of the three axes."""
    for _ in range(3):
        t = torch.tensordot(t, m, dims=([0], [1]))
    return t


def _exact_project(case, seed):
    n = case["n"]
    u, v, w = [f.double() for f in _velocity(n, seed)]
    h, dt = float(np.float32(1.0) / np.float32(n)), float(np.float32(DT))
    fluid = torch.ones((n, n, n), dtype=torch.bool, device=u.device)
    if case["solid"]:
        fluid = torch.from_numpy(_sphere(n, seed) == 0).to(u.device)
    open_faces = []  # a face is open between two fluid cells
    for c in range(3):
        f, d = fluid, 2 - c
        pad = torch.zeros_like(f.narrow(d, 0, 1))
        open_faces.append(torch.cat([pad, f], d) & torch.cat([f, pad], d))
    vel = [a * o for a, o in zip((u, v, w), open_faces)]
    div = sum((a.narrow(2 - c, 1, n) - a.narrow(2 - c, 0, n)) for c, a in enumerate(vel)) / h
    b = torch.where(fluid, -div * (h * h / dt), torch.zeros_like(div))
    b = torch.where(fluid, b - b.sum() / fluid.sum(), torch.zeros_like(b))

    def gradient(p):
        return [o * torch.cat([p.narrow(2 - c, 0, 1) * 0, p.narrow(2 - c, 1, n - 1) - p.narrow(2 - c, 0, n - 1),
                               p.narrow(2 - c, 0, 1) * 0], 2 - c) for c, o in enumerate(open_faces)]

    if not case["solid"]:  # cosine transforms diagonalise the closed box
        k = torch.arange(n, dtype=torch.float64, device=u.device)
        m = torch.cos(math.pi * (k[None, :] + 0.5) * k[:, None] / n) * math.sqrt(2.0 / n)
        m[0] /= math.sqrt(2.0)
        e = 2 - 2 * torch.cos(math.pi * k / n)
        lam = e[:, None, None] + e[None, :, None] + e[None, None, :]
        lam[0, 0, 0] = 1.0
        t = _along_axes(m, b) / lam
        t[0, 0, 0] = 0.0
        p = _along_axes(m.T, t)
    else:  # conjugate gradients on the fluid cells
        def apply(x):
            return -sum(g.narrow(2 - c, 1, n) - g.narrow(2 - c, 0, n) for c, g in enumerate(gradient(x)))
        p, r = torch.zeros_like(b), b.clone()
        d, rr = r.clone(), (r * r).sum()
        stop = 1e-26 * rr
        for k in range(20 * n):
            q = apply(d)
            a = rr / (d * q).sum()
            p, r = p + a * d, r - a * q
            new = (r * r).sum()
            if k % 16 == 0 and bool(new < stop):
                break
            d, rr = r + (new / rr) * d, new
        p = torch.where(fluid, p - p[fluid].mean(), torch.zeros_like(p))
    return [a - dt * g / h for a, g in zip(vel, gradient(p))] + [p]


def _at(field, loc, n, h, pos):
    """Clamped trilinear lookup of `field` (staggered along axis `loc`, -1: cells)."""
    idx = []
    for c in range(3):
        if c == loc:
            g = (pos[c] / h).clamp(0, n)
            i0 = g.long().clamp(max=n - 1)
            i1 = i0 + 1
        else:
            g = (pos[c] / h - 0.5).clamp(0, n - 1)
            i0 = g.long()
            i1 = (i0 + 1).clamp(max=n - 1)
        idx.append((i0, i1, g - i0))
    total = 0.0
    for corner in range(8):
        weight, at = 1.0, []
        for c in range(3):
            i0, i1, t = idx[c]
            high = corner >> c & 1
            at.append(i1 if high else i0)
            weight = weight * (t if high else 1 - t)
        total = total + weight * field[at[2], at[1], at[0]]
    return total


def _exact_advect(case, seed):
    n = case["n"]
    flow = [f.double() for f in _swirl(n, seed, 0.5)]
    fields = [f.double() for f in _swirl(n, seed + 77, 0.5)] + [_smoke(n, seed).double()]
    h, dt = float(np.float32(1.0) / np.float32(n)), float(np.float32(DT))
    out = []
    for field, loc in zip(fields, (0, 1, 2, -1)):
        ijk = torch.meshgrid(*[torch.arange(s, device=field.device) for s in field.shape], indexing="ij")
        pos = [(ijk[2 - c] + (0.0 if c == loc else 0.5)) * h for c in range(3)]
        vel = [_at(flow[c], c, n, h, pos) for c in range(3)]
        back = [p - a * dt for p, a in zip(pos, vel)]
        moved = _at(field, loc, n, h, back)
        if case["method"] == abi.MACCORMACK:
            ahead = [p + a * dt for p, a in zip(pos, vel)]
            leaves = sum(((p < 0) | (p > 1)).int() for p in back + ahead) > 0
            fast = torch.sqrt(sum(a * a for a in vel)) * dt / h > 3.0
            corrected = moved + 0.5 * (field - _at(moved, loc, n, h, ahead))
            lo, hi = torch.full_like(field, math.inf), torch.full_like(field, -math.inf)
            base = [(back[c] / h - (0.0 if c == loc else 0.5)).trunc().long().clamp(0, n if c == loc else n - 1)
                    for c in range(3)]
            for corner in range(8):
                at = [(base[c] + (corner >> c & 1)).clamp(max=field.shape[2 - c] - 1) for c in range(3)]
                donor = field[at[2], at[1], at[0]]
                lo, hi = torch.minimum(lo, donor), torch.maximum(hi, donor)
            moved = torch.where(leaves | fast, moved, torch.minimum(torch.maximum(corrected, lo), hi))
        out.append(moved)
    return out


def _exact_network(case, seed):
    n = case["n"]
    rhs, g = _network_inputs(n, seed)
    x = torch.zeros((1, 16, n, n, n), dtype=torch.float64, device=rhs.device)
    x[0, 0] = rhs.to(torch.bfloat16).double()
    p = torch.from_numpy(np.load(COARSE_WEIGHTS)).double().to(rhs.device).requires_grad_(True)
    offsets, at = [], 0
    for ci, co in LAYERS:
        offsets.append(at)
        at += 27 * ci * co + co
    F = torch.nn.functional

    def conv(i, x):
        ci, co = LAYERS[i]
        w = p[offsets[i]:offsets[i] + 27 * ci * co].reshape(3, 3, 3, co, ci).permute(3, 4, 0, 1, 2)
        taps = F.pad(x, (1,) * 6)  # 27 shifted products: 64-bit matrix products
        s, out = x.shape[2], 0.0
        for k in range(27):
            dz, dy, dx = k // 9, k // 3 % 3, k % 3
            out = out + torch.einsum("oi,bizyx->bozyx", w[:, :, dz, dy, dx],
                                     taps[:, :, dz:dz + s, dy:dy + s, dx:dx + s])
        b = p[offsets[i] + 27 * ci * co:offsets[i] + 27 * ci * co + co]
        return F.relu(out + b[None, :, None, None, None])

    def up(t):
        return t.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4)

    skip1 = conv(1, conv(0, x))
    skip2 = conv(3, conv(2, F.avg_pool3d(skip1, 2)))
    d = conv(5, conv(4, F.avg_pool3d(skip2, 2)))
    d = conv(7, conv(6, torch.cat([up(d), skip2], 1)))
    d = conv(9, conv(8, torch.cat([up(d), skip1], 1)))
    y = torch.einsum("i,bizyx->bzyx", p[at:at + 16], d)[0] + p[at + 16]
    y.backward(g.double())
    return [y.detach(), p.grad.cpu().numpy()]
