"""What a user of this framework has it do, as cases that can be timed and compared.

A case is one frame, solve or network call through the public Python binding of the C ABI (smoke_b200.py): step and views
of one scene, a scene whose obstacle moves, a batch of scenes, the pressure solve alone, the preconditioner network's
evaluation and its training step. `prepare` builds what the program holds before the call (context, fields, weights) from
a seed, `run` makes the call, `exact` restates its result in torch float64 without this library.

Scenes: smooth multi-mode face velocities of about one cell per step, Gaussian density and temperature puffs, a source
at the bottom (and the same sink at the top of a closed box, so that a scene stepped for a long time stays bounded).
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PACKAGE = os.path.join(ROOT, "visual-simulation-of-smoke_b200")
if PACKAGE not in sys.path:
    sys.path.insert(0, PACKAGE)

import smoke_abi as abi  # noqa: E402
import smoke_b200  # noqa: E402

WEIGHTS = os.path.join(PACKAGE, "learned_preconditioner.f32")
OBSTACLE_FRAMES = 4     # positions a moving obstacle cycles through
LEARNING_RATE = 1e-3
SOLVERS = {
    "fixed": None,  # the ABI's own solver: config.pressure_iterations CG iterations from zero
    "jacobi": dict(mode=abi.SOLVER_JACOBI_PCG, reduction=abi.REDUCTION_FP64, max_iterations=2000, tolerance=1e-6, refinement=2),
    "multigrid": dict(mode=abi.SOLVER_MG_FCG, reduction=abi.REDUCTION_FP64, max_iterations=500, tolerance=1e-5, refinement=1, warm_start=True),
    "multigrid_cold": dict(mode=abi.SOLVER_MG_FCG, reduction=abi.REDUCTION_FP64, max_iterations=500, tolerance=1e-6, refinement=3),
    "learned": dict(mode=abi.SOLVER_LEARNED_FCG, reduction=abi.REDUCTION_FP64, max_iterations=500, tolerance=1e-5, refinement=1, warm_start=True),
}


def _step(name, nx, ny, nz, solver, mode, boundary="closed", solids=False, views="velocity"):
    return {"name": name, "kind": "step", "nx": nx, "ny": ny, "nz": nz, "solver": solver, "mode": mode, "boundary": boundary, "solids": solids, "views": views}


def listed():
    return [
        # an interactive preview grid with the ABI's default solver: launches and latency
        _step("step_32_fixed_linear", 32, 32, 32, "fixed", "linear", views="all"),
        # the trilinear configuration with Jacobi-PCG to a tolerance
        _step("step_64_jacobi_linear", 64, 64, 64, "jacobi", "linear"),
        # the reference benchmark's scene and defaults: periodic x and z, outflow top, cubic, 64 CG iterations
        _step("step_128x160x128_fixed_cubic", 128, 160, 128, "fixed", "cubic", boundary="plume", views="all"),
        # the benchmark plume's grid with the multigrid solver, warm-started frames
        _step("step_128_multigrid_cubic", 128, 128, 128, "multigrid", "cubic"),
        # the same frame with the trained preconditioner network
        _step("step_128_learned_cubic", 128, 128, 128, "learned", "cubic"),
        # an odd, ragged grid (no extent a multiple of 2) with obstacles and an outflow top, cell size not a power of two
        _step("step_97x141x83_multigrid_linear", 97, 141, 83, "multigrid", "linear", boundary="plume", solids=True),
        # a production shot: 25 M cells around a sphere
        _step("step_256x384x256_multigrid_cubic", 256, 384, 256, "multigrid", "cubic", solids=True),
        # an obstacle that moves every frame: new occupancy and solid velocity, then the step
        {"name": "obstacle_96x128x96", "kind": "obstacle", "nx": 96, "ny": 128, "nz": 96, "solver": "multigrid", "mode": "linear", "boundary": "closed", "radius": 12.0},
        # the pressure solve alone, from zero, to a tight tolerance (a host that couples its own stages)
        {"name": "solve_160x200x150_multigrid", "kind": "solve", "nx": 160, "ny": 200, "nz": 150, "solver": "multigrid_cold", "mode": "linear", "boundary": "closed", "solids": True},
        # independent scenes of uneven sizes in one batched step
        {"name": "batch_8", "kind": "batch", "count": 8, "low": 40, "high": 112, "solver": "multigrid", "mode": "linear", "boundary": "closed"},
        # the preconditioner network on the volume that a 128^3 scene gives it
        {"name": "net_apply_64", "kind": "net_apply", "nx": 64, "ny": 64, "nz": 64},
        # one training step at the training program's defaults: batch 8 on the volumes of 64^3 scenes
        {"name": "net_train_32_batch8", "kind": "net_train", "nx": 32, "ny": 32, "nz": 32, "count": 8},
    ]


def _extent(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same ranges: steps most often, as in use."""
    kind = rng.choice(["step", "step", "step", "step", "step", "obstacle", "solve", "batch", "net_apply", "net_train"])
    boundary = rng.choice(["closed", "plume"])
    if kind == "step":
        solver = rng.choice(["fixed", "fixed", "multigrid", "multigrid", "jacobi", "learned"])
        mode = rng.choice(["linear", "cubic"])
        lo, hi = (96, 256) if mode == "cubic" else (24, 256)
        if solver == "jacobi":
            lo, hi, mode = 24, 72, "linear"
        elif solver == "learned":
            lo, hi = max(lo, 64), 192
        nx, ny, nz = (_extent(rng, lo, hi) for _ in range(3))
        while nx * ny * nz > 200 ** 3:
            nx, ny, nz = (max(lo, 7 * v // 8) for v in (nx, ny, nz))
        solids = rng.random() < 0.5
        case = _step("", nx, ny, nz, solver, mode, boundary, solids, rng.choice(["velocity", "all"]))
        del case["name"]
        return case
    if kind == "obstacle":
        nx, ny, nz = (_extent(rng, 40, 144) for _ in range(3))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "solver": "multigrid", "mode": "linear", "boundary": boundary, "radius": round(rng.uniform(0.08, 0.16) * min(nx, ny, nz), 2)}
    if kind == "solve":
        nx, ny, nz = (_extent(rng, 32, 208) for _ in range(3))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "solver": rng.choice(["multigrid_cold", "fixed"]), "mode": "linear", "boundary": boundary, "solids": rng.random() < 0.5}
    if kind == "batch":
        low = rng.randint(32, 64)
        return {"kind": kind, "count": rng.randint(2, 12), "low": low, "high": rng.randint(low + 8, 112), "solver": "multigrid", "mode": "linear", "boundary": boundary}
    if kind == "net_apply":
        nx, ny, nz = (_extent(rng, 16, 128) for _ in range(3))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz}
    nx, ny, nz = (_extent(rng, 16, 48) for _ in range(3))
    return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "count": rng.randint(1, 8)}


# ------------------------------------------------------------------------------------------------ scenes from a seed
def _config(case):
    mode = abi.MONOTONIC_CUBIC if case["mode"] == "cubic" else abi.LINEAR
    if case["boundary"] == "plume":  # periodic x and z, no-slip floor, outflow top (the reference benchmark's scene)
        flow = {"x_minus": abi.PERIODIC, "x_plus": abi.PERIODIC, "y_plus": (abi.OUTFLOW, 0.0, 0.0, 0.0, 0.0), "z_minus": abi.PERIODIC, "z_plus": abi.PERIODIC}
        scalar = {"x_minus": abi.SCALAR_PERIODIC, "x_plus": abi.SCALAR_PERIODIC, "y_minus": (abi.FIXED_VALUE, 0.0), "y_plus": (abi.FIXED_VALUE, 0.0), "z_minus": abi.SCALAR_PERIODIC, "z_plus": abi.SCALAR_PERIODIC}
    else:
        flow, scalar = {}, {}
    return abi.make_config(case["nx"], case["ny"], case["nz"], cell_size=1.0 / case["nx"], dt=0.01, pressure_iterations=64, mode=mode, flow=flow, density=scalar, temperature=scalar)


def _axes(shape, offset, device):
    """Coordinates of a field's points over the extents, broadcastable, in [0, 1] (offset 0.5 for cell centres)."""
    out = []
    for a in range(3):
        n, o = shape[a], offset[a]
        cells = n - (1 if o == 0.0 else 0)
        view = [1, 1, 1]
        view[a] = n
        out.append(((torch.arange(n, device=device, dtype=torch.float64) + o) / cells).reshape(view))
    return out


def _puff(shape, rng, device, cy, amplitude):
    z, y, x = _axes(shape, (0.5, 0.5, 0.5), device)
    cx, cz = 0.5 + 0.1 * rng.uniform(-1, 1), 0.5 + 0.1 * rng.uniform(-1, 1)
    s = 0.17 + 0.03 * rng.uniform(0, 1)
    return (amplitude * torch.exp(-0.5 * ((x - cx) ** 2 + (y - cy) ** 2 + (z - cz) ** 2) / (s * s))).float()


def _modes(shape, offset, rng, device, amplitude):
    z, y, x = _axes(shape, offset, device)
    f = torch.zeros(shape, device=device, dtype=torch.float64)
    for _ in range(4):
        k = rng.integers(-1, 2, 3)
        f += rng.uniform(0.3, 1.0) * torch.sin(2 * math.pi * (k[0] * x + k[1] * y + k[2] * z) + rng.uniform(0, 2 * math.pi))
    return (amplitude * 0.5 * f).float()


def _sphere(shape, centre, radius, device):
    z, y, x = (torch.arange(n, device=device, dtype=torch.float64) + 0.5 for n in shape)
    d2 = (x[None, None, :] - centre[0]) ** 2 + (y[None, :, None] - centre[1]) ** 2 + (z[:, None, None] - centre[2]) ** 2
    return (d2 <= radius * radius).to(torch.uint8)


def _scene(case, seed, device="cuda"):
    """The scene's fields as device tensors."""
    cfg = _config(case)
    rng = np.random.default_rng(int(seed))
    shape = abi.cell_shape(cfg)
    su, sv, sw = abi.face_shapes(cfg)
    amplitude = 1.0 * cfg.cell_size / cfg.dt  # about one cell per step
    f = {
        "u": _modes(su, (0.5, 0.5, 0.0), rng, device, amplitude),
        "v": _modes(sv, (0.5, 0.0, 0.5), rng, device, amplitude),
        "w": _modes(sw, (0.0, 0.5, 0.5), rng, device, amplitude),
        "density": _puff(shape, rng, device, 0.4, 1.0),
        "temperature": _puff(shape, rng, device, 0.35, 1.0),
        "density_source": _puff(shape, rng, device, 0.15, 0.5),
        "temperature_source": _puff(shape, rng, device, 0.15, 0.5),
    }
    if case["boundary"] == "closed":
        for k in ("density_source", "temperature_source"):
            f[k] = f[k] - torch.flip(f[k], (1,))
    nz, ny, nx = shape
    f["occupancy"] = []
    if case["kind"] == "obstacle":  # a sphere rising by about a cell a frame, and its velocity
        r, x0, z0 = case["radius"], nx * rng.uniform(0.4, 0.6), nz * rng.uniform(0.4, 0.6)
        f["occupancy"] = [_sphere(shape, (x0, 0.45 * ny + k, z0), r, device) for k in range(OBSTACLE_FRAMES)]
        f["solid_velocity_y"] = torch.full(shape, cfg.cell_size / cfg.dt, device=device)
    elif case.get("solids"):
        occ = _sphere(shape, (nx * rng.uniform(0.45, 0.55), 0.45 * ny, nz * rng.uniform(0.45, 0.55)), 0.155 * min(nx, ny, nz), device)
        occ |= _sphere(shape, (nx * 0.2, ny * rng.uniform(0.6, 0.8), nz * 0.7), 0.06 * min(nx, ny, nz), device)
        f["occupancy"] = [occ]
    return cfg, f


class Outputs(dict):
    """A pass's results, most of them views of the context's own buffers: they keep its owner alive."""

    def __init__(self, owner, values):
        super().__init__(values)
        self.owner = owner


_stream = None


def _program_stream():
    """The program's simulation stream: every context's work runs on it in order, as the successive frames of one scene
    do (a frame needs the one before it), so that a pass's time is a frame's and not a share of several at once."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


class Scene:
    """A context with its fields loaded; closed with the object."""

    sim = None

    def __init__(self, case, seed):
        self.case = case
        self.cfg, f = _scene(case, seed)
        self.fields = f  # device inputs stay alive while the context may read them
        self.stream = _program_stream()
        self.frame = 0
        self.net = None
        sim = self.sim = smoke_b200.Simulation(smoke_b200.SmokeLibrary(), self.cfg, self.stream)
        self.stream.wait_stream(torch.cuda.current_stream())
        sim.update_density(f["density"])
        sim.update_temperature(f["temperature"])
        sim.update_density_source(f["density_source"])
        sim.update_temperature_source(f["temperature_source"])
        sim.set_face_velocity(f["u"], f["v"], f["w"])
        if f["occupancy"]:
            sim.update_occupancy(f["occupancy"][0])
        if "solid_velocity_y" in f:
            sim.update_solid_velocity(None, f["solid_velocity_y"], None)
        if case["solver"] == "learned":
            self.net = smoke_b200.Net(sim.L)
            self.net.set_parameters(np.fromfile(WEIGHTS, np.float32))
            sim.set_preconditioner_net(self.net)
            sim.set_learned_iterations(1)
        if SOLVERS[case["solver"]]:
            sim.set_solver(**SOLVERS[case["solver"]])

    def outputs(self, views):
        sim = self.sim
        out = {"density": sim.view(abi.VIEW_DENSITY), "temperature": sim.view(abi.VIEW_TEMPERATURE), "pressure": sim.view(abi.VIEW_FLOW_PRESSURE), "velocity": sim.view(abi.VIEW_FLOW_VELOCITY), "face": sim.face_velocity()}
        if views == "all":
            out |= {"speed": sim.view(abi.VIEW_FLOW_VELOCITY_MAGNITUDE), "vorticity": sim.view(abi.VIEW_FLOW_VORTICITY), "swirl": sim.view(abi.VIEW_FLOW_VORTICITY_MAGNITUDE)}
        return Outputs(self, out)

    def __del__(self):
        if self.net is not None:
            self.net.close()
        if self.sim is not None:
            self.sim.close()


class Scenes:
    """Scenes advanced by one batch; the batch is closed before its members."""

    batch = None

    def __init__(self, cases, seed):
        self.members = [Scene(c, seed + 7919 * i) for i, c in enumerate(cases)]
        self.batch = smoke_b200.Batch([m.sim for m in self.members], _program_stream())

    def __del__(self):
        if self.batch is not None:
            self.batch.close()


def _batch_cases(case):
    """The members' cases: extents spread over [low, high], one in three with an obstacle."""
    out = []
    for i in range(case["count"]):
        e = [case["low"] + (case["high"] - case["low"]) * ((13 * i + 5 * a) % 17) // 16 for a in range(3)]
        out.append({"kind": "step", "nx": e[0], "ny": e[1], "nz": e[2], "solver": case["solver"], "mode": case["mode"], "boundary": case["boundary"], "solids": i % 3 == 2})
    return out


def _net_inputs(case, seed, device="cuda"):
    """Multi-scale residuals, a solid sphere and (training) smooth targets, as the training program makes them."""
    g = torch.Generator(device=device).manual_seed(int(seed))
    count, shape = case.get("count", 1), (case["nz"], case["ny"], case["nx"])

    def field():
        f = torch.zeros((count, 1) + shape, device=device)
        for level, a in ((2, 1.0), (1, 0.5), (0, 0.1)):
            c = [max(2, -(-v >> level)) for v in shape]
            f += a * torch.nn.functional.interpolate(torch.randn([count, 1] + c, generator=g, device=device), size=shape, mode="trilinear", align_corners=True)
        return f[:, 0].contiguous()

    rhs, target = field(), field()
    nz, ny, nx = shape
    occ = torch.stack([_sphere(shape, (nx * (0.3 + 0.05 * i), ny * 0.6, nz * 0.5), 0.15 * min(shape), device) for i in range(count)])
    return rhs, occ, target


def _net_parameters():
    return np.fromfile(WEIGHTS, np.float32)


# ------------------------------------------------------------------------------------------------ the calls
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step", "obstacle", "solve"):
        scene = Scene(case, seed)
        if kind == "solve":  # the stages up to the pressure solve leave the right-hand side that the call solves
            scene.sim.step_stages(abi.STAGE_PRESSURE)
        return {"case": case, "scene": scene}
    if kind == "batch":
        return {"case": case, "scenes": Scenes(_batch_cases(case), seed)}
    net = smoke_b200.Net(smoke_b200.SmokeLibrary())
    net.set_parameters(_net_parameters())
    rhs, occ, target = _net_inputs(case, seed)
    return {"case": case, "net": NetHolder(net), "rhs": rhs, "occ": occ, "target": target}


class NetHolder:
    def __init__(self, net):
        self.net = net

    def __del__(self):
        self.net.close()


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        scene = state["scene"]
        scene.sim.step()
        return scene.outputs(case["views"])
    if kind == "obstacle":
        scene = state["scene"]
        scene.sim.update_occupancy(scene.fields["occupancy"][scene.frame % OBSTACLE_FRAMES])
        scene.frame += 1
        scene.sim.step()
        return scene.outputs("velocity")
    if kind == "solve":
        scene = state["scene"]
        scene.sim.solve_pressure()
        return Outputs(scene, {"pressure": scene.sim.view(abi.VIEW_FLOW_PRESSURE)})
    if kind == "batch":
        scenes = state["scenes"]
        scenes.batch.step()
        members = [{"density": m.sim.view(abi.VIEW_DENSITY), "pressure": m.sim.view(abi.VIEW_FLOW_PRESSURE), "face": m.sim.face_velocity()} for m in scenes.members]
        return Outputs(scenes, {"members": members})
    net = state["net"].net
    if kind == "net_apply":
        return {"out": net.apply(state["rhs"][0], state["occ"][0])}
    loss = net.train_step(state["rhs"], state["occ"], state["target"], LEARNING_RATE)
    return {"loss": loss, "parameters": net.parameters()}


# ------------------------------------------------------------------------------------------------ least work
NET_LAYERS = [(2, 16, 0), (16, 32, 1), (32, 64, 2), (64, 128, 3), (128, 64, 3), (64, 32, 2), (32, 16, 1), (16, 1, 0)]


def _net_flops(case):
    """Multiply-adds of one forward evaluation, as 2 operations each."""
    n, total = [case["nz"], case["ny"], case["nx"]], 0
    levels = []
    for _ in range(4):
        levels.append(n[0] * n[1] * n[2])
        n = [(v + 1) // 2 for v in n]
    for ci, co, level in NET_LAYERS:
        total += 2 * 27 * ci * co * levels[level]
    return total


def _step_work(case):
    """One frame: fields in (3 face components, 2 scalars, 2 sources, 3 forces, occupancy) and out (3 face components, 2
    scalars, pressure, the views), each once; operations of the stages (about 900 a cell, cubic 2500) and of the solve: per
    iteration a 7-point operator, three updates and two dot products (about 24), a multigrid cycle five times that."""
    cells = case["nx"] * case["ny"] * case["nz"]
    views = {"velocity": 3, "all": 8}.get(case.get("views", "velocity"))
    iterations = {"fixed": 64 * 24, "jacobi": 150 * 24, "multigrid": 8 * 120, "multigrid_cold": 14 * 120, "learned": 9 * 120}[case["solver"]]
    return {"bytes": cells * (4 * 10 + 1 + 4 * 6 + 4 * views), "flops": cells * ((2500 if case["mode"] == "cubic" else 900) + iterations)}


def work(case):
    kind = case["kind"]
    if kind in ("step", "obstacle"):
        return _step_work(case)
    if kind == "solve":
        cells = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": cells * 9, "flops": cells * {"fixed": 64 * 24, "multigrid_cold": 14 * 120}[case["solver"]]}
    if kind == "batch":
        each = [_step_work(c) for c in _batch_cases(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    cells = case["nx"] * case["ny"] * case["nz"]
    parameters = sum(27 * ci * co + co for ci, co, _ in NET_LAYERS)
    if kind == "net_apply":
        return {"bytes": cells * 9 + 2 * parameters, "flops": _net_flops(case)}
    return {"bytes": case["count"] * cells * 9 + 28 * parameters, "flops": 3 * case["count"] * _net_flops(case)}


# ------------------------------------------------------------------------------------------------ 64-bit restatement
class Exact:
    """One step of a scene of this file in torch float64 (the boundary kinds of _config, walls and obstacles)."""

    def __init__(self, case, seed):
        self.case = case
        self.cfg, f = _scene(case, seed)
        c = self.cfg
        self.h, self.dt = float(c.cell_size), float(c.dt)
        self.n = (c.nz, c.ny, c.nx)
        plume = case["boundary"] == "plume"
        self.per = (plume, False, plume)  # z, y, x
        self.out_top = plume
        self.f = {k: v.double() for k, v in f.items() if k != "occupancy"}
        self.occ = f["occupancy"][0].bool() if f["occupancy"] else torch.zeros(self.n, dtype=torch.bool, device="cuda")
        self.solids = bool(f["occupancy"])
        self.solid_v = [torch.zeros(self.n, device="cuda", dtype=torch.float64) for _ in range(3)]  # by tensor axis
        if "solid_velocity_y" in f:
            self.solid_v[1] = f["solid_velocity_y"].double()

    # ---- neighbours along tensor axis a: the value at index + d, `wall` applied beyond a non-periodic end
    def shift(self, x, a, d, lo, hi):
        y = torch.roll(x, -d, a)
        if not self.per[a]:
            n = x.shape[a]
            if d > 0:
                y.narrow(a, n - 1, 1).copy_(hi(x.narrow(a, n - 1, 1)))
            else:
                y.narrow(a, 0, 1).copy_(lo(x.narrow(a, 0, 1)))
        return y

    def pad(self, f, axis, scalar, p):
        """The field with p ghost cells a side: boundary taps resolved in x, y, z order (faces: walls mirror with the sign
        changed, the outflow top copies, and coordinates after the one that met a wall clamp; scalars: walls of a closed
        box copy, fixed faces hold 0). axis: the face component's tensor axis, None for cells."""
        idx, beyond = [], []
        for a in range(3):
            size = f.shape[a]
            i = torch.arange(-p, size + p, device=f.device)
            out = (i < 0) | (i >= size)
            view = [1, 1, 1]
            view[a] = -1
            wrapped = torch.where(out, i % self.n[a], i)
            idx.append((wrapped.reshape(view), i.clamp(0, size - 1).reshape(view)))
            beyond.append((out & (not self.per[a])).reshape(view))
        sign = torch.ones((1, 1, 1), device=f.device, dtype=torch.float64)
        met = torch.zeros((1, 1, 1), device=f.device, dtype=torch.bool)
        use = [None] * 3
        for a in (2, 1, 0):  # x, y, z
            clamp = beyond[a] if scalar else (met | beyond[a])
            use[a] = torch.where(clamp, idx[a][1], idx[a][0])
            if scalar:
                s = 0.0 if (self.case["boundary"] == "plume" and a == 1) else 1.0
                sign = torch.where(beyond[a], sign * s, sign)
            else:
                first = beyond[a] & ~met
                s = torch.full(beyond[a].shape, -1.0, device=f.device, dtype=torch.float64)
                if a == 1 and self.out_top:
                    s[:, p + f.shape[1]:, :] = 1.0
                sign = torch.where(first, s, sign)
                met = met | beyond[a]
        shape = [s + 2 * p for s in f.shape]
        lin = ((use[0] * f.shape[1] + use[1]) * f.shape[2] + use[2]).expand(shape)
        return f.reshape(-1)[lin] * sign

    @staticmethod
    def cubic(p0, p1, p2, p3, t):
        d, m1, m2 = p2 - p1, 0.5 * (p2 - p0), 0.5 * (p3 - p1)
        flat = d.abs() < 1e-6
        m1 = torch.where(flat | (m1 * d <= 0), 0.0, m1)
        m2 = torch.where(flat | (m2 * d <= 0), 0.0, m2)
        t2, t3 = t * t, t * t * t
        return (2 * t3 - 3 * t2 + 1) * p1 + (t3 - 2 * t2 + t) * m1 + (3 * t2 - 2 * t3) * p2 + (t3 - t2) * m2

    def sample(self, padded, p, axis, pos, cubic):
        """padded: pad(f); pos: (z, y, x) world positions, any shape."""
        lo, t = [], []
        for a in range(3):
            x = pos[a]
            if self.per[a]:
                x = torch.remainder(x, self.n[a] * self.h)
            g = x / self.h - (0.0 if axis == a else 0.5)
            i = torch.floor(g)
            t.append(g - i)
            r = 1 if cubic else 0
            lo.append((i.long() + (p - r)).clamp(0, padded.shape[a] - 2 - 2 * r))
        sy, sz = padded.shape[2], padded.shape[1] * padded.shape[2]
        base, flat = lo[0] * sz + lo[1] * sy + lo[2], padded.reshape(-1)
        taps = 4 if cubic else 2
        line = []
        for k in range(taps):
            rows = []
            for j in range(taps):
                v = [flat[base + (k * sz + j * sy + i)] for i in range(taps)]
                rows.append(self.cubic(*v, t[2]) if cubic else v[0] + (v[1] - v[0]) * t[2])
            line.append(self.cubic(*rows, t[1]) if cubic else rows[0] + (rows[1] - rows[0]) * t[1])
        return self.cubic(*line, t[0]) if cubic else line[0] + (line[1] - line[0]) * t[0]

    def blocked(self, pos):
        bad, idx = None, []
        for a in range(3):
            x = torch.remainder(pos[a], self.n[a] * self.h) if self.per[a] else pos[a]
            out = (x < 0) | (x > self.n[a] * self.h)
            bad = out if bad is None else bad | out
            idx.append(torch.floor(x / self.h).long().clamp(0, self.n[a] - 1))
        if self.solids:
            bad = bad | self.occ.reshape(-1)[(idx[0] * self.n[1] + idx[1]) * self.n[2] + idx[2]]
        return bad

    def trace(self, start, padded, p):
        vel = [self.sample(padded[a], p, a, start, False) for a in range(3)]
        mid = [start[a] - 0.5 * self.dt * vel[a] for a in range(3)]
        vel = [self.sample(padded[a], p, a, mid, False) for a in range(3)]
        end = [start[a] - self.dt * vel[a] for a in range(3)]
        bad = self.blocked(end).reshape(-1).nonzero()[:, 0]
        if bad.numel():
            s = [start[a].expand(end[a].shape).reshape(-1)[bad] for a in range(3)]
            e = [end[a].reshape(-1)[bad] for a in range(3)]
            low, high = torch.zeros_like(s[0]), torch.ones_like(s[0])
            for _ in range(10):
                m = 0.5 * (low + high)
                b = self.blocked([s[a] + (e[a] - s[a]) * m for a in range(3)])
                low, high = torch.where(b, low, m), torch.where(b, m, high)
            for a in range(3):
                end[a] = end[a].reshape(-1).index_put((bad,), s[a] + (e[a] - s[a]) * low).reshape(end[a].shape)
        return end

    def settle(self, x, a, outflow_sees_solid):
        """The face rules on x (a face component's stage values): solid faces, walls, the outflow copy, the periodic twin."""
        n = self.n[a]
        raw = x
        if self.solids:
            o, sv = self.occ.double(), self.solid_v[a]
            edge = [o.narrow(a, n - 1, 1), o.narrow(a, 0, 1)]
            ev = [(o * sv).narrow(a, n - 1, 1), (o * sv).narrow(a, 0, 1)]
            left, right = torch.cat([edge[0], o], a), torch.cat([o, edge[1]], a)
            lv, rv = torch.cat([ev[0], o * sv], a), torch.cat([o * sv, ev[1]], a)
            weight = left + right
            x = torch.where(weight > 0, (lv + rv) / weight.clamp(min=1.0), x)
        if x is raw:
            x = x.clone()
        if self.per[a]:
            x.narrow(a, n, 1).copy_(x.narrow(a, 0, 1))
        else:
            x.narrow(a, 0, 1).zero_()
            if a == 1 and self.out_top:
                x.narrow(a, n, 1).copy_((x if outflow_sees_solid else raw).narrow(a, n - 1, 1))
            else:
                x.narrow(a, n, 1).zero_()
        return x

    def centre(self, faces):
        return [0.5 * (faces[a].narrow(a, 0, self.n[a]) + faces[a].narrow(a, 1, self.n[a])) for a in range(3)]

    def curl(self, faces):
        c = self.centre(faces)

        def diff(comp, a):  # central difference of component comp along axis a, walls mirrored, outflow top copied
            neg, same = (lambda v: -v), (lambda v: v)
            return (self.shift(c[comp], a, 1, neg, same if (a == 1 and self.out_top) else neg) - self.shift(c[comp], a, -1, neg, neg)) * (0.5 / self.h)

        # tensor axes: 0 = z, 1 = y, 2 = x
        w = [diff(1, 2) - diff(2, 1), diff(2, 0) - diff(0, 2), diff(0, 1) - diff(1, 0)]  # z, y, x components
        if self.solids:
            w = [torch.where(self.occ, 0.0, v) for v in w]
        return w, torch.sqrt(w[0] ** 2 + w[1] ** 2 + w[2] ** 2)

    # ---- pressure
    def system(self):
        anchor = int((~self.occ).reshape(-1).long().argmax())
        act = ~self.occ
        act.view(-1)[anchor] = False
        self.act = act
        diag = torch.zeros(self.n, device="cuda", dtype=torch.float64)
        fluid = (~self.occ).double()
        zero = (lambda v: torch.zeros_like(v))
        for a in range(3):
            diag += self.shift(fluid, a, 1, zero, (lambda v: torch.ones_like(v)) if (a == 1 and self.out_top) else zero) + self.shift(fluid, a, -1, zero, zero)
        self.diag = diag.clamp(min=1.0)
        self.m = act.double()

    def apply(self, x):  # x is 0 on inactive cells
        y = self.diag * x
        zero = (lambda v: torch.zeros_like(v))
        for a in range(3):
            y -= self.shift(x, a, 1, zero, zero)
            y -= self.shift(x, a, -1, zero, zero)
        return y * self.m

    def solve(self, b, fixed=None):
        self.system()
        b = b * self.m
        x, r = torch.zeros_like(b), b.clone()
        if fixed is not None:  # plain CG, exactly `fixed` iterations
            p, rr = r.clone(), (r * r).sum()
            for _ in range(fixed):
                q = self.apply(p)
                pq = (p * q).sum()
                alpha = torch.where(pq.abs() > 1e-20, rr / pq, 0.0)
                x, r = x + alpha * p, r - alpha * q
                rn = (r * r).sum()
                p = r + torch.where(rr.abs() > 1e-20, rn / rr, 0.0) * p
                rr = rn
            return x
        # CG preconditioned by the box without obstacles, diagonalised axis by axis
        eig = []
        for a in range(3):
            n = self.n[a]
            t = 2 * torch.eye(n, device="cuda", dtype=torch.float64) - torch.diag(torch.ones(n - 1, device="cuda", dtype=torch.float64), 1) - torch.diag(torch.ones(n - 1, device="cuda", dtype=torch.float64), -1)
            if self.per[a]:
                t[0, n - 1] -= 1
                t[n - 1, 0] -= 1
            else:
                t[0, 0] = 1
                t[n - 1, n - 1] = 2 if (a == 1 and self.out_top) else 1
            eig.append(torch.linalg.eigh(t))
        lam = eig[0][0][:, None, None] + eig[1][0][None, :, None] + eig[2][0][None, None, :]
        lam = torch.where(lam < 1e-9, lam.reshape(-1).sort().values[1], lam)

        def precondition(v):
            for a, e in enumerate((eig[0][1], eig[1][1], eig[2][1])):
                v = torch.tensordot(v, e, ([a], [0])).movedim(-1, a)
            v = v / lam
            for a, e in enumerate((eig[0][1], eig[1][1], eig[2][1])):
                v = torch.tensordot(v, e, ([a], [1])).movedim(-1, a)
            return v * self.m

        z = precondition(r)
        p, rz, target = z.clone(), (r * z).sum(), 1e-22 * (b * b).sum()
        for _ in range(400):
            q = self.apply(p)
            alpha = rz / (p * q).sum()
            x, r = x + alpha * p, r - alpha * q
            if bool((r * r).sum() <= target):
                break
            z = precondition(r)
            rn = (r * z).sum()
            p, rz = z + (rn / rz) * p, rn
        return x

    def fill(self, d):
        """Solid cells take the density of their nearest fluid cell: the first Chebyshev shell with one, the smallest
        distance in it, the first in (z, y, x) order."""
        solid = self.occ
        if not self.solids or not bool(solid.any()):
            return d
        per = self.per if self.case["boundary"] == "plume" else (False, False, False)
        left, depth = solid.clone(), 0
        idx = solid.nonzero()
        depth_of = torch.zeros(idx.shape[0], dtype=torch.long, device=d.device)
        reach = ~solid
        while bool(left.any()):
            depth += 1
            for a in range(3):
                grown = reach.clone()
                for s in (1, -1):
                    m = torch.roll(reach, s, a)
                    if not per[a]:
                        m.narrow(a, 0 if s > 0 else self.n[a] - 1, 1).fill_(False)
                    grown |= m
                reach = grown
            now = left & reach
            depth_of[now[idx[:, 0], idx[:, 1], idx[:, 2]]] = depth
            left &= ~reach
        out = torch.where(solid, 0.0, d)
        size = torch.tensor(self.n, device=d.device)
        for r in range(1, depth + 1):
            cells = idx[depth_of == r]
            g = torch.arange(-r, r + 1, device=d.device)
            off = torch.cartesian_prod(g, g, g)
            off = off[off.abs().amax(1) == r]
            d2 = (off * off).sum(1)
            order = torch.arange(off.shape[0], device=d.device)
            for part in cells.split(max(1, 20_000_000 // off.shape[0])):
                q = part[:, None, :] + off[None]
                ok = torch.ones(q.shape[:2], dtype=torch.bool, device=d.device)
                for a in range(3):
                    if not per[a]:
                        ok &= (q[..., a] >= 0) & (q[..., a] < self.n[a])
                q %= size
                lin = (q[..., 0] * self.n[1] + q[..., 1]) * self.n[2] + q[..., 2]
                ok &= ~solid.reshape(-1)[lin]
                key = torch.where(ok, d2[None] * off.shape[0] + order[None], 1 << 60)
                best = key.argmin(1)
                src = lin.gather(1, best[:, None])[:, 0]
                out[part[:, 0], part[:, 1], part[:, 2]] = d.reshape(-1)[src]
        return out

    def run(self, through_solve=False):
        f, c, h, dt, n = self.f, self.cfg, self.h, self.dt, self.n
        cubic = self.case["mode"] == "cubic"
        A = [f["w"], f["v"], f["u"]]  # by tensor axis
        # forces
        w, wm = self.curl(A)
        same = (lambda v: v)
        g = [(self.shift(wm, a, 1, same, same) - self.shift(wm, a, -1, same, same)) * (0.5 / h) for a in range(3)]
        gm = torch.sqrt(g[0] ** 2 + g[1] ** 2 + g[2] ** 2)
        N = [torch.where(gm < 1e-6, 0.0, v / gm.clamp(min=1e-30)) for v in g]
        k = float(c.vorticity_confinement) * h
        force = [k * (N[2] * w[1] - N[1] * w[2]), k * (N[0] * w[2] - N[2] * w[0]), k * (N[1] * w[0] - N[0] * w[1])]
        force[1] = force[1] - float(c.buoyancy_density_factor) * f["density"] + float(c.buoyancy_temperature_factor) * (f["temperature"] - float(c.ambient_temperature))
        if self.solids:
            force = [torch.where(self.occ, 0.0, v) for v in force]
        B = []
        for a in range(3):
            x = A[a].clone()
            x.narrow(a, 1, n[a] - 1).add_(0.5 * dt * (force[a].narrow(a, 0, n[a] - 1) + force[a].narrow(a, 1, n[a] - 1)))
            x.narrow(a, 0, 1).add_(dt * force[a].narrow(a, 0, 1))
            B.append(self.settle(x, a, False))
        del w, wm, g, gm, N, force
        # velocity advection
        p = 6
        padded = [self.pad(B[a], a, False, p) for a in range(3)]
        C = []
        for a in range(3):
            start = []
            for b in range(3):
                view = [1, 1, 1]
                view[b] = -1
                size = n[b] + (1 if a == b else 0)
                i = torch.arange(size, device="cuda", dtype=torch.float64)
                if a == b and self.per[a]:
                    i[n[b]] = 0.0
                start.append(((i + (0.0 if a == b else 0.5)) * h).reshape(view).expand([n[d] + (1 if a == d else 0) for d in range(3)]))
            C.append(self.settle(self.sample(padded[a], p, a, self.trace(start, padded, p), cubic), a, False))
        del padded
        # pressure and projection
        div = sum(C[a].narrow(a, 1, n[a]) - C[a].narrow(a, 0, n[a]) for a in range(3)) / h
        pressure = self.solve(-(h * h / dt) * div, int(c.pressure_iterations) if self.case["solver"] == "fixed" else None)
        if through_solve:
            return {"pressure": pressure}
        V = []
        for a in range(3):
            x = C[a].clone()
            x.narrow(a, 1, n[a] - 1).sub_(dt / h * (pressure.narrow(a, 1, n[a] - 1) - pressure.narrow(a, 0, n[a] - 1)))
            if self.per[a]:
                x.narrow(a, 0, 1).sub_(dt / h * (pressure.narrow(a, 0, 1) - pressure.narrow(a, n[a] - 1, 1)))
            V.append(self.settle(x, a, True))
        # scalars
        t = (torch.where(self.occ, float(c.ambient_temperature), f["temperature"])) + dt * f["temperature_source"]
        d = f["density"] + dt * f["density_source"]
        padded = [self.pad(V[a], a, False, p) for a in range(3)]
        start = []
        for b in range(3):
            view = [1, 1, 1]
            view[b] = -1
            start.append(((torch.arange(n[b], device="cuda", dtype=torch.float64) + 0.5) * h).reshape(view).expand(n))
        end = self.trace(start, padded, p)
        t = self.sample(self.pad(t, None, True, p), p, None, end, cubic)
        d = self.sample(self.pad(d, None, True, p), p, None, end, cubic)
        t = torch.where(self.occ, float(c.ambient_temperature), t)
        d = self.fill(d)
        centre = self.centre(V)
        out = {"density": d, "temperature": t, "pressure": pressure, "velocity": tuple(centre[::-1]), "face": tuple(V[::-1])}
        if self.case.get("views") == "all":
            w, wm = self.curl(V)
            out |= {"speed": torch.sqrt(sum(v * v for v in centre)), "vorticity": tuple(w[::-1]), "swirl": wm}
        return out


def _net_exact(parameters, rhs, occ):
    """The network on one volume in float64: (output before the scale and the mask, the scale, fluid)."""
    import torch.nn.functional as F

    weights, o = [], 0
    for ci, co, _ in NET_LAYERS:
        w = parameters[o:o + 27 * ci * co].reshape(3, 3, 3, ci, co).permute(4, 3, 0, 1, 2)
        o += 27 * ci * co
        weights.append((w, parameters[o:o + co]))
        o += co
    fluid = (occ == 0).double()
    s = torch.sqrt(rhs.numel() / (rhs * rhs).sum())
    conv = (lambda i, x: F.conv3d(x, weights[i][0], weights[i][1], padding=1))
    pool = (lambda x: F.avg_pool3d(x, 2, ceil_mode=True, count_include_pad=False))

    def up(x, like):
        for a in (2, 3, 4):
            x = x.repeat_interleave(2, a).narrow(a, 0, like.shape[a])
        return x + like

    x0 = torch.stack([rhs * s, fluid])[None]
    e0 = conv(0, x0).relu()
    e1 = conv(1, pool(e0)).relu()
    e2 = conv(2, pool(e1)).relu()
    m3 = conv(4, conv(3, pool(e2)).relu()).relu()
    u2 = conv(5, up(m3, e2)).relu()
    u1 = conv(6, up(u2, e1)).relu()
    return conv(7, up(u1, e0))[0, 0], s, fluid


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "obstacle"):
        return Exact(case, seed).run()
    if kind == "solve":
        return Exact(case, seed).run(through_solve=True)
    if kind == "batch":
        got = [Exact(c, seed + 7919 * i).run() for i, c in enumerate(_batch_cases(case))]
        return {"members": [{k: g[k] for k in ("density", "pressure", "face")} for g in got]}
    rhs, occ, target = _net_inputs(case, seed)
    parameters = torch.from_numpy(_net_parameters()).cuda().double()
    if kind == "net_apply":
        y, s, fluid = _net_exact(parameters, rhs[0].double(), occ[0])
        return {"out": fluid * y / s}
    # one Adam step on the mean relative loss
    parameters.requires_grad_(True)
    total = 0.0
    for i in range(case["count"]):
        t = target[i].double()
        y, s, fluid = _net_exact(parameters, rhs[i].double(), occ[i])
        loss = (fluid * (y - s * t) ** 2).sum() / (s * s * (fluid * t * t).sum()) / case["count"]
        loss.backward()
        total += float(loss.detach())
    g = parameters.grad
    new = parameters.detach() - LEARNING_RATE * g / (g.abs() + 1e-8)
    return {"loss": total, "parameters": new}
