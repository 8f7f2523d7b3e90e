"""What a user of this framework has it do, as cases that can be timed and compared.

A case is a dict of plain values. `kind` names the entry point it goes through:

  steps     GpuStepper: upload a scene, step it with the device's own dt, read u, v, p and dye back
  host      fl_step_host: one step of a caller that holds the whole state on the host
  sim       Simulation.step: the reference's host loop (float64 fields, host CFL), one step a pass
  batch     Batch.step: several closed boxes of different sides stepped together
  mg, rb    GpuMultigridSolver.solve, GpuPressureSolver.solve on one pressure problem
  advect    fl_advect_velocity_noalloc on the caller's own device buffers
  unet      Unet.forward, and Unet.train_step with the gradient, of the pressure warm start

Host fields of the steps are pinned, as the engine's copies want them. Every
pass of every kind but `sim` starts from the same inputs, so it gives the same
outputs; a `sim` goes on from where it is.
"""
import ctypes
import math

import numpy as np
import torch

from flowlab_gb300 import configs, engine, native, scenes as sc, warmstart

FLUID, AIR, SOLID = 0, 1, 2


def listed():
    return [
        # a vortex street in a browser-sized window: fixed red-black SOR, launches and latency
        {"name": "street_128", "kind": "steps", "scene": "street", "nx": 128, "ny": 128, "steps": 16},
        # an interactive thermal plume: multigrid to 1e-6 where every level is small
        {"name": "plume_256", "kind": "steps", "scene": "plume", "nx": 256, "ny": 256, "steps": 16},
        # the benchmark's own scene and size
        {"name": "plume_1024", "kind": "steps", "scene": "plume", "nx": 1024, "ny": 1024, "steps": 8},
        # the largest: the obstacle lattice to 1e-8 through the float64 defect correction
        {"name": "lattice_2048", "kind": "steps", "scene": "lattice", "nx": 2048, "ny": 2048, "steps": 2},
        # a host program that keeps the state itself and hands it over each step
        {"name": "host_plume_1024", "kind": "host", "scene": "plume", "nx": 1024, "ny": 1024},
        # the reference's loop with its default parameters on an odd grid, dye refined by two
        {"name": "sim_517x389", "kind": "sim", "nx": 517, "ny": 389, "dye_scale": 2, "scheme": "semiLagrangian"},
        # uneven scenes with obstacles, stepped as one batch
        {"name": "batch_12", "kind": "batch", "scenes": 12, "max_side": 512, "steps": 3, "worklist": True},
        # one pressure problem with obstacles and an open side, three V(2,2) cycles
        {"name": "mg_801x1203", "kind": "mg", "nx": 801, "ny": 1203, "cycles": 3, "pre": 2, "post": 2},
        # the reference's default solver budget: red-black SOR, a residual test every 12 sweeps
        {"name": "rb_640x480", "kind": "rb", "nx": 640, "ny": 480, "iterations": 100, "tol": 5e-3},
        # MacCormack velocity advection in a host's own device memory, ragged
        {"name": "advect_1001x750", "kind": "advect", "nx": 1001, "ny": 750, "mac": True},
        # the learned warm start: inference at the benchmark's size, a training batch with its gradient
        {"name": "unet_1024", "kind": "unet", "train": False, "batch": 1, "h": 1024, "w": 1024},
        {"name": "unet_train_4x256", "kind": "unet", "train": True, "batch": 4, "h": 256, "w": 256},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, lo, hi):
    """Two sides of a box up to 2.5 times as long as high, or as high as long."""
    nx = _log(rng, lo, hi)
    return {"nx": nx, "ny": min(hi, max(lo, _log(rng, nx / 2.5, nx * 2.5)))}


def draw(rng):
    kind = rng.choice(["street", "plume", "lattice", "host", "sim", "batch", "mg", "rb", "advect", "unet", "train"])
    if kind == "street":
        return {"kind": "steps", "scene": "street", **_sides(rng, 64, 400),
                "steps": rng.randint(4, 16)}
    if kind == "plume":
        return {"kind": "steps", "scene": "plume", **_sides(rng, 64, 1024),
                "steps": rng.randint(2, 8)}
    if kind == "lattice":
        return {"kind": "steps", "scene": "lattice", **_sides(rng, 256, 2048),
                "steps": rng.randint(1, 2)}
    if kind == "host":
        return {"kind": "host", "scene": rng.choice(["plume", "street"]), **_sides(rng, 64, 1024)}
    if kind == "sim":
        return {"kind": "sim", **_sides(rng, 64, 700), "dye_scale": rng.randint(1, 2),
                "scheme": rng.choice(["semiLagrangian", "macCormack"])}
    if kind == "batch":
        return {"kind": "batch", "scenes": rng.randint(4, 12), "max_side": rng.choice([64, 128, 256, 512]),
                "steps": rng.randint(1, 3), "worklist": rng.random() < 0.5}
    if kind == "mg":
        return {"kind": "mg", "nx": _log(rng, 64, 1500), "ny": _log(rng, 64, 1500), "cycles": rng.randint(1, 4),
                "pre": rng.randint(1, 3), "post": rng.randint(1, 3)}
    if kind == "rb":
        return {"kind": "rb", "nx": _log(rng, 64, 800), "ny": _log(rng, 64, 800), "iterations": rng.randint(20, 120),
                "tol": rng.choice([0.0, 5e-3])}
    if kind == "advect":
        return {"kind": "advect", "nx": _log(rng, 64, 1040), "ny": _log(rng, 64, 1040), "mac": rng.random() < 0.7}
    if kind == "unet":
        return {"kind": "unet", "train": False, "batch": 1, "h": 8 * _log(rng, 8, 128), "w": 8 * _log(rng, 8, 128)}
    return {"kind": "unet", "train": True, "batch": rng.randint(1, 4), "h": 8 * _log(rng, 8, 32),
            "w": 8 * _log(rng, 8, 32)}


# ------------------------------------------------------------------ inputs

def _pinned(a, dtype=np.float32):
    """`a` in page-locked host memory (a numpy view of it)."""
    t = torch.empty(int(np.size(a)), dtype=torch.from_numpy(np.empty(0, dtype)).dtype, pin_memory=True)
    t.numpy()[:] = np.ravel(a)
    return t.numpy()


def _scene(case, seed):
    """(grid, float64 fields, dye patch, engine parameters): the configurations' scenes on any
    grid, each with seeded 1e-3 noise on its interior faces."""
    nx, ny, scale = case["nx"], case["ny"], case.get("dye_scale", 1)
    g = sc.Grid(nx, ny, 1.0 / ny)
    dg = sc.dye_grid(g, scale)
    w = nx * g.h
    if case["scene"] == "plume":
        spec = sc.SceneSpec(seed=sc.draught(), dye_source=sc.gaussian_sources([(0.35 * w, 0.1), (0.65 * w, 0.1)]))
        prm = configs.plume_params()
    elif case["scene"] == "street":
        spec = sc.SceneSpec(labels=sc.all_labels(sc.open_right(), sc.solid_disk(0.25 * w, 0.5, 0.1 * min(w, 1.0))),
                            seed=sc.uniform_flow(1.0), dye=lambda d, q: sc.add_dye_stripes(d, q))
        prm = configs.karman_params()
    else:
        centres, side = configs.turbulence_lattice(ny)
        half = 0.5 * side * g.h
        rects = [sc.solid_rect(x * g.h - half, y * g.h - half, x * g.h + half, y * g.h + half)
                 for x, y in centres if x + side < nx - 1]
        spec = sc.SceneSpec(labels=sc.all_labels(sc.open_right(), *rects), seed=sc.uniform_flow(1.0),
                            dye=lambda d, q: sc.add_dye_stripes(d, q))
        prm = configs.turbulence_params()
    f, patch = sc.reset_fields(g, dg, spec)
    rng = np.random.default_rng([seed, nx, ny])
    f.u.reshape(ny, nx + 1)[:, 1:-1] += 1e-3 * (2 * rng.random((ny, nx - 1), np.float32) - 1)
    f.v.reshape(ny + 1, nx)[1:-1] += 1e-3 * (2 * rng.random((ny - 1, nx), np.float32) - 1)
    sc.commit_labels(g, f)
    return g, dg, f, patch, prm


def _boxes(case, seed):
    """The batch's scenes: sides in turn over the powers of two up to the largest."""
    sides = [s for s in (64, 128, 256, 512) if s <= case["max_side"]]
    return [configs.random_scene(sides[k % len(sides)], 1000 * seed + k)[:2] for k in range(case["scenes"])]


def _smooth(rng, ny, nx, cells):
    """A smooth random field of unit RMS: seeded values `cells` apart, interpolated."""
    a = torch.from_numpy(rng.standard_normal((1, 1, ny // cells + 3, nx // cells + 3)).astype(np.float32))
    q = torch.nn.functional.interpolate(a, size=(ny, nx), mode="bicubic", align_corners=True)[0, 0]
    return (q / q.square().mean().sqrt()).numpy()


def _obstacles(rng, ny, nx):
    """Labels with a solid block and a disc, an open right column."""
    label = np.zeros((ny, nx), np.uint8)
    label[ny // 4:ny // 2, nx // 4:(3 * nx) // 8] = SOLID
    cy, cx, r = ny * rng.uniform(0.6, 0.8), nx * rng.uniform(0.4, 0.7), 0.08 * min(nx, ny)
    jj, ii = np.ogrid[:ny, :nx]
    label[(jj - cy) ** 2 + (ii - cx) ** 2 < r * r] = SOLID
    label[:, -1] = AIR
    return label


def _problem(case, seed):
    """A pressure problem: the divergence of a smooth flow with noise, p zero, scale of a CFL-2 step."""
    nx, ny = case["nx"], case["ny"]
    rng = np.random.default_rng([seed, nx, ny])
    label = _obstacles(rng, ny, nx)
    div = (_smooth(rng, ny, nx, 16) + 0.1 * rng.standard_normal((ny, nx))).astype(np.float32)
    h = 1.0 / ny
    return sc.Grid(nx, ny, h), div.ravel(), label.ravel(), h * h / (2 * h)


def _flow(case, seed):
    """A smooth swirling velocity of speed about 1 with noise, obstacles, dt of CFL 2."""
    nx, ny = case["nx"], case["ny"]
    rng = np.random.default_rng([seed, nx, ny])
    label = _obstacles(rng, ny, nx)
    u = 0.7 * _smooth(rng, ny, nx + 1, 40) + 0.02 * rng.standard_normal((ny, nx + 1)).astype(np.float32)
    v = 0.7 * _smooth(rng, ny + 1, nx, 40) + 0.02 * rng.standard_normal((ny + 1, nx)).astype(np.float32)
    return u.astype(np.float32), v.astype(np.float32), label, 1.0 / ny, float(np.float32(2.0 / ny))


def _pairs(case, seed):
    """Warm-start training pairs: (b / s_b, mask, p_prev / s_p) and a smooth correction."""
    B, H, W = case["batch"], case["h"], case["w"]
    rng = np.random.default_rng([seed, H, W])
    x, t = np.empty((B, H, W, 3), np.float32), np.empty((B, H, W), np.float32)
    for k in range(B):
        m = (_obstacles(rng, H, W) == FLUID).astype(np.float32)
        x[k, ..., 0] = (_smooth(rng, H, W, 8) + 0.2 * rng.standard_normal((H, W))) * m
        x[k, ..., 1] = m
        x[k, ..., 2] = _smooth(rng, H, W, 32) * m
        t[k] = 0.05 * _smooth(rng, H, W, 16) * m
    return x, t, x[..., 1].copy()


class State:
    """The inputs and handles of one case; the engine objects are given back with it."""

    def __init__(self, case, seed):
        self.case = case
        self.open = []

    def own(self, x):
        self.open.append(x)
        return x

    def __del__(self):
        for x in reversed(self.open):
            (x.destroy if hasattr(x, "destroy") else x.close)()


def _fields32(g, dg, f):
    """Pinned float32 fields to hand over, and others of the same sizes to read into."""
    make = lambda: sc.Fields(*(_pinned(a) for a in (f.p, f.u, f.v)), _pinned(f.label, np.uint8), _pinned(f.dye))  # noqa: E731
    return make(), make()


def prepare(case, seed):
    s = State(case, seed)
    kind = case["kind"]
    ctx = engine.GpuContext(0)
    if kind in ("steps", "host"):
        g, dg, f, patch, prm = _scene(case, seed)
        s.f, s.out = _fields32(g, dg, f)
        s.stepper = s.own(engine.GpuStepper(ctx, g, dg, prm))
        s.stepper.set_dye_patch(patch)
        if kind == "host":
            P = native.ptr
            s.args = [native.FL_F32, P(s.f.u), P(s.f.v), P(s.f.p), P(s.f.label), P(s.f.dye), P(s.out.u), P(s.out.v),
                      P(s.out.p), P(s.out.dye), None]
    elif kind == "sim":
        g, dg, f, patch, _ = _scene(dict(case, scene="street"), seed)
        s.sim = engine.Simulation(case["nx"], case["ny"], {"scheme": case["scheme"]}, dye_scale=case["dye_scale"],
                                  ctx=ctx)
        s.own(s.sim.stepper)
        for name in ("u", "v", "p", "label", "dye"):
            getattr(s.sim.f, name)[:] = getattr(f, name)
        s.p = np.zeros_like(s.sim.f.p)
    elif kind == "batch":
        boxes = _boxes(case, seed)
        s.f = [_fields32(g, g, f) for g, f in boxes]
        prm = configs.random_scene_params(mixed=1)
        s.steppers = [s.own(engine.GpuStepper(ctx, g, None, prm)) for g, _ in boxes]
        for st, (f, _) in zip(s.steppers, s.f):
            st.upload(f)
        s.batch = s.own(native.Batch([st.eng for st in s.steppers]))
        if not case["worklist"]:
            s.batch.set_worklist(False)
    elif kind in ("mg", "rb"):
        g, s.div, s.label, s.scale = _problem(case, seed)
        s.g, s.p = g, np.zeros(case["nx"] * case["ny"], np.float32)
        if kind == "mg":
            s.solver = s.own(engine.GpuMultigridSolver(ctx, g, cycles=case["cycles"], pre=case["pre"],
                                                       post=case["post"]))
        else:
            s.solver = s.own(engine.GpuPressureSolver(ctx, g))
    elif kind == "advect":
        u, v, label, s.h, s.dt = _flow(case, seed)
        s.lib = native.load()
        s.u, s.v, s.label = (torch.from_numpy(a).cuda() for a in (u, v, label))
        s.uo, s.vo = torch.empty_like(s.u), torch.empty_like(s.v)
    else:
        s.x, s.t, s.m = (_pinned(a).reshape(a.shape) for a in _pairs(case, seed))
        s.net = s.own(native.Unet(case["batch"] * case["h"] * case["w"]))
        s.net.set_params(warmstart.load(warmstart.DEFAULT_WEIGHTS)[0])
    return s


def run(s):
    c = s.case
    kind = c["kind"]
    if kind == "steps":
        s.stepper.invalidate()
        s.stepper.step_auto(s.f, c["steps"])
        return _read(s.stepper, s.out)
    if kind == "host":
        s.stepper.eng.call("fl_step_host", *s.args)
        return {"u": s.out.u, "v": s.out.v, "p": s.out.p, "dye": s.out.dye}
    if kind == "sim":
        s.sim.step()
        s.sim.stepper.read_pressure(s.p)
        return {"u": s.sim.f.u, "v": s.sim.f.v, "p": s.p, "div": s.sim.div}
    if kind == "batch":
        for st, (f, _) in zip(s.steppers, s.f):
            st.upload(f)
        s.batch.step(c["steps"])
        return [_read(st, out) for st, (_, out) in zip(s.steppers, s.f)]
    if kind in ("mg", "rb"):
        s.p[:] = 0
        it, tol = (0, 0.0) if kind == "mg" else (c["iterations"], c["tol"])
        used = s.solver.solve(s.g, s.p, s.div, s.label, s.scale, it, engine.optimal_omega(c["nx"], c["ny"]), tol)
        return {"p": s.p, "used": used}
    if kind == "advect":
        st = s.lib.fl_advect_velocity_noalloc(
            int(c["mac"]), c["nx"], c["ny"], s.h, s.dt, s.u.data_ptr(), s.v.data_ptr(), s.uo.data_ptr(),
            s.vo.data_ptr(), s.label.data_ptr(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if st != native.FL_OK:
            raise native.FlowlabError(st, s.lib.fl_last_error(None).decode())
        return {"u": s.uo, "v": s.vo}
    if not c["train"]:
        return s.net.forward(s.x)
    loss, grad = s.net.train_step(s.x, s.t, s.m, update=False, want_grad=True)
    return {"loss": loss, "grad": grad}


def _read(stepper, out):
    stepper.read_velocity(out)
    stepper.read_pressure(out.p)
    stepper.read_dye(out.dye)
    return {"u": out.u, "v": out.v, "p": out.p, "dye": out.dye}


# ------------------------------------------------------------------ work

def _cycle_flops(cells, pre, post):
    """One V-cycle: 7 operations an update, the residual, restriction and prolongation; all levels."""
    return 4 / 3 * cells * (7 * (pre + post) + 16)


def _step_work(nx, ny, scale, solve_flops):
    """A step: the state and labels read once, the state written once; about 200 operations a
    cell and dye cell for the advections and the other passes."""
    n, d = nx * ny, nx * ny * scale * scale
    return 4 * 2 * ((nx + 1) * ny + nx * (ny + 1) + n + 3 * d) + n, 100 * (n + d) + solve_flops


def work(case):
    kind = case["kind"]
    if kind in ("unet",):
        flops = warmstart.forward_flops(case["h"], case["w"])[0] * case["batch"]
        px = case["batch"] * case["h"] * case["w"]
        params = 4 * warmstart.he_init().size
        return {"bytes": 16 * px + params + (8 * px + params if case["train"] else 0),
                "flops": flops * (3 if case["train"] else 1)}
    if kind == "batch":
        sides = [s for s in (64, 128, 256, 512) if s <= case["max_side"]]
        per = [_step_work(n, n, 1, 8 * _cycle_flops(n * n, 3, 3))
               for n in (sides[k % len(sides)] for k in range(case["scenes"]))]
        return {"bytes": case["steps"] * sum(b for b, _ in per), "flops": case["steps"] * sum(q for _, q in per)}
    nx, ny = case["nx"], case["ny"]
    n = nx * ny
    if kind == "advect":
        faces = (nx + 1) * ny + nx * (ny + 1)
        return {"bytes": 8 * faces + n, "flops": (130 if case["mac"] else 60) * faces}
    if kind == "mg":
        return {"bytes": 13 * n, "flops": case["cycles"] * _cycle_flops(n, case["pre"], case["post"])}
    if kind == "rb":
        return {"bytes": 13 * n, "flops": 7 * n * case["iterations"]}
    scene = case.get("scene", "sim")
    solve = {"plume": 4 * _cycle_flops(n, 3, 3), "lattice": 18 * _cycle_flops(n, 3, 3), "street": 60 * 7 * n,
             "sim": 2 * _cycle_flops(n, 2, 2)}[scene]
    b, q = _step_work(nx, ny, case.get("dye_scale", 1), solve)
    return {"bytes": b * case.get("steps", 1), "flops": q * case.get("steps", 1)}


# ------------------------------------------------------- 64-bit restatement
#
# The same formulas in float64 torch: fields are (rows, columns) tensors.

def _t(a, *shape):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    return torch.as_tensor(np.asarray(a)).to(dev, torch.float64).reshape(shape)


def _axis(pos, count):
    c = pos.clamp(0, count - 1)
    i = c.floor().clamp(max=count - 2)
    return i.long(), c - i


def _corners(q, px, py):
    i, fx = _axis(px, q.shape[1])
    j, fy = _axis(py, q.shape[0])
    return (q[j, i], q[j, i + 1], q[j + 1, i], q[j + 1, i + 1]), fx, fy


def _sample(q, px, py):
    (a, b, c, d), fx, fy = _corners(q, px, py)
    lo, hi = a + fx * (b - a), c + fx * (d - c)
    return lo + fy * (hi - lo)


def _clamped(val, q, px, py):
    k, _, _ = _corners(q, px, py)
    k = torch.stack(k)
    return torch.maximum(torch.minimum(val, k.amax(0)), k.amin(0))


class _Grid64:
    def __init__(self, nx, ny, h, label, scale=1):
        self.nx, self.ny, self.h, self.scale = nx, ny, h, scale
        self.label = _t(label, ny, nx)
        solid = self.label == SOLID
        wall = torch.nn.functional.pad(solid, (1, 1, 1, 1), value=True)
        self.no_u = wall[1:-1, :-1] | wall[1:-1, 1:]     # a face beside a solid cell or the outside
        self.no_v = wall[:-1, 1:-1] | wall[1:, 1:-1]
        self.solid, self.fluid = solid, self.label == FLUID

    def at(self, rows, cols, oy, ox, h):
        d = self.label.device
        y = (torch.arange(rows, device=d, dtype=torch.float64) + oy) * h
        x = (torch.arange(cols, device=d, dtype=torch.float64) + ox) * h
        return x[None, :].expand(rows, cols), y[:, None].expand(rows, cols)

    def su(self, u, x, y):
        return _sample(u, x / self.h, y / self.h - 0.5)

    def sv(self, v, x, y):
        return _sample(v, x / self.h - 0.5, y / self.h)

    def back(self, u, v, x, y, dt):
        mx, my = x - 0.5 * dt * self.su(u, x, y), y - 0.5 * dt * self.sv(v, x, y)
        return x - dt * self.su(u, mx, my), y - dt * self.sv(v, mx, my)

    def advect(self, q, skip, u, v, pos, off, h, dt, mac):
        """q at positions pos, its index of a point (x, y) being (x / h - off[0], y / h - off[1])."""
        at = lambda b: (b[0] / h - off[0], b[1] / h - off[1])  # noqa: E731
        b = at(self.back(u, v, *pos, dt))
        hat = torch.where(skip, q, _sample(q, *b))
        if not mac:
            return hat
        rev = _sample(hat, *at(self.back(u, v, *pos, -dt)))
        return torch.where(skip, q, _clamped(hat + 0.5 * (q - rev), q, *b))

    def advect_velocity(self, u, v, dt, mac):
        nx, ny, h = self.nx, self.ny, self.h
        return (self.advect(u, self.no_u, u, v, self.at(ny, nx + 1, 0.5, 0, h), (0, 0.5), h, dt, mac),
                self.advect(v, self.no_v, u, v, self.at(ny + 1, nx, 0, 0.5, h), (0.5, 0), h, dt, mac))

    def advect_dye(self, dye, u, v, dt, mac):
        n, dh = self.scale, self.h / self.scale
        skip = self.solid.repeat_interleave(n, 0).repeat_interleave(n, 1)
        pos = self.at(self.ny * n, self.nx * n, 0.5, 0.5, dh)
        return torch.stack([self.advect(q, skip, u, v, pos, (0.5, 0.5), dh, dt, mac) for q in dye])

    def forces(self, u, v, dye, dt, beta, alpha, eps):
        nx, ny, h = self.nx, self.ny, self.h
        if eps:
            curl = (v[1:-1, 1:] - v[1:-1, :-1]) / h - (u[1:, 1:-1] - u[:-1, 1:-1]) / h    # corners 1..n-1
            i, j = (torch.arange(n, device=u.device) for n in (nx, ny))
            lo, hi = (lambda k, n: (k.clamp(1, n - 1) - 1)), (lambda k, n: ((k + 1).clamp(1, n - 1) - 1))
            w = 0.25 * sum(curl[a][:, b] for a in (lo(j, ny), hi(j, ny)) for b in (lo(i, nx), hi(i, nx)))
            ie, iw, jn, js = (i + 1).clamp(max=nx - 1), (i - 1).clamp(min=0), (j + 1).clamp(max=ny - 1), (j - 1).clamp(min=0)
            gx = (w[:, ie].abs() - w[:, iw].abs()) / ((ie - iw) * h)
            gy = (w[jn].abs() - w[js].abs()) / ((jn - js) * h)[:, None]
            mag = (gx * gx + gy * gy).sqrt() + 1e-20
            fx, fy = eps * h * gy / mag * w, -eps * h * gx / mag * w
            fx, fy = fx * ~self.solid, fy * ~self.solid
        x, y = self.at(ny + 1, nx, 0, 0.5, h)
        dh = h / self.scale
        add = sum((gain * _sample(dye[c], x / dh - 0.5, y / dh - 0.5) for c, gain in ((0, beta * dt), (1, -alpha * dt)) if gain),
                  torch.zeros_like(v))
        if eps:
            add[1:-1] += 0.5 * dt * (fy[:-1] + fy[1:])
            u = u.clone()
            u[:, 1:-1] += 0.5 * dt * (fx[:, :-1] + fx[:, 1:]) * ~self.no_u[:, 1:-1]
        v = v.clone()
        v[1:-1] += (add * ~self.no_v)[1:-1]
        return u, v

    def divergence(self, u, v):
        return (u[:, 1:] - u[:, :-1] + v[1:] - v[:-1]) / self.h

    def project(self, p, u, v, gs):
        u, v = u.clone(), v.clone()
        u[:, 1:-1] -= gs * (p[:, 1:] - p[:, :-1]) * ~self.no_u[:, 1:-1]
        v[1:-1] -= gs * (p[1:] - p[:-1]) * ~self.no_v[1:-1]
        air = self.label == AIR
        for a, inner, outer, open_, keep in ((u.T, 1, 0, air[:, 0], torch.minimum), (u.T, -2, -1, air[:, -1], torch.maximum),
                                             (v, 1, 0, air[0], torch.minimum), (v, -2, -1, air[-1], torch.maximum)):
            a[inner] = torch.where(open_, keep(a[inner], torch.zeros_like(a[inner])), a[inner])
            a[outer] = torch.where(open_, a[inner], a[outer])
        return u, v


class _Level64:
    def __init__(self, label):
        self.label, (self.ny, self.nx) = label, label.shape
        links = torch.nn.functional.pad((label != SOLID).double(), (1, 1, 1, 1))
        self.cnt = links[1:-1, 2:] + links[1:-1, :-2] + links[2:, 1:-1] + links[:-2, 1:-1]
        self.on = (label == FLUID) & (self.cnt > 0)
        j, i = torch.meshgrid(*(torch.arange(n, device=label.device) for n in label.shape), indexing="ij")
        self.colour = [self.on & ((i + j) % 2 == c) for c in (0, 1)]
        self.inv = 1 / self.cnt.clamp(min=1)

    def nsum(self, x):
        q = torch.nn.functional.pad(x, (1, 1, 1, 1))
        return q[1:-1, 2:] + q[1:-1, :-2] + q[2:, 1:-1] + q[:-2, 1:-1]

    def sweeps(self, x, sb, pairs, omega=1.0):
        for _ in range(pairs):
            for c in self.colour:
                x = torch.where(c, (1 - omega) * x + omega * (self.nsum(x) - sb) * self.inv, x)
        return x

    def residual(self, x, b):
        return torch.where(self.on, b - (self.cnt * x - self.nsum(x)), torch.zeros_like(x))

    def coarser(self):
        q = torch.nn.functional.pad(self.label, (0, self.nx % 2, 0, self.ny % 2), value=SOLID)
        k = torch.stack([q[a::2, b::2] for a in (0, 1) for b in (0, 1)])
        one = torch.ones_like(k[0])
        return _Level64(torch.where((k == AIR).any(0), AIR * one, torch.where((k == FLUID).any(0), FLUID * one, SOLID * one)))


def _levels64(label, coarsest):
    out = [_Level64(label)]
    while out[-1].nx > coarsest or out[-1].ny > coarsest:
        out.append(out[-1].coarser())
    return out


def _cycle64(levels, x, b, pre, post, coarse, l=0):
    L = levels[l]
    if l == len(levels) - 1:
        return L.sweeps(x, -b, coarse)
    x = L.sweeps(x, -b, pre)
    r = torch.nn.functional.pad(L.residual(x, b), (0, L.nx % 2, 0, L.ny % 2))
    bc = r[::2, ::2] + r[::2, 1::2] + r[1::2, ::2] + r[1::2, 1::2]
    e = _cycle64(levels, torch.zeros_like(bc), bc, pre, post, coarse, l + 1)
    near = lambda n, m: (torch.arange(n, device=x.device) // 2,  # noqa: E731
                         (torch.arange(n, device=x.device) // 2 + 2 * (torch.arange(n, device=x.device) % 2) - 1).clamp(0, m - 1))
    (i, i2), (j, j2) = near(L.nx, e.shape[1]), near(L.ny, e.shape[0])
    add = 0.5625 * e[j][:, i] + 0.1875 * (e[j][:, i2] + e[j2][:, i]) + 0.0625 * e[j2][:, i2]
    return L.sweeps(torch.where(L.label == FLUID, x + add, x), -b, post)


def _solve64(levels, p, b, fluid, tol, cycles, shape, first_test):
    """Cycles to a relative residual, tested before the first one too where asked; (p, cycles)."""
    rms = lambda r, on: float((r[on].square().mean()).sqrt()) if bool(on.any()) else 0.0  # noqa: E731
    L, brms = levels[0], rms(b, fluid)
    if brms == 0:
        return torch.zeros_like(p), 0
    for k in range(cycles + 1):
        if (k or first_test) and tol > 0 and rms(L.residual(p, b), L.on) <= tol * brms or k == cycles:
            return p, k
        p = _cycle64(levels, p, b, *shape)


def _steps64(nx, ny, h, f, patch, prm, steps, scale=1):
    """`steps` whole steps from fields f; (u, v, p, dye, the last step's divergence after it)."""
    G = _Grid64(nx, ny, h, f.label, scale)
    u, v, p = _t(f.u, ny, nx + 1), _t(f.v, ny + 1, nx), _t(f.p, ny, nx)
    dye = _t(f.dye, 3, ny * scale, nx * scale)
    mac, mg = prm.scheme == native.FL_MACCORMACK, prm.solver == native.FL_SOLVER_MG
    levels = _levels64(G.label, prm.mg_coarsest) if mg else [_Level64(G.label)]
    for _ in range(steps):
        umax = max(float(u.abs().max()), float(v.abs().max()))
        dt = min(prm.dt_max, prm.cfl_target * h / umax) if umax > 1e-9 else prm.dt_max
        k, gs = prm.rho * h * h / dt, dt / (prm.rho * h)
        u, v = G.advect_velocity(u, v, dt, mac)
        u, v = G.forces(u, v, dye, dt, prm.beta, prm.alpha, prm.confinement)
        div = G.divergence(u, v)
        if mg:
            p, _ = _solve64(levels, p, -k * div, G.fluid, prm.tol, prm.mg_max_cycles,
                            (prm.mg_pre, prm.mg_post, prm.mg_coarse_sweeps), bool(prm.mixed))
        else:
            p = levels[0].sweeps(p, k * div, prm.pressure_iters, prm.omega)
        u, v = G.project(p, u, v, gs)
        dye = G.advect_dye(dye, u, v, dt, mac)
        dye = dye * _t([math.exp(-d * dt) for d in prm.dye_decay], 3, 1, 1)
        if patch is not None:
            q = _t(patch.data, 4, patch.ny, patch.nx)
            box = dye[:, patch.j0:patch.j0 + patch.ny, patch.i0:patch.i0 + patch.nx]
            box += q[3] * (q[:3] - box)
    return u, v, p, dye, G.divergence(u, v)


def _net64(theta, x):
    at = 0
    acts = []
    conv = torch.nn.functional.conv2d
    pool = lambda q: torch.nn.functional.avg_pool2d(q, 2)  # noqa: E731
    up = lambda q, skip: torch.cat([q.repeat_interleave(2, 2).repeat_interleave(2, 3), skip], 1)  # noqa: E731

    def layer(q, k):
        nonlocal at
        cin, cout, size, _ = warmstart.LAYERS[k]
        w = theta[at:at + cout * size * size * cin].reshape(cout, size, size, cin).permute(0, 3, 1, 2)
        at += w.numel() + cout
        q = conv(q, w, theta[at - cout:at], padding=size // 2)
        return torch.relu(q) if size == 3 else q

    q = x.permute(0, 3, 1, 2)
    for k in (0, 2, 4):
        acts.append(layer(layer(q, k), k + 1))
        q = pool(acts[-1])
    q = layer(layer(q, 6), 7)
    for k in (8, 10, 12):
        q = layer(layer(up(q, acts.pop()), k), k + 1)
    return layer(q, 14)[:, 0]


def _host(d):
    return {k: v.detach().cpu().numpy().reshape(-1) if isinstance(v, torch.Tensor) else v for k, v in d.items()}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("steps", "host"):
        g, dg, f, patch, prm = _scene(case, seed)
        for name in ("p", "u", "v", "dye"):
            setattr(f, name, getattr(f, name).astype(np.float32))
        u, v, p, dye, _ = _steps64(g.nx, g.ny, g.h, f, patch, prm, case.get("steps", 1))
        return _host({"u": u, "v": v, "p": p, "dye": dye})
    if kind == "sim":
        g, dg, f, _, _ = _scene(dict(case, scene="street"), seed)
        prm = native.default_params(scheme=engine.SCHEMES[case["scheme"]])
        u, v, p, _, div = _steps64(g.nx, g.ny, g.h, f, None, prm, 1, case["dye_scale"])
        return dict(_host({"u": u, "v": v, "p": p}), div=None)  # what is left of a divergence is rounding
    if kind == "batch":
        prm = configs.random_scene_params(mixed=1)
        out = []
        for g, f in _boxes(case, seed):
            for name in ("p", "u", "v", "dye"):
                setattr(f, name, getattr(f, name).astype(np.float32))
            u, v, p, dye, _ = _steps64(g.nx, g.ny, g.h, f, None, prm, case["steps"])
            out.append(_host({"u": u, "v": v, "p": p, "dye": dye}))
        return out
    if kind == "mg":
        g, div, label, scale = _problem(case, seed)
        levels = _levels64(_t(label, g.ny, g.nx), 4)
        b = -scale * _t(div, g.ny, g.nx)
        p, used = _solve64(levels, torch.zeros_like(b), b, levels[0].label == FLUID, 0.0, case["cycles"],
                           (case["pre"], case["post"], 8), False)
        return dict(_host({"p": p}), used=used)
    if kind == "rb":
        g, div, label, scale = _problem(case, seed)
        L, d = _Level64(_t(label, g.ny, g.nx)), _t(div, g.ny, g.nx)
        target = case["tol"] * float(d[L.label == FLUID].square().mean().sqrt())
        p, used = torch.zeros_like(d), case["iterations"]
        for k in range(1, case["iterations"] + 1):
            p = L.sweeps(p, scale * d, 1, engine.optimal_omega(g.nx, g.ny))
            if target > 0 and k % 12 == 0 and float((L.residual(p, -scale * d) / scale)[L.on].square().mean().sqrt()) <= target:
                used = k
                break
        return dict(_host({"p": p}), used=used)
    if kind == "advect":
        u, v, label, h, dt = _flow(case, seed)
        ny, nx = label.shape
        u, v = _Grid64(nx, ny, h, label).advect_velocity(_t(u, ny, nx + 1), _t(v, ny + 1, nx), dt, case["mac"])
        return _host({"u": u, "v": v})
    x, t, m = _pairs(case, seed)
    theta = _t(warmstart.load(warmstart.DEFAULT_WEIGHTS)[0], -1)
    if not case["train"]:
        with torch.no_grad():
            return _net64(theta, _t(x, *x.shape)).cpu().numpy()
    theta.requires_grad_(True)
    m = _t(m, *m.shape)
    loss = (((_net64(theta, _t(x, *x.shape)) - _t(t, *t.shape)) * m).square().sum()) / m.sum()
    loss.backward()
    return {"loss": float(loss.detach()), "grad": theta.grad.cpu().numpy()}
