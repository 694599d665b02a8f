"""The framework's workloads as measured cases: what a program asks of it through
its public entry points (aether_fluid's FluidSolver3D, Ensemble, Adjoint and
DeviceMedium, and the C entry afl_solve_cg_noalloc).

Kinds:
  frame     steps of the smoke solver, then the read a renderer or a checkpoint
            makes of the state (FluidMedium.from_solver, or every field)
  ensemble  steps of a batch of plumes of uneven sizes, then their densities
  adjoint   a rollout and its gradient with respect to the initial velocity and
            the source's amplitude map
  rays      the renderer's medium queries on host ray buffers
  pressure  a pressure solve on the caller's device buffers

exact() restates each kind in plain 64-bit torch, without the framework.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "aether-core-engine_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

BOUNDS = ((-1.0, -1.0, -1.0), (1.0, 1.0, 1.0))
SIGMA_T, PHASE_G = 1.42, 0.34  # the reference program's medium (src/main.rs:109)


# ---- cases -------------------------------------------------------------------
def _frame(nx, ny, nz, steps, precision="fp64", solver="cg", iters=200, rel_tol=1e-6,
           source="sphere", read="frame", each=False):
    return {"kind": "frame", "nx": nx, "ny": ny, "nz": nz, "steps": steps,
            "precision": precision, "solver": solver, "iters": iters, "rel_tol": rel_tol,
            "source": source, "read": read, "each": each}


def listed():
    return [
        # The reference program's own fluid stage: 36x52x36 with the two jets, 28 CG
        # iterations, step() and its telemetry one call at a time, then the hand-off to
        # the renderer.  Latency and launches are all there is.
        dict(_frame(36, 52, 36, 10, iters=28, rel_tol=0.0, source="jets", each=True),
             name="jets 36x52x36"),
        # The small smoke plume as it is checked against the oracle: CG to 1e-6, whole state.
        dict(_frame(64, 64, 64, 12, read="state"), name="plume 64 fp64"),
        # The headline plume, FP64 drop-in form, whole state at the end.
        dict(_frame(128, 128, 128, 12, read="state"), name="plume 128 fp64"),
        # The same plume in the mixed form, read as a renderer's frame.
        dict(_frame(128, 128, 128, 12, precision="mixed"), name="plume 128 mixed"),
        # The same plume with the reference's other pressure solver.
        dict(_frame(128, 128, 128, 12, solver="sor", iters=80, rel_tol=0.0),
             name="plume 128 sor"),
        # A ragged grid whose extents are no multiple of any tile (a scene's own proportions).
        dict(_frame(90, 133, 77, 10, read="state"), name="plume 90x133x77 fp64"),
        # The large plume, mixed and FP64: the working set leaves the chip and L2.
        dict(_frame(256, 256, 256, 6, precision="mixed"), name="plume 256 mixed"),
        dict(_frame(256, 256, 256, 4), name="plume 256 fp64"),
        # The benchmark ensemble: 48 plumes of three sizes in one batch.
        {"name": "ensemble 48", "kind": "ensemble", "small": 16, "middle": 16, "large": 16,
         "steps": 4},
        # Inverse design on a small grid: rollout and gradient.
        {"name": "adjoint 48", "kind": "adjoint", "nx": 48, "ny": 48, "nz": 48, "steps": 12,
         "every": 4},
        # A frame's shadow and camera rays against the medium of a 128^3 plume.
        {"name": "rays 1M", "kind": "rays", "nx": 128, "ny": 128, "nz": 128, "rays": 1 << 20},
        # A game's or render thread's pressure solve on its own device buffers.
        {"name": "pressure 40x36x30", "kind": "pressure", "nx": 40, "ny": 36, "nz": 30,
         "iters": 60},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame"] * 6 + ["ensemble", "adjoint", "rays", "pressure"])
    if kind == "frame":
        base = _log_int(rng, 24, 200)
        nx, ny, nz = (max(16, min(220, int(base * rng.uniform(0.75, 1.35)))) for _ in range(3))
        source = "jets" if rng.random() < 0.25 else "sphere"
        solver = "sor" if rng.random() < 0.25 else "cg"
        precision = "mixed" if source == "sphere" and rng.random() < 0.45 else "fp64"
        iters = rng.randint(20, 80) if solver == "sor" or source == "jets" else 200
        rel_tol = 1e-6 if solver == "cg" and source == "sphere" else 0.0
        big = nx * ny * nz > 4e6
        read = "state" if precision == "fp64" and not big and rng.random() < 0.5 else "frame"
        return _frame(nx, ny, nz, 3 if big else rng.randint(3, 8), precision, solver, iters, rel_tol, source,
                      read, rng.random() < 0.3)
    if kind == "ensemble":
        return {"kind": "ensemble", "small": rng.randint(1, 16), "middle": rng.randint(0, 16),
                "large": rng.randint(0, 12), "steps": rng.randint(2, 4)}
    if kind == "adjoint":
        nx, ny, nz = (rng.randint(20, 52) for _ in range(3))
        return {"kind": "adjoint", "nx": nx, "ny": ny, "nz": nz, "steps": rng.randint(4, 12),
                "every": rng.randint(2, 6)}
    if kind == "rays":
        nx, ny, nz = (_log_int(rng, 24, 140) for _ in range(3))
        return {"kind": "rays", "nx": nx, "ny": ny, "nz": nz, "rays": _log_int(rng, 1000, 1 << 20)}
    nx, ny, nz = (_log_int(rng, 10, 64) for _ in range(3))
    return {"kind": "pressure", "nx": nx, "ny": ny, "nz": nz, "iters": rng.randint(20, 200)}


# ---- inputs, from the seed alone ------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _uniform(case, seed, count, lo, hi):
    n = case["nx"] * case["ny"] * case["nz"]
    g = _gen(seed)
    return [torch.rand(n, dtype=torch.float64, device="cuda", generator=g) * (hi - lo) + lo
            for _ in range(count)]


def _sphere(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    return (nx / 2, 0.1 * ny, nz / 2), 5.0 * nx / 64.0


def _dt(case):
    # one cell per unit speed for the fast jets, half a cell for the plumes
    return ((1.0 if case.get("source") == "jets" else 0.5) /
            max(case["nx"], case["ny"], case["nz"]))


def _knobs(case):
    if case.get("source") == "jets":  # src/main.rs:84-86 and the defaults of src/fluid.rs:79-83
        return dict(vorticity_eps=6.5, buoyancy_beta=6.8, gravity_alpha=0.45)
    return dict(vorticity_eps=0.3, buoyancy_beta=0.4, gravity_alpha=0.08)


def _smoke(case, seed):
    """Density and temperature of a risen plume: a wavy column that thins out upward."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    ax = [torch.linspace(0, 1, m, dtype=torch.float64, device="cuda") for m in (nz, ny, nx)]
    z, y, x = torch.meshgrid(*ax, indexing="ij")
    ph = torch.rand(6, dtype=torch.float64, device="cuda", generator=_gen(seed)) * 6.28
    cx = 0.5 + 0.10 * y * torch.sin(7 * y + ph[0])
    cz = 0.5 + 0.10 * y * torch.cos(6 * y + ph[1])
    r = 0.07 + 0.16 * y
    d2 = ((x - cx) ** 2 + (z - cz) ** 2) / r ** 2
    lumps = 1.0 + 0.5 * (torch.sin(23 * x + ph[2]) * torch.sin(19 * y + ph[3]) *
                         torch.sin(21 * z + ph[4]))
    dens = torch.clamp((1.0 - d2) * lumps * (1.15 - y), min=0.0)
    return dens.reshape(-1), (0.8 * dens * (1.1 - y)).reshape(-1)


def _rays(case, seed):
    """Rays as rows: origin, direction, t_min, end.  Camera rays from in front of the box."""
    g = _gen(seed + 7)
    n = case["rays"]
    u = torch.rand(n, 6, dtype=torch.float64, device="cuda", generator=g)
    rows = torch.empty(n, 8, dtype=torch.float64, device="cuda")
    rows[:, 0] = 3.0 * (u[:, 0] - 0.5)
    rows[:, 1] = 2.0 * (u[:, 1] - 0.5)
    rows[:, 2] = -3.0 - u[:, 2]
    target = 1.6 * (u[:, 3:6] - 0.5)
    rows[:, 3:6] = target - rows[:, 0:3]
    rows[:, 6] = 1e-4
    rows[:, 7] = 2.0 + 6.0 * u[:, 2]
    return rows


def _rhs(case, seed):
    """A divergence-like right-hand side: zero on the walls, zero mean inside."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    b = torch.zeros(nz, ny, nx, dtype=torch.float64, device="cuda")
    r = torch.randn(nz - 2, ny - 2, nx - 2, dtype=torch.float64, device="cuda",
                    generator=_gen(seed)) * 1e-3
    b[1:-1, 1:-1, 1:-1] = r - r.mean()
    return b.reshape(-1)


# ---- what a program holds before the call --------------------------------------------
def _host(t):
    return t.cpu().numpy()


def _solver(case):
    import aether_fluid as af
    s = af.FluidSolver3D(case["nx"], case["ny"], case["nz"],
                         precision=af.Precision.MIXED if case["precision"] == "mixed"
                         else af.Precision.FP64)
    s.set_params(solver_kind=0 if case["solver"] == "cg" else 1, solver_iters=case["iters"],
                 cg_rel_tol=case["rel_tol"], sor_omega=1.7, **_knobs(case))
    return s


def prepare(case, seed):
    import aether_fluid as af
    kind = case["kind"]
    if kind == "frame":
        s = _solver(case)
        for name, v in zip("uvw", _uniform(case, seed, 3, -0.01, 0.01)):
            s.set_field(name, _host(v))
        s.enforce_wall_velocity_bc()
        if case["source"] == "sphere":
            s.set_sphere_source(*_sphere(case))
        s.synchronize()
        return {"case": case, "solver": s, "t": 0.0}
    if kind == "ensemble":
        from aether_fluid.ensemble import Ensemble, InstanceSpec
        rng = np.random.default_rng(seed)
        specs = []
        for count, (nx, ny, nz) in ((case["small"], (32, 32, 32)), (case["middle"], (48, 48, 48)),
                                    (case["large"], (64, 128, 64))):
            for _ in range(count):
                at = [b + (2 * x - 1) * 0.1 * e for b, x, e in
                      zip((nx / 2, 0.1 * ny, nz / 2), rng.random(3), (nx, ny, nz))]
                specs.append(InstanceSpec(nx, ny, nz, int(rng.integers(1 << 31)),
                                          alpha=0.05 + 0.05 * rng.random(),
                                          beta=0.3 + 0.2 * rng.random(), center=tuple(at)))
        return {"case": case, "ensemble": Ensemble(specs, precision=af.Precision.MIXED)}
    if kind == "adjoint":
        from aether_fluid.adjoint import Adjoint
        center, radius = _sphere(case)
        u, v, w, amp, target = _adjoint_inputs(case, seed)
        adj = Adjoint(case["nx"], case["ny"], case["nz"], center=center, radius=radius,
                      checkpoint_every=case["every"])
        return {"case": case, "adjoint": adj, "x": [_host(a) for a in (u, v, w, amp)],
                "target": _host(target)}
    if kind == "rays":
        s = af.FluidSolver3D(case["nx"], case["ny"], case["nz"])
        for name, v in zip(("density", "temperature"), _smoke(case, seed)):
            s.set_field(name, _host(v))
        medium = af.DeviceMedium.from_solver(s, af.Aabb(*BOUNDS), 4.0 * SIGMA_T, PHASE_G)
        s.close()
        return {"case": case, "medium": medium, "rays": _host(_rays(case, seed)),
                "seed": int(seed)}
    b = _rhs(case, seed)
    return {"case": case, "b": b, "p": torch.empty_like(b), "lib": af.load()}


def _adjoint_inputs(case, seed):
    u, v, w, a, t = _uniform(case, seed, 5, 0.0, 1.0)
    # velocity in [-0.01, 0.01], amplitude in [0.5, 1.5], target density in [0, 0.1]
    return 0.02 * u - 0.01, 0.02 * v - 0.01, 0.02 * w - 0.01, 0.5 + a, 0.1 * t


# ---- one pass ------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "frame":
        return _run_frame(state, case)
    if kind == "ensemble":
        e = state["ensemble"]
        tel, _ = e.run(case["steps"])
        # float32: the mixed form's own precision
        return {"telemetry": tel.astype(np.float32),
                "density": np.concatenate([e.field(m, "density") for m in range(e.count)])
                .astype(np.float32)}
    if kind == "adjoint":
        a = state["adjoint"]
        rho = a.forward(*state["x"], case["steps"], _dt(case))
        grads = a.backward(rho - state["target"])
        return {"rho": rho, "grads": list(grads)}
    if kind == "rays":
        m = state["medium"]
        tr = m.transmittance(state["rays"], state["seed"])
        hit, t, rho, temp = m.sample_interaction(state["rays"], state["seed"])
        return {"transmittance": tr, "hit": hit, "t": t, "density": rho, "temperature": temp}
    from aether_fluid._lib import AflSolveInfo, check
    p = state["p"].zero_()
    info = AflSolveInfo()
    check(state["lib"].afl_solve_cg_noalloc(
        state["b"].data_ptr(), p.data_ptr(), case["nx"], case["ny"], case["nz"], case["iters"],
        0.0, torch.cuda.current_stream().cuda_stream, ctypes.byref(info)))
    return {"pressure": p, "residual": info.final_residual}


def _run_frame(state, case):
    from aether_fluid import Aabb, FluidMedium
    s, dt = state["solver"], _dt(case)
    if case["each"]:
        tel = []
        for _ in range(case["steps"]):
            tel.append(s.step(dt, state["t"]).as_array())
            state["t"] += dt
        tel = np.stack(tel)
    else:
        tel, _ = s.run(case["steps"], dt, t0=state["t"])
        state["t"] += case["steps"] * dt
    if case["read"] == "state":
        out = {f: s.get_field(f) for f in ("u", "v", "w", "density", "temperature")}
    else:
        m = FluidMedium.from_solver(s, Aabb(*BOUNDS), SIGMA_T, PHASE_G)
        out = {"density": m.density, "temperature": m.temperature, "max": m.max_density}
    out["telemetry"] = tel
    if case["precision"] == "mixed":  # the mixed form's fields are float32 by nature
        out = {k: np.asarray(v, dtype=np.float32) for k, v in out.items()}
    return out


# ---- what a pass cannot do without ---------------------------------------------------
def work(case):
    """Bytes: each input of a pass read once and each output written once; a step's
    state once each way.  Flops: the arithmetic of the stages and of every solver
    iteration (CG: 7-point operator, two products, three updates = 21 per cell)."""
    kind = case["kind"]
    if kind == "frame":
        n = case["nx"] * case["ny"] * case["nz"]
        e = 4 if case["precision"] == "mixed" else 8
        per = 21 if case["solver"] == "cg" else 12
        steps = case["steps"]
        out = (5 if case["read"] == "state" else 2) * 8 * n
        return {"bytes": steps * n * (10 * e + 16) + out,
                "flops": steps * n * (per * case["iters"] + 700)}
    if kind == "ensemble":
        n = case["small"] * 32 ** 3 + case["middle"] * 48 ** 3 + case["large"] * 64 * 128 * 64
        return {"bytes": case["steps"] * n * 56 + 8 * n,
                "flops": case["steps"] * n * (21 * 150 + 700)}
    if kind == "adjoint":
        n = case["nx"] * case["ny"] * case["nz"]
        solves = 3 * case["steps"]  # forward, recomputed forward, adjoint
        return {"bytes": n * 8 * (10 + 10 * solves), "flops": n * solves * (21 * 150 + 1000)}
    if kind == "rays":
        return {"bytes": case["rays"] * (64 + 8 + 4 + 24) + 16 * case["nx"] * case["ny"] *
                case["nz"], "flops": case["rays"] * 2 * 8 * 120}
    n = case["nx"] * case["ny"] * case["nz"]
    return {"bytes": 24 * n, "flops": 21 * n * case["iters"]}


# ---- the same in plain 64-bit torch ------------------------------------------------------
class _Ref:
    """The smoke step (src/fluid.rs:94-672) on [nz, ny, nx] float64 tensors."""

    def __init__(self, case):
        self.nx, self.ny, self.nz = case["nx"], case["ny"], case["nz"]
        self.dims = (self.nx, self.ny, self.nz)
        self.h = 1.0 / max(self.dims)
        ax = [torch.arange(m, device="cuda", dtype=torch.float64)
              for m in (self.nz, self.ny, self.nx)]
        self.k, self.j, self.i = torch.meshgrid(*ax, indexing="ij")
        shape = (self.nz, self.ny, self.nx)
        self.inner = torch.zeros(shape, dtype=torch.bool, device="cuda")
        self.inner[1:-1, 1:-1, 1:-1] = True
        self.f = [torch.zeros(shape, dtype=torch.float64, device="cuda") for _ in range(5)]
        self.p = torch.zeros(self.nz - 2, self.ny - 2, self.nx - 2, dtype=torch.float64,
                             device="cuda")
        one = torch.ones_like(self.p)
        self.diag = self._neighbours(one)

    def walls(self, f):
        for a in range(3):  # u, v, w: every wall cell, and the first face along its own axis
            f[a] = torch.where(self.inner, f[a], 0.0)
            f[a].select(2 - a, 1).zero_()

    def _corner(self, disp):
        base, ts = 0, []
        for g, d, m, stride in zip((self.i, self.j, self.k), disp, self.dims,
                                   (1, self.nx, self.nx * self.ny)):
            x = torch.clamp(g - d, 0.5, m - 1.500001)
            c = torch.floor(x)
            ts.append(x - c)
            base = base + c.to(torch.int64) * stride
        return base, ts

    def _eight(self, q, base):
        flat, sy, sz = q.reshape(-1), self.nx, self.nx * self.ny
        return [flat[base + o] for o in (0, 1, sy, sy + 1, sz, sz + 1, sz + sy, sz + sy + 1)]

    def _sample(self, q, disp):
        base, (tx, ty, tz) = self._corner(disp)
        c = self._eight(q, base)
        c = [c[m] * (1 - tx) + c[m + 1] * tx for m in (0, 2, 4, 6)]
        c = [c[m] * (1 - ty) + c[m + 1] * ty for m in (0, 2)]
        return c[0] * (1 - tz) + c[1] * tz

    def advect(self, q, dt, diss, nonneg):
        vel, s = self.f[:3], dt / self.h
        back = [s * a for a in vel]
        fwd = torch.where(self.inner, self._sample(q, back), 0.0)
        bwd = self._sample(fwd, [-a for a in back])
        mc = fwd + 0.5 * (q - bwd)
        c = self._eight(q, self._corner(back)[0])
        lo, hi = c[0], c[0]
        for x in c[1:]:
            lo, hi = torch.minimum(lo, x), torch.maximum(hi, x)
        val = torch.minimum(torch.maximum(mc, lo), hi)
        near = torch.zeros_like(self.inner)
        for g, d, m in zip((self.i, self.j, self.k), back, self.dims):
            near |= (g - d < 1.5) | (g - d > m - 2.5)
        out = torch.where(self.inner, torch.where(near, fwd, val) * diss, 0.0)
        return torch.clamp(out, min=0.0) if nonneg else out

    def sphere(self, center, radius, amp=None):
        d2 = (self.i - center[0]) ** 2 + (self.j - center[1]) ** 2 + (self.k - center[2]) ** 2
        m = self.inner & (d2 < radius * radius)
        self.f[3] = torch.where(m, 1.0, self.f[3])
        self.f[4] = torch.where(m, 1.0 if amp is None else amp, self.f[4])

    def jets(self, t, dt):
        tau = 6.283185307179586
        pulse = (0.65 + 0.35 * math.sin(t * tau * 0.55) +
                 0.25 * max(math.cos(t * tau * 1.35), 0.0))
        ca, sa = math.cos(1.85 * t), math.sin(1.85 * t)
        cx, cz, orbit = 0.5 * self.nx, 0.5 * self.nz, 0.14 * self.nx
        y = min(3, self.ny - 3)
        r2 = max(0.105 * self.nx, 2.2) ** 2
        for c, vel in (((cx + orbit * ca, y + 1.5, cz + orbit * sa),
                        (-2.6 * sa, 7.2 * pulse, 2.6 * ca)),
                       ((cx - orbit * ca, y + 2.0, cz - orbit * sa),
                        (2.6 * sa, 6.4 * pulse, -2.6 * ca))):
            d2 = (self.i - c[0]) ** 2 + (self.j - c[1]) ** 2 + (self.k - c[2]) ** 2
            m = self.inner & (d2 < r2)
            wf = torch.exp(-2.2 * d2 / r2)
            self.f[3] = torch.where(m, torch.clamp(self.f[3] + dt * 9.5 * pulse * wf, max=3.8),
                                    self.f[3])
            self.f[4] = torch.where(m, torch.clamp(self.f[4] + dt * 8.2 * pulse * wf, max=4.5),
                                    self.f[4])
            for a in range(3):
                self.f[a] = torch.where(m, self.f[a] + dt * vel[a] * wf * 4.2, self.f[a])

    def _curl(self):
        u, v, w = self.f[:3]
        c = 0.5 / self.h
        dx = lambda q: (q[1:-1, 1:-1, 2:] - q[1:-1, 1:-1, :-2]) * c  # noqa: E731
        dy = lambda q: (q[1:-1, 2:, 1:-1] - q[1:-1, :-2, 1:-1]) * c  # noqa: E731
        dz = lambda q: (q[2:, 1:-1, 1:-1] - q[:-2, 1:-1, 1:-1]) * c  # noqa: E731
        return dy(w) - dz(v), dz(u) - dx(w), dx(v) - dy(u)

    def forces(self, dt, eps, beta, alpha):
        o = self._curl()
        mag = torch.sqrt(o[0] ** 2 + o[1] ** 2 + o[2] ** 2)  # of the interior
        c = 0.5 / self.h
        g = [(mag[1:-1, 1:-1, 2:] - mag[1:-1, 1:-1, :-2]) * c,
             (mag[1:-1, 2:, 1:-1] - mag[1:-1, :-2, 1:-1]) * c,
             (mag[2:, 1:-1, 1:-1] - mag[:-2, 1:-1, 1:-1]) * c]
        length = torch.sqrt(g[0] ** 2 + g[1] ** 2 + g[2] ** 2) + 1e-10
        n = [x / length for x in g]
        o = [x[1:-1, 1:-1, 1:-1] for x in o]
        f = [x.clone() for x in self.f[:3]]
        for a in range(3):
            b, d = (a + 1) % 3, (a + 2) % 3
            f[a][2:-2, 2:-2, 2:-2] += dt * (eps * self.h * (n[b] * o[d] - n[d] * o[b]))
        lift = beta * self.f[4] - alpha * self.f[3]
        f[1] = torch.where(self.inner, f[1] + dt * lift, f[1])
        self.walls(f)
        self.f[:3] = f

    def _neighbours(self, x):
        s = torch.zeros_like(x)
        s[:, :, 1:] += x[:, :, :-1]
        s[:, :, :-1] += x[:, :, 1:]
        s[:, 1:] += x[:, :-1]
        s[:, :-1] += x[:, 1:]
        s[1:] += x[:-1]
        s[:-1] += x[1:]
        return s

    def cg(self, b, p, iters, rel_tol):
        op = lambda x: self.diag * x - self._neighbours(x)  # noqa: E731
        dot = lambda x, y: torch.dot(x.reshape(-1), y.reshape(-1)).item()  # noqa: E731
        r = b - op(p)
        delta = last = dot(r, r)
        tol2 = rel_tol ** 2 * dot(b, b) if rel_tol > 0 else -1.0
        if not delta > 1e-24 or delta <= tol2:
            return p, math.sqrt(delta)
        d = r.clone()
        for _ in range(iters):
            q = op(d)
            dq = dot(d, q)
            if abs(dq) < 1e-28:
                break
            alpha = delta / dq
            p = p + alpha * d
            r = r - alpha * q
            last = dot(r, r)
            if last < 1e-20 or last <= tol2:
                break
            d = r + (last / delta) * d
            delta = last
        return p, math.sqrt(last)

    def sor(self, b, p, sweeps, omega):
        red = ((self.i + self.j + self.k)[1:-1, 1:-1, 1:-1] % 2) == 0
        for _ in range(sweeps):
            for colour in (red, ~red):
                target = (b + self._neighbours(p)) / self.diag
                p = torch.where(colour, (1.0 - omega) * p + omega * target, p)
        return p

    def project(self, case):
        u, v, w = self.f[:3]
        c = u[1:-1, 1:-1, 1:-1], v[1:-1, 1:-1, 1:-1], w[1:-1, 1:-1, 1:-1]
        div = ((u[1:-1, 1:-1, 2:] - c[0]) + (v[1:-1, 2:, 1:-1] - c[1]) +
               (w[2:, 1:-1, 1:-1] - c[2]))
        if case.get("solver", "cg") == "sor":
            self.p = self.sor(-self.h * div, self.p, case["iters"], 1.7)
        else:
            self.p, _ = self.cg(-self.h * div, self.p, case["iters"], case["rel_tol"])
        f = [u.clone(), v.clone(), w.clone()]
        p, inv = self.p, 1.0 / self.h
        f[0][1:-1, 1:-1, 2:-1] -= (p[:, :, 1:] - p[:, :, :-1]) * inv
        f[1][1:-1, 2:-1, 1:-1] -= (p[:, 1:] - p[:, :-1]) * inv
        f[2][2:-1, 1:-1, 1:-1] -= (p[1:] - p[:-1]) * inv
        self.walls(f)
        self.f[:3] = f

    def telemetry(self, t):
        dv = self.h ** 3
        u, v, w, rho = (x[1:-1, 1:-1, 1:-1] for x in self.f[:4])
        o = self._curl()
        w2 = o[0] ** 2 + o[1] ** 2 + o[2] ** 2
        wgt = torch.where(rho > 1e-8, rho * dv, 0.0)
        mass = wgt.sum().item()
        com = []
        for g, m in zip((self.i, self.j, self.k), self.dims):
            x = (wgt * (2.0 * (g[1:-1, 1:-1, 1:-1] / (m - 1)) - 1.0)).sum().item()
            com.append(min(max(x / mass if mass > 1e-12 else x, -1.0), 1.0))
        return [t, (0.5 * (u * u + v * v + w * w) * dv).sum().item(),
                (0.5 * w2 * dv).sum().item(), math.sqrt(w2.max().item()), mass, *com]

    def step(self, case, t, dt, knobs, amp=None, source="sphere"):
        for a in range(3):
            self.f[a] = self.advect(self.f[a], dt, 0.996, False)
        if source == "jets":
            self.jets(t, dt)
        else:
            self.sphere(*_sphere(case), amp)
        self.forces(dt, knobs["vorticity_eps"], knobs["buoyancy_beta"], knobs["gravity_alpha"])
        self.project(case)
        self.f[3], self.f[4] = (self.advect(self.f[3], dt, 0.996, True),
                                self.advect(self.f[4], dt, 0.985, True))
        return self.telemetry(t)


def _exact_rays(case, seed):
    """Ratio tracking and delta tracking (src/fluid.rs:739-874), all rays in step; ray r
    draws from its own generator seeded seed + r (src/rng.rs:5-88)."""
    dens, temp = _smoke(case, seed)
    rows = _rays(case, seed)
    n = rows.shape[0]
    dims = (case["nx"], case["ny"], case["nz"])
    scale = 4.0 * SIGMA_T
    majorant = max(dens.max().item() * scale, 1e-4)
    inv_maj = 1.0 / majorant
    o, d = rows[:, 0:3], rows[:, 3:6]
    d = d * (1.0 / d.norm(dim=1, keepdim=True))
    lo = torch.tensor(BOUNDS[0], dtype=torch.float64, device="cuda")
    hi = torch.tensor(BOUNDS[1], dtype=torch.float64, device="cuda")
    t0, t1 = (lo - o) / d, (hi - o) / d
    enter = torch.maximum(rows[:, 6], torch.minimum(t0, t1).amax(1))
    leave = torch.minimum(rows[:, 7], torch.maximum(t0, t1).amin(1))

    def shr(x, k):
        return (x >> k) & ((1 << (64 - k)) - 1)

    def rotl(x, k):
        return (x << k) | shr(x, 64 - k)

    def signed(x):
        return x - (1 << 64) if x >= 1 << 63 else x

    def states():
        sm = (torch.arange(n, dtype=torch.int64, device="cuda") + int(seed)) ^ signed(
            0xA5A55A5AF0F00F0F)
        out = []
        for _ in range(4):
            sm = sm + signed(0x9E3779B97F4A7C15)
            z = (sm ^ shr(sm, 30)) * signed(0xBF58476D1CE4E5B9)
            z = (z ^ shr(z, 27)) * signed(0x94D049BB133111EB)
            out.append(z ^ shr(z, 31))
        return out

    def next_f64(s, m):
        """A draw for the rays of mask m; the others keep their state."""
        out = rotl(s[0] + s[3], 23) + s[0]
        a, b, c, e = s
        t = b << 17
        c, e = c ^ a, e ^ b
        b, a, c = b ^ c, a ^ e, c ^ t
        e = rotl(e, 45)
        for x, new in zip(range(4), (a, b, c, e)):
            s[x] = torch.where(m, new, s[x])
        return shr(out, 11).double() * (1.0 / 9007199254740992.0)

    def sample(t):
        pnt = o + d * t[:, None]
        inside = ((pnt >= lo) & (pnt <= hi)).all(1)
        u = (pnt - lo) / torch.clamp(hi - lo, min=1e-9)
        fx, fz = (torch.clamp(4.0 * u[:, a] * (1.0 - u[:, a]), 0.0, 1.0) for a in (0, 2))
        fy = torch.clamp(1.0 - torch.clamp(u[:, 1] - 0.95, min=0.0) / 0.05, 0.0, 1.0)
        feather = torch.sqrt(fx * fz * fy)
        base, ts, stride = 0, [], 1
        for a in range(3):
            x = torch.clamp(u[:, a] * (dims[a] - 1), 0.5, dims[a] - 1.500001)
            c = torch.floor(x)
            ts.append((x - c))
            base = base + c.to(torch.int64) * stride
            stride *= dims[a]
        sy, sz = dims[0], dims[0] * dims[1]
        out = []
        for q in (dens, temp):
            c = [q[base + k] for k in (0, 1, sy, sy + 1, sz, sz + 1, sz + sy, sz + sy + 1)]
            c = [c[m] * (1 - ts[0]) + c[m + 1] * ts[0] for m in (0, 2, 4, 6)]
            c = [c[m] * (1 - ts[1]) + c[m + 1] * ts[1] for m in (0, 2)]
            out.append(torch.where(inside, (c[0] * (1 - ts[2]) + c[1] * ts[2]) * feather, 0.0))
        return out

    tr = torch.ones(n, dtype=torch.float64, device="cuda")
    s, t, live = states(), enter.clone(), enter < leave
    for _ in range(256):
        if not live.any():
            break
        u = torch.clamp(1.0 - next_f64(s, live), min=1e-15)
        t = torch.where(live, t - torch.log(u) * inv_maj, t)
        live = live & (t < leave)
        rho, _ = sample(t)
        sigma = torch.clamp(rho * scale, max=majorant)
        tr = torch.where(live, tr * (1.0 - sigma * inv_maj), tr)
        low = live & (tr < 0.05)
        q = torch.clamp(1.0 - tr, max=0.95)
        dead = next_f64(s, low) < q
        tr = torch.where(low, torch.where(dead, 0.0, tr / (1.0 - q)), tr)
        live = live & ~(low & dead)
    tr = torch.clamp(tr, 0.0, 1.0)

    hit = torch.zeros(n, dtype=torch.int32, device="cuda")
    got = [torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(3)]
    s, t, live = states(), enter.clone(), enter < leave
    for _ in range(256):
        if not live.any():
            break
        u = torch.clamp(1.0 - next_f64(s, live), min=1e-15)
        t = torch.where(live, t - torch.log(u) * inv_maj, t)
        live = live & (t < leave)
        rho, tmp = sample(t)
        now = live & (next_f64(s, live) * majorant < rho * scale)
        hit[now] = 1
        for x, v in zip(got, (t, rho, tmp)):
            x[now] = v[now]
        live = live & ~now
    return {"transmittance": _host(tr), "hit": _host(hit), "t": _host(got[0]),
            "density": _host(got[1]), "temperature": _host(got[2])}


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        return None  # its noise is one serial generator per plume: too long in plain numpy
    if kind == "rays":
        return _exact_rays(case, seed)
    ref = _Ref(case)
    shape = ref.f[0].shape
    if kind == "pressure":
        b = _rhs(case, seed).reshape(shape)[1:-1, 1:-1, 1:-1].contiguous()
        p, res = ref.cg(b, torch.zeros_like(b), case["iters"], 0.0)
        out = torch.zeros(shape, dtype=torch.float64, device="cuda")
        out[1:-1, 1:-1, 1:-1] = p
        return {"pressure": out.reshape(-1), "residual": res}
    if kind == "adjoint":
        u, v, w, amp, _ = _adjoint_inputs(case, seed)
        for a, x in enumerate((u, v, w)):
            ref.f[a] = x.reshape(shape).clone()
        inner = {"solver": "cg", "iters": 2000, "rel_tol": 1e-10, **case}
        for n in range(case["steps"]):
            ref.step(inner, n * _dt(case), _dt(case), _knobs(case), amp.reshape(shape))
        # the gradients' limiter branches have no 64-bit value of their own
        return {"rho": _host(ref.f[3].reshape(-1)), "grads": [None] * 4}
    for a, x in enumerate(_uniform(case, seed, 3, -0.01, 0.01)):
        ref.f[a] = x.reshape(shape)
    ref.walls(ref.f)
    t, dt, tel = 0.0, _dt(case), []
    for n in range(case["steps"]):
        now = t if case["each"] else n * dt
        tel.append(ref.step(case, now, dt, _knobs(case), source=case["source"]))
        t += dt
    out = {"telemetry": np.array(tel)}
    if case["read"] == "state":
        names = ("u", "v", "w", "density", "temperature")
        out.update({k: _host(x.reshape(-1)) for k, x in zip(names, ref.f)})
    else:
        out.update(density=_host(ref.f[3].reshape(-1)), temperature=_host(ref.f[4].reshape(-1)),
                   max=max(ref.f[3].max().item(), 0.0))
    return {k: (np.asarray(v) if case["precision"] == "mixed" else v) for k, v in out.items()}
