"""Performance cases of the WCSPH step.

Each case is one call that a program makes of this framework, through its
public entry points (``sph.core``, ``sph.state``, ``sph.batch``,
``sph.adjoint``), over the range of scenes, sizes, kernels, precision forms
and integrators that it takes:

* ``run``       steps from a given state, launched one by one (``core.run``),
                as ``Solver.run`` and ``Solver.step`` do;
* ``graph``     the same steps replayed from a CUDA graph
                (``core.StepGraph``), as a long simulation does;
* ``eval``      one derivative evaluation (``core.compute``), the work of
                ``Solver._compute``;
* ``ensemble``  steps of many independent tanks at once
                (``batch.Ensemble.capture``);
* ``adjoint``   a wall-load loss and its gradients
                (``adjoint.WallLoadLoss``), forward and backward;
* ``probe``     a neighbour build and the density and pressure at a set of
                points (``core.nn_update``, ``core.probe_density``).

Scenes are a dam break (an nx x ny column in a tank 4x its width and 1.5x its
height, two wall layers at dx/2) and an all-fluid lattice, both with seeded
jitter and velocities.  Steps start from the same state in every pass.

The FP64 form's results are returned as they are.  The mixed form holds
positions, densities and dt in FP64 and sums velocities' rates in FP32: what
it computed in FP32 is returned as FP32, which is how a program that chose
the form for its speed reads it.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (ROOT, os.path.join(ROOT, "offshore-sph_gb300")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

from sph import adjoint, batch, core, state  # noqa: E402
from sph.Common import particle_dtype  # noqa: E402

DEV = "cuda"
F64 = torch.float64
KERNELS = {"cubic": 0, "gaussian": 1, "wendland": 2}
INTEGRATORS = {"pec": 0, "euler": 1, "verlet": 2}
RHO0, GRAV, ALPHA, EPS, GAMMA = 1000.0, 9.81, 0.01, 0.5, 7.0
CFL_F = 0.25


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _scene(kind, scene, nx, ny, dx, kernel="cubic", precision="fp64", integrator="pec", xsph=False,
           sumdens=False, fixed_h=True, steps=1):
    return dict(kind=kind, scene=scene, nx=nx, ny=ny, dx=dx, kernel=kernel, precision=precision,
                integrator=integrator, xsph=xsph, sumdens=sumdens, fixed_h=fixed_h, steps=steps)


def listed():
    return [
        # the smallest call: one step of a toy tank, as an interactive run or
        # one that exports every step makes it (latency and launches)
        dict(_scene("run", "tank", 8, 16, 0.025), name="step_tank128_fp64"),
        # the reference's own size (3200 fluid particles, the configuration
        # its CPU code runs), the drop-in default form, a chunk of steps
        dict(_scene("run", "tank", 40, 80, 0.025, steps=20), name="run_tank3200_fp64"),
        # the same scene in the mixed form, replayed from a graph
        dict(_scene("graph", "tank", 40, 80, 0.025, precision="mixed", steps=20), name="graph_tank3200_mixed"),
        # one derivative evaluation of 1M particles, mixed form
        dict(_scene("eval", "lattice", 1000, 1000, 0.01, precision="mixed"), name="eval_lattice1m_mixed"),
        # one FP64 evaluation with the Gaussian on an odd-sized lattice (the
        # reference's truncated stencil)
        dict(_scene("eval", "lattice", 317, 313, 0.01, kernel="gaussian"), name="eval_lattice99k_gauss_fp64"),
        # Gaussian with XSPH in the mixed form, launched step by step
        dict(_scene("run", "lattice", 523, 479, 0.01, kernel="gaussian", precision="mixed", xsph=True, steps=8),
             name="run_lattice250k_gauss_xsph_mixed"),
        # the reference's default of a smoothing length from the density
        # (no fixed h), with the Wendland kernel, FP64
        dict(_scene("run", "tank", 157, 321, 0.01, kernel="wendland", fixed_h=False, steps=4),
             name="run_tank50k_wendland_dynh_fp64"),
        # the flagship: a 1M-particle dam break, mixed form, graph replay
        dict(_scene("graph", "tank", 707, 1414, 0.01, precision="mixed", steps=20), name="graph_tank1m_mixed"),
        # the same scene in the drop-in default form
        dict(_scene("run", "tank", 707, 1414, 0.01, steps=4), name="run_tank1m_fp64"),
        # 256 uneven tanks at once, as a parameter study runs them
        dict(kind="ensemble", count=256, dx_lo=0.02, dx_hi=0.05, steps=10, name="ensemble256_mixed"),
        # gradients of the wall load through 40 steps of a 20k-particle column
        dict(kind="adjoint", nx=100, ny=200, dx=0.01, steps=40, checkpoint=20, precision="fp64",
             name="adjoint_tank20k_fp64"),
        # pressure gauges: a neighbour build and 2000 probe points
        dict(kind="probe", nx=317, ny=631, dx=0.01, points=2000, name="probe_tank200k"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    what = rng.choice(["steps"] * 6 + ["eval"] * 2 + ["ensemble", "adjoint", "probe"])
    if what == "ensemble":
        return dict(kind="ensemble", count=int(_log(rng, 8, 256)), dx_lo=0.02 + 0.01 * rng.random(),
                    dx_hi=0.04 + 0.01 * rng.random(), steps=rng.randint(2, 10))
    if what == "adjoint":
        ny = int(_log(rng, 30, 200))
        return dict(kind="adjoint", nx=max(10, int(ny * rng.uniform(0.3, 0.5))), ny=ny, dx=2.0 / ny,
                    steps=rng.randint(8, 40), checkpoint=rng.choice([5, 10, 20]),
                    precision=rng.choice(["fp64", "mixed"]))
    if what == "probe":
        n = _log(rng, 1e3, 1e6)
        nx = max(8, int(math.sqrt(n / 2) * rng.uniform(0.7, 1.4)))
        return dict(kind="probe", nx=nx, ny=max(8, int(n / nx)), dx=0.01, points=int(_log(rng, 1, 20000)))
    precision = rng.choice(["fp64", "mixed"])
    scene = rng.choice(["tank", "tank", "lattice"])
    n = _log(rng, 300, 1e6)
    nx = max(8, int(math.sqrt(n / (2 if scene == "tank" else 1)) * rng.uniform(0.7, 1.4)))
    ny = max(8, int(n / nx))
    kernel = rng.choice(["cubic", "cubic", "gaussian", "wendland"])
    xsph = rng.random() < 0.25
    sumdens = rng.random() < 0.1
    fixed_h = rng.random() < 0.7
    # no more than the work of the largest listed case
    cost = nx * ny * (2.5 if kernel == "gaussian" else 1.0) * (8 if precision == "fp64" else 1)
    steps = 1 if what == "eval" else max(1, min(rng.randint(1, 20), int(3.2e7 / cost)))
    return _scene("eval" if what == "eval" else rng.choice(["run", "graph"]), scene, nx, ny, rng.choice([0.01, 0.025]),
                  kernel=kernel, precision=precision,
                  integrator="pec" if what == "eval" else rng.choice(["pec", "pec", "pec", "euler", "verlet"]),
                  xsph=xsph, sumdens=sumdens, fixed_h=fixed_h, steps=steps)


# ---------------------------------------------------------------------------
# scenes (on the GPU, from the seed alone)
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _uniform(n, lo, hi, g):
    return lo + (hi - lo) * torch.rand(n, dtype=F64, device=DEV, generator=g)


def _normal(n, s, g):
    return s * torch.randn(n, dtype=F64, device=DEV, generator=g)


def _grid(xs, ys):
    x, y = torch.meshgrid(xs, ys, indexing="ij")
    return x.reshape(-1), y.reshape(-1)


def _range(n):
    return torch.arange(n, dtype=F64, device=DEV)


def _tank(nx, ny, dx, g, side="left"):
    """Column, then floor, left and right wall: label, m, rho, x, y, vx, vy."""
    s, layers = dx / 2, 2
    width, tank_w, tank_h = nx * dx, 4 * nx * dx, 1.5 * ny * dx
    fx, fy = _grid((_range(nx) + 0.5) * dx, (_range(ny) + 0.5) * dx)
    if side == "right":
        fx = fx + (tank_w - width)
    nf = nx * ny
    fx = fx + _uniform(nf, -0.02 * dx, 0.02 * dx, g)
    fy = fy + _uniform(nf, -0.02 * dx, 0.02 * dx, g)
    nbx, nby = int(round(tank_w / s)), int(round(tank_h / s)) + layers
    off = -(_range(layers) + 0.5) * s
    wy = (_range(nby) + 0.5) * s - layers * s
    walls = [_grid((_range(nbx) + 0.5) * s, off), _grid(off, wy), _grid(tank_w - off, wy)]
    x = torch.cat([fx] + [w[0] for w in walls])
    y = torch.cat([fy] + [w[1] for w in walls])
    n = x.numel()
    z = torch.zeros(n - nf, dtype=F64, device=DEV)
    label = torch.ones(n, dtype=torch.int8, device=DEV)
    label[:nf] = 0
    full = lambda v: torch.cat([torch.full((nf,), v, dtype=F64, device=DEV), z])  # noqa: E731
    return dict(label=label, m=full(RHO0 * dx * dx), rho=full(RHO0), x=x, y=y,
                vx=torch.cat([_normal(nf, 0.01, g), z]), vy=torch.cat([_normal(nf, 0.01, g), z]))


def _lattice(nx, ny, dx, g):
    n = nx * ny
    x, y = _grid((_range(nx) + 0.5) * dx, (_range(ny) + 0.5) * dx)
    return dict(label=torch.zeros(n, dtype=torch.int8, device=DEV),
                m=torch.full((n,), RHO0 * dx * dx, dtype=F64, device=DEV),
                rho=RHO0 * (1.0 + _uniform(n, -0.01, 0.01, g)),
                x=x + _uniform(n, -0.05 * dx, 0.05 * dx, g), y=y + _uniform(n, -0.05 * dx, 0.05 * dx, g),
                vx=_normal(n, 0.1, g), vy=_normal(n, 0.1, g))


def _inputs(case, seed):
    g = _gen(seed)
    return (_tank if case["scene"] == "tank" else _lattice)(case["nx"], case["ny"], case["dx"], g)


def _cfl(case):
    return 0.3 if case["scene"] == "tank" else 0.25


def _ensemble(case, seed):
    """Per tank: (particle array, dict(height, dx)), the columns and spacings
    drawn with the count alone, the positions and velocities from the seed."""
    shape = np.random.default_rng(case["count"])
    rng = np.random.default_rng(int(seed))
    out = []
    for _ in range(case["count"]):
        w, h = shape.uniform(0.5, 2.0), shape.uniform(1.0, 3.0)
        dx = float(shape.uniform(case["dx_lo"], case["dx_hi"]))
        nx, ny = max(1, int(round(w / dx))), max(1, int(round(h / dx)))
        s, tank_w, tank_h = dx / 2, 4 * nx * dx, 1.5 * ny * dx
        nf = nx * ny
        gx, gy = np.meshgrid((np.arange(nx) + 0.5) * dx, (np.arange(ny) + 0.5) * dx, indexing="ij")
        off = -(np.arange(2) + 0.5) * s
        bx = (np.arange(int(round(tank_w / s))) + 0.5) * s
        wy = (np.arange(int(round(tank_h / s)) + 2) + 0.5) * s - 2 * s
        walls = [np.meshgrid(a, b, indexing="ij") for a, b in ((bx, off), (off, wy), (tank_w - off, wy))]
        x = np.concatenate([gx.ravel()] + [a.ravel() for a, _ in walls])
        y = np.concatenate([gy.ravel()] + [b.ravel() for _, b in walls])
        pa = np.zeros(len(x), dtype=particle_dtype)
        pa["x"], pa["y"] = x, y
        pa["label"][nf:] = 1
        pa["m"][:nf] = RHO0 * dx * dx
        pa["rho"][:nf] = RHO0
        for k in ("x", "y"):
            pa[k][:nf] += rng.uniform(-0.02 * dx, 0.02 * dx, nf)
        for k in ("vx", "vy"):
            pa[k][:nf] = rng.normal(0.0, 0.01, nf)
        out.append((pa, dict(height=ny * dx, dx=dx)))
    return out


# ---------------------------------------------------------------------------
# the framework's calls
# ---------------------------------------------------------------------------
def _device_state(f, wc, cfg, hydrostatic):
    dp = state.DeviceParticles(f["x"].numel())
    dp.label.copy_(f["label"])
    for k, v in f.items():
        if k != "label":
            dp.fields[k].copy_(v)
    rho = dp.rho.clone()
    core.initialize(dp, wc, cfg)  # h, hydrostatic rho, p and c of the fluid
    if not hydrostatic:
        dp.rho.copy_(rho)
        core.eos(dp, wc)
    return dp


def _wcsph(case):
    return core.wcsph_struct(case["ny"] * case["dx"], case["dx"], RHO0, use_xsph=case.get("xsph", False),
                             use_summation_density=case.get("sumdens", False))


def _config(case):
    return core.config_struct(kernel=KERNELS[case["kernel"]], precision=case["precision"],
                              integrator=INTEGRATORS[case["integrator"]], pec_use_xsph=case["xsph"],
                              h_fixed=1.3 * case["dx"] if case["fixed_h"] else 0.0, cfl_c=_cfl(case), cfl_f=CFL_F)


class _S:
    pass


def prepare(case, seed):
    s = _S()
    s.case = case
    kind = case["kind"]
    if kind == "ensemble":
        s.E = batch.Ensemble(_ensemble(case, seed))
        s.snap = s.E.snapshot()
        s.graph = s.E.capture(case["steps"])
        return s
    if kind == "adjoint":
        f = _tank(case["nx"], case["ny"], case["dx"], _gen(seed), side="right")
        pa = np.zeros(f["x"].numel(), dtype=particle_dtype)
        for k, v in f.items():
            pa[k] = v.cpu().numpy()
        s.wl = adjoint.WallLoadCase(pa, height=case["ny"] * case["dx"], r0=case["dx"], h=1.3 * case["dx"],
                                    dt=_adjoint_dt(case), nsteps=case["steps"],
                                    wall_x=4 * case["nx"] * case["dx"], checkpoint=case["checkpoint"],
                                    adjoint_precision=case["precision"])
        s.alpha = torch.tensor(ALPHA, dtype=F64, device=DEV, requires_grad=True)
        s.pos = s.wl.positions().requires_grad_(True)
        s.vel = s.wl.velocities().requires_grad_(True)
        return s
    if kind == "probe":
        f = _tank(case["nx"], case["ny"], case["dx"], _gen(seed))
        h = 1.3 * case["dx"]
        s.wc = core.wcsph_struct(case["ny"] * case["dx"], case["dx"], RHO0)
        s.cfg = core.config_struct(h_fixed=h)
        s.dp = _device_state(f, s.wc, s.cfg, True)
        s.ws = state.DeviceWorkspace(s.dp.n)
        s.px, s.py = _points(case, seed)
        s.h = torch.full_like(s.px, h)
        return s
    f = _inputs(case, seed)
    s.wc, s.cfg = _wcsph(case), _config(case)
    s.dp = _device_state(f, s.wc, s.cfg, case["scene"] == "tank")
    s.ws = state.DeviceWorkspace(s.dp.n)
    if kind != "eval":
        s.start = s.dp._buf.clone()
        if kind == "graph":
            s.graph = core.StepGraph(s.dp, s.wc, s.cfg, s.ws, case["steps"])
        else:
            s.hist = torch.zeros((case["steps"], 3), dtype=F64, device=DEV)
    return s


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "ensemble":
        s.E.restore(s.snap)
        s.graph.replay()
        f = s.E.dp.fields
        return {**{k: f[k] for k in ("x", "y", "rho")}, **{k: f[k].float() for k in ("vx", "vy", "ax", "ay", "drho")}}
    if kind == "adjoint":
        loss = adjoint.WallLoadLoss.apply(s.alpha, s.pos, s.vel, s.wl)
        ga, gp, gv = torch.autograd.grad(loss, (s.alpha, s.pos, s.vel))
        if case["precision"] == "mixed":
            ga, gp, gv = ga.float(), gp.float(), gv.float()
        return {"loss": loss.detach(), "alpha": ga, "pos": gp, "vel": gv}
    if kind == "probe":
        core.nn_update(s.dp, s.cfg, s.ws)
        rho, p = core.probe_density(s.dp, s.wc, 0, s.ws, s.px, s.py, s.h, s.h)
        return {"rho": rho, "p": p}
    out = {}
    if kind == "eval":
        core.compute(s.dp, s.wc, s.cfg, s.ws)
        keep, rates = ("h",), ("p", "ax", "ay", "drho")
    else:
        s.dp._buf.copy_(s.start)
        if kind == "graph":
            s.graph.replay()
        else:
            core.run(s.dp, s.wc, s.cfg, s.ws, case["steps"], s.hist)
            out["dt"] = s.hist
        keep, rates = ("x", "y", "rho"), ("vx", "vy", "ax", "ay", "drho", "p")
    if case["xsph"]:
        rates += ("xsphx", "xsphy")
    if case["precision"] == "mixed":
        # FP32: the pair sums, h from the density, a summed density
        low = set(rates) | {"h", "dt"} | ({"rho"} if case["sumdens"] else set())
    else:
        low = set()
    for k in keep + rates:
        out[k] = s.dp.fields[k]
    return {k: v.float() if k in low else v for k, v in out.items()}


# ---------------------------------------------------------------------------
# the work that a pass cannot do without
# ---------------------------------------------------------------------------
def _counts(case):
    """(fluid, all) particles."""
    nf = case["nx"] * case["ny"]
    if case.get("scene") == "lattice":
        return nf, nf
    s = case["dx"] / 2
    nb = int(round(4 * case["nx"] * case["dx"] / s)) * 2 + 4 * (int(round(1.5 * case["ny"] * case["dx"] / s)) + 2)
    return nf, nf + nb


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        shape = np.random.default_rng(case["count"])
        nf = n = 0
        for _ in range(case["count"]):
            w, h = shape.uniform(0.5, 2.0), shape.uniform(1.0, 3.0)
            dx = float(shape.uniform(case["dx_lo"], case["dx_hi"]))
            a, b = _counts(dict(nx=max(1, int(round(w / dx))), ny=max(1, int(round(h / dx))), dx=dx))
            nf, n = nf + a, n + b
        return {"bytes": 385 * n * case["steps"], "flops": 21 * 40 * nf * case["steps"]}
    nf, n = _counts(case)
    if kind == "adjoint":
        # forward, the replay and the adjoint step, each over the state
        return {"bytes": (2 * 385 + 400) * n * case["steps"], "flops": 21 * (2 * 40 + 90) * nf * case["steps"]}
    if kind == "probe":
        return {"bytes": (8 * 3 + 1) * n + 21 * 33 * case["points"] + 40 * case["points"],
                "flops": 21 * 30 * case["points"]}
    pairs = 48 if case["kernel"] == "gaussian" else 21
    flops = pairs * (40 + (10 if case["xsph"] else 0) + (15 if case["sumdens"] else 0))
    if kind == "eval":
        # m, rho, x, y, vx, vy, h and the label in; p, c, h, drho, ax, ay and
        # the XSPH velocity out
        return {"bytes": 121 * n, "flops": flops * nf}
    # a step: dt 32, predict 144, build 24, pair 81, correct 104
    return {"bytes": 385 * n * case["steps"], "flops": flops * nf * case["steps"]}


# ---------------------------------------------------------------------------
# the same results in plain FP64 torch
# ---------------------------------------------------------------------------
def _adjoint_dt(case):
    return 0.24 * 1.3 * case["dx"] / (10.0 * math.sqrt(2 * GRAV * case["ny"] * case["dx"]))


def _points(case, seed):
    g = _gen(seed + 7919)
    n = case["points"]
    w, h = case["nx"] * case["dx"], case["ny"] * case["dx"]
    return _uniform(n, 0.0, w, g), _uniform(n, 0.0, h, g)


def _w(kernel, r, h):
    q = r / h
    if kernel == "cubic":
        a = 10.0 / (7.0 * math.pi) / (h * h)
        return a * torch.where(q > 1.0, 0.25 * torch.clamp(2.0 - q, min=0.0) ** 3, 1.0 - 1.5 * q * q * (1.0 - 0.5 * q))
    if kernel == "wendland":
        return 9.0 / (4.0 * math.pi) / (h * h) * torch.clamp(1.0 - 0.5 * q, min=0.0) ** 6 * \
            (35.0 / 12.0 * q * q + 3.0 * q + 1.0)
    return 1.0 / (math.pi * h * h) * torch.exp(-q * q) * (q <= 3.0)


def _grad(kernel, r, h):
    """dW/dr / r, for r > 0."""
    q = r / h
    if kernel == "cubic":
        a = 10.0 / (7.0 * math.pi) / (h * h)
        g = torch.where(q > 1.0, -0.75 * torch.clamp(2.0 - q, min=0.0) ** 2, -3.0 * q * (1.0 - 0.75 * q))
        return a * g / (h * r)
    if kernel == "wendland":
        a = 9.0 / (4.0 * math.pi) / (h * h)
        return a * torch.clamp(1.0 - 0.5 * q, min=0.0) ** 5 * (-14.0 / 3.0) * q * (1.0 + 2.5 * q) / (h * r)
    return -2.0 / (math.pi * h ** 4) * torch.exp(-q * q) * (q <= 3.0)


class _Flow:
    """The step's physics over one particle set (inst: the tank of each
    particle, with its own constants, or None)."""

    def __init__(self, f, kernel, height, r0, h_fixed, xsph=False, sumdens=False, inst=None):
        self.f = {k: v.clone() for k, v in f.items()}
        self.kernel, self.inst = kernel, inst
        self.xsph, self.sumdens = xsph, sumdens
        self.r0, self.h_fixed = r0, h_fixed
        self.co = 10.0 * torch.sqrt(2 * GRAV * torch.as_tensor(height, dtype=F64, device=DEV))
        self.B = self.co * self.co * RHO0 / GAMMA
        self.D = 5 * GRAV * torch.as_tensor(height, dtype=F64, device=DEV)
        self.fluid = f["label"] == 0
        n = f["x"].numel()
        self.h = torch.where(self.fluid, self._new_h(f["m"], f["rho"]), torch.zeros((), dtype=F64, device=DEV))
        for k in ("ax", "ay", "drho", "xsphx", "xsphy"):
            self.f[k] = torch.zeros(n, dtype=F64, device=DEV)
        self.height = torch.as_tensor(height, dtype=F64, device=DEV)

    def hydrostatic(self):
        rho = RHO0 * (1.0 + RHO0 * GRAV * (self.height - self.f["y"]) / self.B) ** (1.0 / GAMMA)
        self.f["rho"] = torch.where(self.fluid, rho, self.f["rho"])

    def _new_h(self, m, rho):
        if self.h_fixed is not None:
            return torch.as_tensor(self.h_fixed, dtype=F64, device=DEV).expand(m.shape)
        return 1.3 * torch.sqrt(m / torch.where(rho > 1e-12, rho, torch.ones_like(rho)))

    def _pairs(self, x, y, h_old, h, qx=None, qy=None, qh=None):
        """Chunks (queries, i, j) of the pairs within the interaction radius
        and the 3x3 stencil of the reference's cells."""
        support = 3.0 if self.kernel == "gaussian" else 2.0
        hm = float(h.max())
        R = max(support * hm, min(float(torch.as_tensor(self.r0).max()), 3.0 * hm)) * (1 + 1e-9)
        ox, oy = float(x.min()), float(y.min())
        cx, cy = torch.floor((x - ox) / R).long(), torch.floor((y - oy) / R).long()
        nx, ny = int(cx.max()) + 3, int(cy.max()) + 3
        base = torch.zeros_like(cx) if self.inst is None else self.inst * (nx * ny)
        key, order = torch.sort(base + (cy + 1) * nx + cx + 1)
        cs = float(h_old.min()) * 2.0
        cs = 1.0 if cs < 1e-6 else cs
        # the reference's stencil cuts pairs only where its cells are smaller
        # than the interaction radius
        cut = cs < R * (1 + 1e-6)
        if qx is None:
            queries = torch.nonzero(self.fluid).squeeze(1)
            ax, ay, ah, abase = x, y, h, base
        else:
            queries = torch.arange(qx.numel(), device=DEV)
            ax, ay, ah, abase = qx, qy, qh, torch.zeros(qx.numel(), dtype=torch.long, device=DEV)
        acx, acy = torch.floor((ax - ox) / R).long(), torch.floor((ay - oy) / R).long()
        if cut:
            rx, ry = torch.floor((x - ox) / cs), torch.floor((y - oy) / cs)
            arx, ary = torch.floor((ax - ox) / cs), torch.floor((ay - oy) / cs)
        for c in torch.split(queries, 100000):
            ii, jj = [], []
            for dy in (-1, 0, 1):
                k0 = abase[c] + (acy[c] + 1 + dy) * nx + acx[c] + 1
                s, e = torch.searchsorted(key, k0 - 1), torch.searchsorted(key, k0 + 1, right=True)
                cnt = e - s
                i = torch.repeat_interleave(c, cnt)
                first = torch.cumsum(cnt, 0) - cnt
                j = order[torch.arange(i.numel(), device=DEV) - torch.repeat_interleave(first - s, cnt)]
                ii.append(i)
                jj.append(j)
            i, j = torch.cat(ii), torch.cat(jj)
            dx, dy = ax[i] - x[j], ay[i] - y[j]
            r = torch.sqrt(dx * dx + dy * dy)
            hij = 0.5 * (ah[i] + h[j])
            ok = r <= 3.0 * hij
            if qx is None:
                ok &= i != j
            if cut:
                ok &= ((arx[i] - rx[j]).abs() <= 1) & ((ary[i] - ry[j]).abs() <= 1)
            yield c, i[ok], j[ok]

    def evaluate(self, alpha=ALPHA, wall_x=None):
        """h reset, EOS and the derivatives of the present state."""
        f, fl = self.f, self.fluid
        x, y, vx, vy, m, rho = (f[k] for k in ("x", "y", "vx", "vy", "m", "rho"))
        h_old = self.h
        with torch.no_grad():
            self.h = torch.where(fl, self._new_h(m, rho), self.h)
        h = self.h
        one = torch.ones_like(rho)
        p = torch.where(fl, self.B * ((rho / RHO0) ** GAMMA - 1.0), torch.zeros_like(rho))
        per = (lambda v, i: v[i] if torch.is_tensor(v) and v.dim() else v)
        with torch.no_grad():
            chunks = list(self._pairs(x, y, h_old, h))
        if self.sumdens:
            new = torch.zeros_like(rho)
            w0 = m * _w(self.kernel, torch.zeros_like(h), torch.where(fl, h, one))
            for _, i, j in chunks:
                k = fl[j]
                i, j = i[k], j[k]
                r = torch.sqrt((x[i] - x[j]) ** 2 + (y[i] - y[j]) ** 2)
                new = new.index_add(0, i, m[j] * _w(self.kernel, r, 0.5 * (h[i] + h[j])))
            rho = f["rho"] = torch.where(fl, new + w0, rho)
        rs = torch.where(fl, rho, one)
        oth = p / (rs * rs)
        ax, ay, dr, sx, sy = (torch.zeros_like(x) for _ in range(5))
        load = torch.zeros((), dtype=F64, device=DEV)
        for _, i, j in chunks:
            b = ~fl[j]
            bi, bj = i[b], j[b]
            i, j = i[~b], j[~b]
            dx, dy = x[i] - x[j], y[i] - y[j]
            d2 = dx * dx + dy * dy
            r = torch.sqrt(d2)
            hij = 0.5 * (h[i] + h[j])
            g = _grad(self.kernel, r, hij)
            dvx, dvy = vx[i] - vx[j], vy[i] - vy[j]
            dot = dvx * dx + dvy * dy
            hb = 0.5 * (h[i] + hij)
            mu = hb * dot / (d2 + 0.01 * hb * hb)
            PI = torch.where(dot < 0.0, -alpha * 0.5 * per(self.co, i) * mu / (0.5 * (rs[i] + rs[j])),
                             torch.zeros_like(mu))
            S = oth[i] + oth[j] + PI
            ax = ax.index_add(0, i, -m[j] * S * g * dx)
            ay = ay.index_add(0, i, -m[j] * S * g * dy)
            if not self.sumdens:
                dr = dr.index_add(0, i, m[j] * g * dot)
            if self.xsph:
                k = -EPS * m[j] * _w(self.kernel, r, hij) / (0.5 * (rs[i] + rs[j]))
                sx, sy = sx.index_add(0, i, k * dvx), sy.index_add(0, i, k * dvy)
            dx, dy = x[bi] - x[bj], y[bi] - y[bj]
            d2 = dx * dx + dy * dy
            r0 = per(self.r0, bi)
            s2 = r0 * r0 / d2
            fac = torch.where(s2 >= 1.0, per(self.D, bi) * (s2 * s2 - s2) / d2, torch.zeros_like(d2))
            ax, ay = ax.index_add(0, bi, fac * dx), ay.index_add(0, bi, fac * dy)
            if wall_x is not None:
                load = load - (m[bi] * fac * dx * (x[bj] >= wall_x)).sum()
        z = torch.zeros_like(x)
        f["ax"], f["ay"], f["drho"] = ax, torch.where(fl, ay - GRAV, z), dr
        f["xsphx"], f["xsphy"] = (torch.where(fl, vx + sx, z), torch.where(fl, vy + sy, z)) if self.xsph else (z, z)
        f["p"] = p
        return load

    def timestep(self, cfl_c):
        """dt (3,), or per tank (tanks, 3)."""
        h = torch.where(self.fluid, self.h, torch.full_like(self.h, math.inf))
        a2 = torch.where(self.fluid, self.f["ax"] ** 2 + self.f["ay"] ** 2, torch.zeros_like(h))
        if self.inst is None:
            h, a2, co = h.min(), a2.max(), self.co
        else:
            t = int(self.inst.max()) + 1
            h = torch.full((t,), math.inf, dtype=F64, device=DEV).scatter_reduce(0, self.inst, h, "amin")
            a2 = torch.zeros(t, dtype=F64, device=DEV).scatter_reduce(0, self.inst, a2, "amax")
            co = torch.zeros(t, dtype=F64, device=DEV).scatter_reduce(0, self.inst, self.co, "amax")
        c = cfl_c * h / co
        f = torch.where(a2 < 1e-12, torch.full_like(a2, 1e10), CFL_F * torch.sqrt(h / torch.clamp(a2, min=1e-300)))
        return torch.stack([torch.minimum(c, f), c, f], -1)

    def step(self, dt, integrator="pec", alpha=ALPHA, wall_x=None):
        f, fl = self.f, self.fluid
        keep = {k: f[k] for k in ("x", "y", "vx", "vy", "rho")}
        mv = lambda a, d, v: torch.where(fl, a + d * v, a)  # noqa: E731
        drift = ("xsphx", "xsphy") if self.xsph else ("vx", "vy")
        if integrator == "pec":
            a = dict(f)
            for k, v, t in (("x", drift[0], 0.5), ("y", drift[1], 0.5), ("vx", "ax", 0.5), ("vy", "ay", 0.5),
                            ("rho", "drho", 0.5)):
                f[k] = mv(a[k], t * dt, a[v])
        elif integrator == "verlet":
            f["x"], f["y"] = mv(f["x"], 0.5 * dt, f["vx"]), mv(f["y"], 0.5 * dt, f["vy"])
        load = self.evaluate(alpha, wall_x)
        if integrator == "pec":
            x, y = mv(keep["x"], dt, f[drift[0]]), mv(keep["y"], dt, f[drift[1]])
            f["x"], f["y"] = x, y
            f["vx"], f["vy"] = mv(keep["vx"], dt, f["ax"]), mv(keep["vy"], dt, f["ay"])
            # a summed density is the evaluation's; the corrector starts from
            # the density before the step
            f["rho"] = mv(keep["rho"], dt, f["drho"])
        elif integrator == "euler":
            f["x"] = mv(mv(f["x"], dt, f["vx"]), 0.5 * dt * dt, f["ax"])
            f["y"] = mv(mv(f["y"], dt, f["vy"]), 0.5 * dt * dt, f["ay"])
            f["vx"], f["vy"] = mv(f["vx"], dt, f["ax"]), mv(f["vy"], dt, f["ay"])
            f["rho"] = mv(f["rho"], dt, f["drho"])
        else:
            f["vx"], f["vy"] = mv(f["vx"], dt, f["ax"]), mv(f["vy"], dt, f["ay"])
            f["x"], f["y"] = mv(f["x"], 0.5 * dt, f[drift[0]]), mv(f["y"], 0.5 * dt, f[drift[1]])
        return load


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        tanks = _ensemble(case, seed)
        inst = torch.repeat_interleave(torch.arange(len(tanks), device=DEV),
                                       torch.tensor([len(pa) for pa, _ in tanks], device=DEV))
        per = lambda k: torch.tensor([c[k] for _, c in tanks], dtype=F64, device=DEV)[inst]  # noqa: E731
        f = {k: torch.from_numpy(np.concatenate([pa[k] for pa, _ in tanks])).to(DEV)
             for k in ("label", "m", "rho", "x", "y", "vx", "vy")}
        flow = _Flow(f, "cubic", per("height"), per("dx"), 1.3 * per("dx"), inst=inst)
        flow.hydrostatic()
        for _ in range(case["steps"]):
            flow.step(flow.timestep(0.3)[:, 0][inst])
        return {k: flow.f[k] for k in ("x", "y", "rho", "vx", "vy", "ax", "ay", "drho")}
    h = 1.3 * case["dx"] if case.get("fixed_h", True) else None
    height = case["ny"] * case["dx"]
    if kind == "adjoint":
        f = _tank(case["nx"], case["ny"], case["dx"], _gen(seed), side="right")
        flow = _Flow(f, "cubic", height, case["dx"], h)
        flow.hydrostatic()
        fi = torch.nonzero(flow.fluid).squeeze(1)
        alpha = torch.tensor(ALPHA, dtype=F64, device=DEV, requires_grad=True)
        pos = torch.stack((f["x"][fi], f["y"][fi]), 1).requires_grad_(True)
        vel = torch.stack((f["vx"][fi], f["vy"][fi]), 1).requires_grad_(True)
        for k, v in (("x", pos[:, 0]), ("y", pos[:, 1]), ("vx", vel[:, 0]), ("vy", vel[:, 1])):
            flow.f[k] = flow.f[k].index_put((fi,), v)
        dt, loss = _adjoint_dt(case), 0.0
        for _ in range(case["steps"]):
            loss = loss + dt * flow.step(dt, alpha=alpha, wall_x=4 * case["nx"] * case["dx"])
        ga, gp, gv = torch.autograd.grad(loss, (alpha, pos, vel))
        return {"loss": loss.detach(), "alpha": ga, "pos": gp, "vel": gv}
    if kind == "probe":
        flow = _Flow(_tank(case["nx"], case["ny"], case["dx"], _gen(seed)), "cubic", height, case["dx"], h)
        flow.hydrostatic()
        px, py = _points(case, seed)
        hk = torch.full_like(px, h)
        x, y, m, rho = (flow.f[k] for k in ("x", "y", "m", "rho"))
        num, den = torch.zeros_like(px), torch.zeros_like(px)
        for _, i, j in flow._pairs(x, y, flow.h, flow.h, px, py, hk):
            k = flow.fluid[j]
            i, j = i[k], j[k]
            w = _w("cubic", torch.sqrt((px[i] - x[j]) ** 2 + (py[i] - y[j]) ** 2), hk[i])
            num, den = num.index_add(0, i, m[j] * w), den.index_add(0, i, w * m[j] / rho[j])
        out = num / den
        return {"rho": out, "p": ((out / RHO0) ** GAMMA - 1.0) * flow.B}
    flow = _Flow(_inputs(case, seed), case["kernel"], height, case["dx"], h, case["xsph"], case["sumdens"])
    if case["scene"] == "tank":
        flow.hydrostatic()
    if kind == "eval":
        flow.evaluate()
        out = {k: flow.f[k] for k in ("p", "ax", "ay", "drho")}
        out["h"] = flow.h
    else:
        hist = []
        for _ in range(case["steps"]):
            hist.append(flow.timestep(_cfl(case)))
            flow.step(hist[-1][0], case["integrator"])
        out = {k: flow.f[k] for k in ("x", "y", "rho", "vx", "vy", "ax", "ay", "drho", "p")}
        if kind == "run":
            out["dt"] = torch.stack(hist)
    if case["xsph"]:
        out["xsphx"], out["xsphy"] = flow.f["xsphx"], flow.f["xsphy"]
    return out
