"""Performance cases: what users of this package have it do, through its public entry points.

Five kinds of work, each over the sizes of the package's own workloads and tests:

* ``solve``: a single instance stepped from its initial condition by
  ``B200SpectralSolver`` -- straight tracks (constant properties, one forcing pass per
  step), nonlinear rasters and the temperature-dependent example (latent heat, property
  correction, Picard to a tolerance), box tracks (latent heat on a laser-following fine
  box) -- in FP64 or in mixed precision, step by step or as one device-resident run;
* ``batch``: many cuboids of uneven size stepped together by ``BatchSolver`` or
  ``LaneBatch``, in mixed precision or FP64, one forcing pass or a Picard loop per step;
* ``dct``: the backend's ``DCT_II`` / ``IDCT_II`` pair on a field;
* ``nodal``: the node-centred output field of a set of modes.

``exact`` restates the same work in plain torch FP64.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from spectral_galerkin_heat_b200 import B200SpectralSolver, SimulationContext, kernels, workloads
from spectral_galerkin_heat_b200.batch import BatchSolver, LaneBatch
from spectral_galerkin_heat_b200.laser import RasterPath, StraightTrack

UM = 1e-6


def listed():
    return [
        # the smallest solve: a single short track stepped call by call, as a host loop
        # that reads the metrics of every step does; bound by latency and launches
        dict(name="track_64x32x16", kind="solve", form="track", nx=64, ny=32, nz=16, steps=8,
             precision="fp64", by_step=True, tol=0.0, cap=1),
        # a large track run device-resident, metrics read at the end (the precision study's grid)
        dict(name="track_256x128x64", kind="solve", form="track", nx=256, ny=128, nz=64, steps=6,
             precision="fp64", by_step=False, tol=0.0, cap=1),
        # the full nonlinear raster, Picard to 1e-8: about a hundred volume iterations per step
        dict(name="raster_128x64x32", kind="solve", form="raster", nx=128, ny=64, nz=32, steps=2,
             precision="fp64", by_step=True, tol=1e-8, cap=400),
        # the same raster in mixed precision at the tolerance that form converges to
        dict(name="raster_mixed_128x64x32", kind="solve", form="raster", nx=128, ny=64, nz=32, steps=3,
             precision="mixed", by_step=True, tol=1e-5, cap=400),
        # distinct temperature-dependent phases, latent heat and property correction at a
        # ragged grid-mode size
        dict(name="tdep_75x45x37", kind="solve", form="tdep", nx=75, ny=45, nz=37, steps=4,
             precision="fp64", by_step=True, tol=1e-4, cap=80),
        # the production layout for large pools: latent heat on a laser-following fine box
        dict(name="box_80x48x120", kind="solve", form="box", nx=80, ny=48, nz=120, steps=4,
             precision="fp64", by_step=True, tol=1e-4, cap=30),
        # a serving chunk: every class of the request mix in flight, two lanes, mixed precision
        dict(name="serving_mixed_48", kind="batch", mix="serving", per_class=4, largest=512, precision="mixed",
             lanes=2, steps=5, tol=0.0, cap=1, dt=5e-6),
        # the same chunk of the smaller classes in FP64, for users who need the plain form
        dict(name="serving_fp64_18", kind="batch", mix="serving", per_class=2, largest=256, precision="fp64",
             lanes=1, steps=6, tol=0.0, cap=1, dt=5e-6),
        # a parameter study: uneven cuboids with the Picard loop at the reference defaults
        dict(name="uneven_mixed_32", kind="batch", mix="uneven", slots=32, largest=256, precision="mixed",
             lanes=1, steps=3, tol=1e-4, cap=30, dt=5e-6),
        # a handful of small ragged cuboids: batch stepping at its smallest
        dict(name="ragged_mixed_4", kind="batch", mix="ragged", slots=4, largest=64, precision="mixed",
             lanes=1, steps=8, tol=1e-4, cap=30, dt=5e-6),
        # the transform pair of the backend on an odd-sized volume
        dict(name="dct_96x60x100", kind="dct", dims=3, n0=96, n1=60, n2=100),
        # full-volume output at the largest serving grid
        dict(name="nodal_512x256x64", kind="nodal", nx=512, ny=256, nz=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["track", "raster", "tdep", "box", "batch", "batch", "batch", "dct", "nodal"])
    if kind == "track":
        nx = _log(rng, 24, 256)
        return dict(kind="solve", form="track", nx=nx, ny=max(8, nx // 2 + rng.randint(-3, 3)), nz=_log(rng, 6, 64),
                    steps=rng.randint(3, 8), precision="fp64", by_step=rng.random() < 0.5, tol=0.0, cap=1)
    if kind == "raster":
        nx = _log(rng, 32, 128)
        mixed = rng.random() < 0.3
        return dict(kind="solve", form="raster", nx=nx, ny=nx // 2 + rng.randint(-2, 2), nz=_log(rng, 10, 32),
                    steps=2, precision="mixed" if mixed else "fp64", by_step=rng.random() < 0.5,
                    tol=1e-5 if mixed else rng.choice([1e-6, 1e-8]), cap=400)
    if kind == "tdep":
        nx = _log(rng, 30, 100)
        return dict(kind="solve", form="tdep", nx=nx, ny=max(12, int(0.6 * nx)), nz=_log(rng, 16, 64),
                    steps=rng.randint(2, 4), precision="fp64", by_step=rng.random() < 0.5, tol=1e-4, cap=80)
    if kind == "box":
        nx = _log(rng, 40, 80)
        return dict(kind="solve", form="box", nx=nx, ny=int(0.6 * nx) + rng.randint(0, 2), nz=_log(rng, 40, 120),
                    steps=rng.randint(2, 4), precision="fp64", by_step=rng.random() < 0.5, tol=1e-4, cap=30)
    if kind == "batch":
        mix = rng.choice(["serving", "uneven", "ragged"])
        mixed = rng.random() < 0.75
        c = dict(kind="batch", mix=mix, precision="mixed" if mixed else "fp64", dt=5e-6)
        if mix == "serving":
            c.update(per_class=rng.randint(1, 4) if mixed else rng.randint(1, 2),
                     largest=rng.choice([128, 256, 512]) if mixed else rng.choice([128, 256]),
                     lanes=rng.choice([1, 2]), steps=rng.randint(3, 5), tol=0.0, cap=1)
        elif mix == "uneven":
            c.update(slots=_log(rng, 4, 32), largest=rng.choice([128, 192, 256]), lanes=1, steps=rng.randint(2, 3),
                     tol=1e-4, cap=30)
        else:
            c.update(slots=_log(rng, 1, 16), largest=rng.choice([48, 64, 100]), lanes=1, steps=rng.randint(4, 8),
                     tol=1e-4, cap=30)
        return c
    if kind == "dct":
        dims = rng.choice([1, 2, 3, 3])
        if dims == 1:
            return dict(kind="dct", dims=1, n0=_log(rng, 64, 1024), n1=1, n2=1)
        if dims == 2:
            return dict(kind="dct", dims=2, n0=_log(rng, 16, 256), n1=_log(rng, 32, 512), n2=1)
        return dict(kind="dct", dims=3, n0=_log(rng, 6, 100), n1=_log(rng, 16, 128), n2=_log(rng, 24, 256))
    nx = _log(rng, 32, 400)
    return dict(kind="nodal", nx=nx, ny=max(8, nx // 2 + rng.randint(-3, 3)), nz=_log(rng, 8, 64))


# ---------------------------------------------------------------------------
# the cases as configurations of the package
# ---------------------------------------------------------------------------

def _solve_inputs(case, seed):
    """``(cfg, path)`` of a single-instance solve; power, speed and position from the seed."""
    r = np.random.default_rng([7, int(seed)])
    nx, ny, nz, steps = case["nx"], case["ny"], case["nz"], case["steps"]
    form = case["form"]
    if form == "track":
        # the 64 x 32 x 16 track's cell size, halved towards the 256 x 128 x 64 grid
        h = 31.25 * UM * (64.0 / max(nx, 64)) ** 0.5
        size = (nx * h, ny * h, nz * h)
        cfg, _ = workloads.straight_track(nx, ny, nz, steps=steps, size=size)
        path = StraightTrack(r.uniform(0.2, 0.4) * size[0], r.uniform(0.4, 0.6) * size[1], r.uniform(0.5, 2.0), 0.0,
                             r.uniform(150.0, 400.0))
    elif form == "raster":
        cfg, path = workloads.nonlinear_raster(nx, ny, nz, steps=steps, seed=int(seed) & 0x7fffffff, tol=case["tol"],
                                               cap=case["cap"], power=r.uniform(150.0, 250.0))
    elif form == "tdep":
        cfg, _ = workloads.example03(nx, ny, nz, steps=steps)
        path = StraightTrack(r.uniform(0.18e-3, 0.3e-3), 0.15e-3, r.uniform(0.1, 0.2), 0.0, r.uniform(22.0, 30.0))
    else:
        cfg, _ = workloads.box_track(nx, ny, nz, steps=steps)
        path = StraightTrack(r.uniform(0.12e-3, 0.3e-3), 0.2e-3, r.uniform(0.3, 0.5), 0.0, r.uniform(100.0, 140.0))
    cfg["simulation"].update({"max_picard_iter": case["cap"]})
    if case["tol"] > 0:
        cfg["simulation"]["picard_tol"] = case["tol"]
    return cfg, path


def _batch_inputs(case, seed):
    """``(cfg, path)`` of every slot of a batch."""
    r = np.random.default_rng([11, int(seed)])
    shapes = np.random.default_rng([13, case.get("slots", 0), case["largest"]])  # the mix itself does not vary
    out = []
    if case["mix"] == "serving":
        grids = [(nx, nx // 2, nz) for nx in (64, 128, 256, 512) if nx <= case["largest"] for nz in (16, 32, 64)]
        grids = [g for g in grids for _ in range(case["per_class"])]
    elif case["mix"] == "uneven":
        grids = []
        for _ in range(case["slots"]):
            nx = int(shapes.choice([n for n in (64, 96, 128, 192, 256) if n <= case["largest"]]))
            grids.append((nx, nx // 2, int(shapes.choice((16, 32, 64)))))
    else:
        grids = []
        for _ in range(case["slots"]):
            nx = int(shapes.integers(24, case["largest"] + 1))
            grids.append((nx, max(8, nx // 2 + int(shapes.integers(-2, 3))), int(shapes.integers(5, 18))))
    for nx, ny, nz in grids:
        if case["mix"] == "serving":
            size = (2e-3, 1e-3, 0.5e-3)
        else:
            size = (2e-3 * nx / 64, 1e-3 * ny / 32, 0.5e-3)
        absorptivity = 0.35 if case["mix"] == "serving" else float(r.uniform(0.3, 0.45))
        cfg, _ = workloads.straight_track(nx, ny, nz, steps=case["steps"], dt=case["dt"], size=size,
                                          absorptivity=absorptivity)
        if case["cap"] > 1:
            cfg["simulation"].update({"max_picard_iter": case["cap"], "picard_omega": 0.1, "picard_tol": case["tol"]})
        # one explicit forcing pass per step amplifies rounding once the surface boils on the
        # fine serving grids; at these powers it evaporates and stays well conditioned
        power = float(r.uniform(60.0, 120.0) if case["mix"] == "serving" else r.uniform(150.0, 400.0))
        speed = float(r.uniform(0.5, 2.0))
        x0, y0 = float(r.uniform(0.2, 0.4)) * size[0], float(r.uniform(0.35, 0.65)) * size[1]
        if case["mix"] == "serving":
            path = RasterPath(0.25e-3, y0, 1.5e-3, 50 * UM, 4, speed, power)
        else:
            path = StraightTrack(x0, y0, speed, 0.0, power)
        out.append((cfg, path))
    return out


def _context(cfg, path):
    ctx = SimulationContext.from_dict(cfg)
    ctx.laser_path = path
    return ctx


def _field(case, seed):
    """A smooth field with a hot spot and some noise, as temperature fields are (FP64)."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) & 0x7fffffff)
    if case["kind"] == "dct":
        shape = [case["n0"], case["n1"], case["n2"]][:case["dims"]]
        x = 300.0 + torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)
        axes = torch.meshgrid(*[torch.linspace(-1, 1, n, device="cuda", dtype=torch.float64) for n in shape],
                              indexing="ij")
        return x + 2000.0 * torch.exp(-8.0 * sum(a * a for a in axes))
    # modes of a temperature field decay with the wave number
    shape = (case["nz"], case["ny"], case["nx"])
    a = torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)
    k2 = sum((torch.arange(n, device="cuda", dtype=torch.float64) / n).view([-1 if i == j else 1 for j in range(3)]) ** 2
             for i, n in enumerate(shape))
    a = a * torch.exp(-6.0 * k2) * 1e-6
    a[0, 0, 0] = 300.0 * math.sqrt(2e-3 * 1e-3 * 0.5e-3)
    return a


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        ctx = _context(*_solve_inputs(case, seed))
        s = B200SpectralSolver(None, ctx, precision=case["precision"])
        s.initialize()
        return {"case": case, "solver": s, "dt": float(ctx.num.dt)}
    if kind == "batch":
        ctxs = [_context(c, p) for c, p in _batch_inputs(case, seed)]
        b = LaneBatch(ctxs, case["precision"], lanes=case["lanes"]) if case["lanes"] > 1 \
            else BatchSolver(ctxs, case["precision"])
        owner = b.lanes[0] if case["lanes"] > 1 else b
        tables = [owner.laser_table(c, 0.0, case["steps"]) for c in ctxs]
        return {"case": case, "batch": b, "tables": tables}
    x = _field(case, seed)
    state = {"case": case, "x": x}
    if kind == "nodal":
        nz, ny, nx = x.shape
        small = SimulationContext.from_dict(workloads.straight_track(nx, ny, nz)[0])
        s = B200SpectralSolver(None, small)  # the state that the reconstruction takes its lengths from
        s.initialize()
        state["solver"] = s
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "solve":
        s, dt = state["solver"], state["dt"]
        s.reset()
        if case["by_step"]:
            metrics = [s.step(i * dt, dt)[1] for i in range(case["steps"])]
        else:
            metrics = s.run(0.0, case["steps"])
        if case["precision"] != "fp64":
            return {"modes": s.state.a.float()}  # FP32 values: what the mixed form keeps
        out = {"modes": s.state.a, "surface": s.surface_temperature(),
               "T_max": [m["T_surface_max"] for m in metrics], "iterations": [m["n_evap_iter"] for m in metrics]}
        if case["form"] == "box":
            out["box"] = s.state.fine_mesh.T_prev
        elif case["form"] != "track":
            out["field"] = s.state.T_prev
        return out
    if kind == "batch":
        b = state["batch"]
        for i, table in enumerate(state["tables"]):
            b.start(i, case["steps"], record=False, table=table)
        b.step(case["steps"])
        return {"modes": [b.modes(i) for i in range(b.n)]}
    if kind == "dct":
        c = kernels.DCT_II(state["x"])
        return {"forward": c, "back": kernels.IDCT_II(c)}
    return {"field": kernels.reconstruct_temperature_DCT(state["x"], state["solver"].state)}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

_ITERS = {"raster": 110, "tdep": 30, "box": 30}  # Picard iterations that a step of each form takes, about


def _dct_flops(shape):
    """A separable transform by dense contractions, each halved by the cosine's symmetry."""
    return float(np.prod([float(n) for n in shape])) * sum(shape)


def work(case):
    kind = case["kind"]
    if kind == "dct":
        shape = [case["n0"], case["n1"], case["n2"]][:case["dims"]]
        return {"bytes": 8.0 * 3 * float(np.prod(shape)), "flops": 2 * _dct_flops(shape)}
    if kind == "nodal":
        v = float(case["nx"] * case["ny"] * case["nz"])
        return {"bytes": 8.0 * 2 * v, "flops": _dct_flops((case["nx"], case["ny"], case["nz"]))}
    if kind == "solve":
        nx, ny, nz, steps = case["nx"], case["ny"], case["nz"], case["steps"]
        v, s = float(nx * ny * nz), float(nx * ny)
        if case["form"] == "track":
            return {"bytes": steps * (32 * v + 8 * s), "flops": steps * (8 * v + 4 * s * (nx + ny))}
        iters = _ITERS[case["form"]] if case["precision"] == "fp64" else 60
        per = 4 * v * (nx + ny + nz) if case["form"] != "box" else 16 * v * (nx + ny + nz)
        return {"bytes": steps * 40 * v, "flops": steps * iters * per}
    modes = faces = contraction = 0.0
    for cfg, _ in _batch_inputs(case, 0):
        nx, ny, nz = cfg["domain"]["mesh"]
        modes += nx * ny * nz
        faces += nx * ny
        contraction += float(nx * ny) * (nx + ny)
    iters = case["cap"]
    size = 4 if case["precision"] == "mixed" else 8
    return {"bytes": case["steps"] * (2 * size * modes + 16.0 * faces),
            "flops": case["steps"] * (8 * modes + (2 + 2 * iters) * contraction)}


# ---------------------------------------------------------------------------
# the same in plain torch FP64
# ---------------------------------------------------------------------------

_F = torch.float64


def _dct_matrix(n):
    k = torch.arange(n, device="cuda", dtype=torch.int64)
    m = (k[:, None] * (2 * k[None, :] + 1)) % (4 * n)
    w = torch.full((n, 1), math.sqrt(2.0 / n), device="cuda", dtype=_F)
    w[0, 0] = math.sqrt(1.0 / n)
    return w * torch.cos(m.to(_F) * (math.pi / (2 * n)))


def _along(x, mats):
    """Contract every axis of x with a matrix (out, in)."""
    for ax, m in enumerate(mats):
        x = torch.movedim(torch.tensordot(m, x, dims=([1], [ax])), 0, ax)
    return x


def _shift(f, sy, sx, nearest):
    """Order-1 translation of the last two axes, edge values or zero outside."""
    def taps(n, s):
        p = torch.arange(n, device="cuda", dtype=_F) - s
        fl = torch.floor(p)
        i = fl.to(torch.int64)
        return i.clamp(0, n - 1), (i + 1).clamp(0, n - 1), p - fl, (p >= 0) & (p <= n - 1)
    a, b, ty, iny = taps(f.shape[-2], sy)
    c, d, tx, inx = taps(f.shape[-1], sx)
    ty = ty[:, None]
    fa, fb = f[..., a, :], f[..., b, :]
    out = (1 - ty) * ((1 - tx) * fa[..., c] + tx * fa[..., d]) + ty * ((1 - tx) * fb[..., c] + tx * fb[..., d])
    return out if nearest else torch.where(iny[:, None] & inx[None, :], out, torch.zeros((), device="cuda", dtype=_F))


_K_FORM = {
    "raster": (lambda T: 15 + 20 * (T - 300) / 2700,) * 2,
    "tdep": (lambda T: 9.248 + 0.01571 * T, lambda T: 12.41 + 0.003279 * T),
}
_RHO_FORM = {
    "raster": (lambda T: 7900.0 + 0 * T,) * 2,
    "tdep": (lambda T: 8084.2 - 0.42086 * T - 3.8942e-5 * T ** 2, lambda T: 7432.7 + 0.039338 * T - 1.8007e-4 * T ** 2),
}
_C_FORM = {
    "raster": (lambda T: 450 + 350 * (T - 300) / 2700,) * 2,
    "tdep": (lambda T: 458.98 + 0.1328 * T, lambda T: 769.86 + 0 * T),
}


def _ref_const(v):
    return float(v["reference"]) if isinstance(v, dict) else float(v)


class _Exact:
    """One instance of the time step in plain torch FP64."""

    def __init__(self, cfg, form):
        self.form = form
        sim, mat = cfg["simulation"], cfg["material"]
        nx, ny, nz = cfg["domain"]["mesh"]
        L = [float(v) for v in cfg["domain"]["size"]]
        self.n, self.L, self.dt = (nx, ny, nz), L, float(sim["dt"])
        self.d = [l / n for l, n in zip(L, self.n)]
        self.mat = {k: _ref_const(v) for k, v in mat.items() if k != "name"}
        m = self.mat
        self.omega, self.tol = float(sim.get("picard_omega", 0.1)), float(sim.get("picard_tol", 1e-4))
        self.cap = int(sim.get("max_picard_iter", 30))
        self.correct = form in ("raster", "tdep")
        self.M = [_dct_matrix(n) for n in (nz, ny, nx)]
        self.MT = [q.t().contiguous() for q in self.M]
        kz, ky, kx = [(math.pi * torch.arange(n, device="cuda", dtype=_F) / l) ** 2 for n, l in zip((nz, ny, nx), L[::-1])]
        rc = m["rho"] * m["Cp"]
        lam = (m["k"] / rc) * (kz[:, None, None] + ky[None, :, None] + kx[None, None, :])
        self.K = torch.exp(-lam * self.dt)
        lam[0, 0, 0] = 1.0
        self.KK = -torch.expm1(-lam * self.dt) / lam / rc
        self.KK[0, 0, 0] = self.dt / rc
        c = torch.full((nz,), math.sqrt(2.0 / L[2]), device="cuda", dtype=_F)
        c[0] = math.sqrt(1.0 / L[2])
        self.Cb = c
        self.Ct = c * (1.0 - 2.0 * (torch.arange(nz, device="cuda") % 2).to(_F))
        self.a = torch.zeros((nz, ny, nx), device="cuda", dtype=_F)
        self.a[0, 0, 0] = m["T0"] * math.sqrt(L[0] * L[1] * L[2])
        self.q_evap = torch.zeros((ny, nx), device="cuda", dtype=_F)
        self.sdV = math.sqrt(self.d[0] * self.d[1] * self.d[2])
        self.recon = math.sqrt(nx * ny) / math.sqrt(L[0] * L[1])
        self.fscale = self.d[0] * self.d[1] * math.sqrt(nx * ny / (L[0] * L[1]))
        self.Tprev = torch.full((nz, ny, nx), m["T0"], device="cuda", dtype=_F)
        self.Qm = None
        self.laser = cfg["laser"]
        self.boxed = cfg.get("fine_mesh")
        if self.boxed:
            r = int(self.boxed["refinement"])
            self.bd = [q / r for q in self.d]
            bs = [float(v) for v in self.boxed["box_size"]]
            self.btot = [int(np.ceil(l / q)) for l, q in zip((L[0], L[1], bs[2]), self.bd)]
            self.bn = [min(int(np.ceil(b / q)), t) for b, q, t in zip(bs, self.bd, self.btot)]
            z0 = (0.0, 0.0, L[2] - bs[2])
            self.basis = []
            for n, l, t, q, o in zip(self.n, L, self.btot, self.bd, z0):
                co = torch.full((n, 1), math.sqrt(2.0 / l), device="cuda", dtype=_F)
                co[0, 0] = math.sqrt(1.0 / l)
                x = o + (torch.arange(t, device="cuda", dtype=_F) + 0.5) * q
                self.basis.append(co * torch.cos(math.pi * torch.arange(n, device="cuda", dtype=_F)[:, None] * x[None] / l))
            self.bT = self.bQ = None

    def _window(self, x, y):
        def start(p, q, tot, n):
            return max(0, min(round(max(0.0, min(p / q, tot - 1))) - n // 2, max(0, tot - n)))
        i = [start(x, self.bd[0], self.btot[0], self.bn[0]), start(y, self.bd[1], self.btot[1], self.bn[1]), 0]
        self.W = [b[:, k:k + n] for b, k, n in zip(self.basis, i, self.bn)][::-1]

    def _box(self, a):
        return _along(a, [w.t() for w in self.W])

    def _project_box(self, f):
        return _along(f, self.W) * (self.bd[0] * self.bd[1] * self.bd[2])

    def _face(self, q):
        return self.fscale * (self.M[1] @ q @ self.MT[2])

    def _surface(self, a, w):
        return self.recon * (self.MT[1] @ torch.tensordot(w, a, dims=([0], [0])) @ self.M[2])

    def _fl(self, T):
        ts, tl = self.mat["T_solidus"], self.mat["T_liquidus"]
        return ((T - ts) * (1.0 / (tl - ts))).clamp(0.0, 1.0)

    def _blend(self, props, T):
        fl = self._fl(T)
        return (1 - fl) * props[0](T) + fl * props[1](T)

    def _latent(self, T, Tp):
        rho = self._blend(_RHO_FORM[self.form], T) if self.correct else self.mat["rho"]
        return -rho * self.mat["L_f"] / self.dt * (self._fl(T) - self._fl(Tp))

    def _correction(self, a):
        T = _along(a, self.MT) / self.sdV
        kp = self._blend(_K_FORM[self.form], T) - self.mat["k"]
        ap = self._blend(_RHO_FORM[self.form], T) * self._blend(_C_FORM[self.form], T) - self.mat["rho"] * self.mat["Cp"]
        f = -ap * (T - self.Tprev) / self.dt
        for ax, h in zip((2, 1, 0), self.d):
            g = kp * torch.gradient(T, spacing=h, dim=ax)[0]
            f = f + torch.gradient(g, spacing=h, dim=ax)[0]
        return _along(f, self.M) * self.sdV

    def _evaporation(self, T):
        m = self.mat
        f1 = 0.82 * m["DeltaH_LV"] * m["Pa"] / math.sqrt(2 * math.pi * m["R_v"])
        f2 = m["DeltaH_LV"] / (m["R_v"] * m["T_boil"])
        hot = T >= m["T_liquidus"]
        Ts = torch.where(hot, T, torch.full_like(T, m["T_liquidus"]))
        return torch.where(hot, f1 / torch.sqrt(Ts) * torch.exp(f2 * (1.0 - m["T_boil"] / Ts)), torch.zeros_like(T))

    def step(self, st):
        m, (nx, ny, nz), d = self.mat, self.n, self.d
        rad = float(self.laser["radius"])
        I0 = float(self.laser["absorptivity"]) * st.power / (0.5 * math.pi * rad * rad) if st.is_on else 0.0
        x = (torch.arange(nx, device="cuda", dtype=_F) + 0.5) * d[0]
        y = (torch.arange(ny, device="cuda", dtype=_F) + 0.5) * d[1]
        q_las = I0 * torch.exp(-2.0 * (((x - st.x) / rad)[None, :] ** 2 + ((y - st.y) / rad)[:, None] ** 2))
        vx, vy = st.v
        aK, KK = self.a * self.K, self.KK
        kt, kb = KK * self.Ct[:, None, None], KK * self.Cb[:, None, None]
        a = aK + kt * self._face(q_las - _shift(self.q_evap, vy * self.dt / d[1], vx * self.dt / d[0], False))
        if self.boxed:
            self._window(st.x, st.y)
            if self.bT is None:
                self.bT = self._box(aK)
                self.bQ = torch.zeros_like(self.bT)
            sy, sx = -(vy * self.dt) / self.bd[1], -(vx * self.dt) / self.bd[0]
            self.bT, self.bQ = _shift(self.bT, sy, sx, True), _shift(self.bQ, sy, sx, False)
            a = a + KK * self._project_box(self.bQ)
        elif self.Qm is not None:
            a = a + KK * self.Qm
        ht, hb = m.get("h_conv_top", 0.0), m.get("h_conv_bottom", 0.0)
        if ht > 0:
            a = a + kt * self._face(-ht * (self._surface(a, self.Ct) - m["T0"]))
        S_bot = None
        if hb > 0:
            a = a + kb * self._face(-hb * (self._surface(a, self.Cb) - m["T0"]))
            Tb = self._surface(a, self.Cb)
            qb = -hb * (Tb - m["T0"])
            S_bot = self._face(qb * (m["k"] / self._blend(_K_FORM[self.form], Tb)) if self.correct else qb)
        it = 0
        for it in range(1, self.cap + 1):
            Ts = self._surface(a, self.Ct)
            qe = self._evaporation(Ts)
            q = q_las - qe - ht * (Ts - m["T0"])
            if self.correct:
                q = q * (m["k"] / self._blend(_K_FORM[self.form], Ts))
            new = aK + kt * self._face(q)
            Q = None
            if self.boxed:
                Q = self._latent(self._box(a), self.bT)
                new = new + KK * self._project_box(Q)
            elif m["L_f"] > 0:
                self.Qm = _along(self._latent(_along(a, self.MT) / self.sdV, self.Tprev), self.M) * self.sdV
                new = new + KK * self.Qm
            if S_bot is not None:
                new = new + kb * S_bot
            if self.correct:
                new = new + KK * self._correction(new)
            res = new - a
            rel = float(res.norm() / math.sqrt(a.numel())) / max(float(a.norm()) / math.sqrt(a.numel()), 1e-9)
            a = a + self.omega * res
            self.q_evap = qe
            if rel < self.tol:
                break
        self.a = a
        if self.boxed:
            self.bT = self._box(a)
            self.bQ = Q
        elif m["L_f"] > 0 or self.correct:
            self.Tprev = _along(a, self.MT) / self.sdV
        Ts = self._surface(a, self.Ct)
        return float(Ts.max()), it

    def solve(self, path, steps):
        return [self.step(path.get_state(i * self.dt, self.dt)) for i in range(steps)]


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        cfg, path = _solve_inputs(case, seed)
        e = _Exact(cfg, case["form"])
        got = e.solve(path, case["steps"])
        if case["precision"] != "fp64":
            return {"modes": e.a}
        out = {"modes": e.a, "surface": e._surface(e.a, e.Ct), "T_max": [g[0] for g in got],
               "iterations": [g[1] for g in got]}
        if case["form"] == "box":
            out["box"] = e.bT
        elif case["form"] != "track":
            out["field"] = e.Tprev
        return out
    if kind == "batch":
        modes = []
        for cfg, path in _batch_inputs(case, seed):
            e = _Exact(cfg, "track")
            e.solve(path, case["steps"])
            modes.append(e.a)
        return {"modes": modes}
    x = _field(case, seed)
    if kind == "dct":
        return {"forward": _along(x, [_dct_matrix(n) for n in x.shape]), "back": x}
    nodes = []
    for n, l in zip(x.shape, (0.5e-3, 1e-3, 2e-3)):
        j, m = torch.arange(n + 1, device="cuda", dtype=torch.int64), torch.arange(n, device="cuda", dtype=torch.int64)
        w = torch.full((n,), math.sqrt(2.0 / l), device="cuda", dtype=_F)
        w[0] = math.sqrt(1.0 / l)
        nodes.append(w * torch.cos(((j[:, None] * m[None, :]) % (2 * n)).to(_F) * (math.pi / n)))
    return {"field": _along(x, nodes).permute(2, 1, 0).contiguous()}
