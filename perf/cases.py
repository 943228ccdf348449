"""What a user of this package has it do, as cases whose time is measured.

A case is a dict of plain values; ``prepare`` makes its inputs on the GPU from
a seed, ``run`` takes them once through the package's public entry points, and
``exact`` is the same result in float64, written here in plain torch.  The
sizes are those of the benchmark's configurations, the drivers and the tests.

Kinds of case
  step     one ``PFSolver.stepper`` call, as the reference's Python driver
           loops make it: the temperature is an array, the moving gradient of
           the solidification driver, the moving point source of the scan
           drivers, or the interpolation of the coupled driver
  laser    ``HeatPFRun``: a saved state is loaded and advanced 20 coupled
           steps (the drivers' check interval) under a moving laser
  heat     one ``gamma.update_T`` call on the reference's ghosted field
  record   ``PFSolver.diagnostics`` or ``PFSolver.inspect`` of a state
  serve    ``BatchServer``: a batch of solidification jobs, submitted to done
  adjoint  ``HeatPFObjective``: objective and gradients of a laser run
  cfd      one ``AM_3d.time_integration`` of the implicit CFD solver
  grains   ``segment_grains`` of an orientation map

The states are mid-run ones: every grain is 1 inside, falls smoothly to an
exact 0 over a few cells at its boundary, and temperatures have a melt pool.
"""
import math

import numpy as np
import torch

from jax_am_gb300.adjoint import HeatPFObjective, LaserTrackProblem
from jax_am_gb300.cfd import cfd_am
from jax_am_gb300.cfd.gamma import update_T
from jax_am_gb300.phase_field.allen_cahn import PFSolver, Quench
from jax_am_gb300.phase_field.coupling import InterpolatedT
from jax_am_gb300.phase_field.grains import segment_grains
from jax_am_gb300.phase_field.point_source import PointSource
from jax_am_gb300.runner import HeatPFRun, raster
from jax_am_gb300.serving import BatchServer, Job

H = 1e-6  # cell size [m]
PF = dict(gas_const=8.3, Qg=1.4e5, L0=3.5e3, kappa_g=2.77e-6, m_g=2.4e5, ad_hoc=1.0)
GAMMA = dict(eta=0.4, r=5e-5, rho=8440.0, h=10.0, eps=0.4, SB=5.67e-8, T0=300.0, Ts=1563.0,
             Tl=1623.0, L=290e3 / 60.0)
T_MELT = 1700.0        # solidification jobs
T_LIQUIDUS = 1623.0    # laser runs
DT_PF = float(np.float32(6e-8))    # within the phase field's stability limit
DT_LASER = float(np.float32(3e-8))  # within the heat step's
POWER, SPEED = 200.0, 0.8


def listed():
    return [
        # the solidification driver's step at the size of its example: the
        # smallest call, repeated thousands of times from Python
        dict(name="step_gradient_128k", kind="step", source="gradient", nx=64, ny=64, nz=32,
             oris=20, grains=40, aniso=0.0, periodic=True, force=True),
        # a driver that computes its own temperature array; odd extents and an
        # orientation count that is no whole number of vectors
        dict(name="step_array_ragged", kind="step", source="array", nx=97, ny=61, nz=37, oris=13,
             grains=100, aniso=0.0, periodic=False, force=False),
        # the multi-scan driver: moving point source, anisotropic grain boundaries
        dict(name="step_point_1m", kind="step", source="point", nx=160, ny=120, nz=60, oris=20,
             grains=300, aniso=0.15, periodic=False, force=False),
        # the single-track laser run on a quick-look grid
        dict(name="laser_125k", kind="laser", nx=100, ny=50, nz=25, oris=20, grains=40,
             aniso=0.15, steps=20),
        # the single-track laser run of the benchmark
        dict(name="laser_8m", kind="laser", nx=400, ny=200, nz=100, oris=20, grains=2000,
             aniso=0.15, steps=20),
        # the multi-track run's 30 orientations, on its reduced raster
        dict(name="laser_4m_30", kind="laser", nx=320, ny=160, nz=80, oris=30, grains=1000,
             aniso=0.15, steps=20),
        # the standalone heat driver on the largest grid
        dict(name="heat_64m", kind="heat", nx=800, ny=400, nz=200),
        # energy, mass and orientation changes of the benchmark's state
        dict(name="diagnostics_8m", kind="record", record="diagnostics", nx=400, ny=200, nz=100,
             oris=20, grains=2000),
        # a burst of solidification jobs of the serving stream's mix
        dict(name="serve_16_jobs", kind="serve", jobs=16, mix=4, steps=48),
        # gradients of the differentiable run (a part of its 500 steps)
        dict(name="adjoint_1m", kind="adjoint", nx=128, ny=128, nz=64, oris=10, grains=300,
             aniso=0.0, steps=24, every=8),
        # the standalone CFD driver's case
        dict(name="cfd_2m", kind="cfd", nx=464, ny=93, nz=46),
        # grain statistics of the benchmark's final state
        dict(name="grains_8m", kind="grains", nx=400, ny=200, nz=100, oris=20, grains=2000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, lo, hi):
    """A flat box of lo .. hi cells: nx >= ny >= nz, any parity."""
    cells = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    ay, az = rng.uniform(0.4, 1.0), rng.uniform(0.2, 0.6)
    nx = max(8, int((cells / (ay * az)) ** (1.0 / 3.0)))
    return dict(nx=nx, ny=max(6, int(nx * ay)), nz=max(5, int(nx * az)))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "laser", "laser", "heat", "record", "serve",
                       "adjoint", "cfd", "grains"])
    c = dict(kind=kind)
    if kind == "step":
        c.update(_grid(rng, 3e4, 1.5e6), source=rng.choice(["gradient", "array", "point",
                                                            "interpolated"]))
        c["oris"] = 20 if rng.random() < 0.4 else rng.randint(10, 30)
        c["aniso"] = rng.choice([0.0, 0.15])
        c["periodic"] = c["source"] == "gradient" and rng.random() < 0.5
        c["force"] = c["source"] == "gradient"
    elif kind == "laser":
        c.update(_grid(rng, 6e4, 4e6), oris=rng.choice([20, 20, 30, 12, 10]), aniso=0.15, steps=20)
    elif kind == "heat":
        c.update(_grid(rng, 1e5, 6e7))
    elif kind == "record":
        c.update(_grid(rng, 6e4, 8e6), record=rng.choice(["diagnostics", "diagnostics", "inspect"]),
                 oris=rng.choice([20, 20, 10, 13, 30]))
    elif kind == "serve":
        c.update(jobs=rng.randint(4, 16), mix=rng.randint(5, 1 << 20), steps=rng.choice([32, 48]))
    elif kind == "adjoint":
        c.update(_grid(rng, 6e4, 1e6), oris=rng.choice([10, 10, 20, 7]),
                 aniso=rng.choice([0.0, 0.0, 0.15]), steps=rng.choice([10, 16, 24]), every=8)
    elif kind == "cfd":
        c.update(nx=_log_int(rng, 60, 440), ny=_log_int(rng, 24, 90), nz=_log_int(rng, 16, 44))
    else:
        c.update(_grid(rng, 6e4, 8e6), oris=rng.choice([20, 20, 10, 30]))
    if "oris" in c:
        c["grains"] = max(2, c["nx"] * c["ny"] * c["nz"] // 4000)
    return c


# ---- inputs --------------------------------------------------------------------

def _cells(c):
    return c["nx"] * c["ny"] * c["nz"]


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


class _Crystal:
    """What a solver takes from a polycrystal: cell size and cube axes."""

    def __init__(self, oris, seed, h=H):
        rng = np.random.default_rng(seed)
        q = rng.normal(size=(oris, 4))
        w, x, y, z = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
        R = np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)],
                      [2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)],
                      [2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)]])
        self.mesh_h_xyz = (h, h, h)
        self.unique_grain_directions = np.ascontiguousarray(R.transpose(1, 2, 0))


def _voronoi(nx, ny, nz, oris, grains, seed, width=None):
    """Cells of nearest-seed grains, z-major.  Without ``width``: the (N,)
    orientation indices.  With it: the (N, oris) order parameters, each grain
    falling from 1 to an exact 0 over ``width`` cells across its boundary."""
    g = _generator(seed)
    pts = torch.rand(grains, 3, generator=g, device="cuda") * torch.tensor(
        [nx, ny, nz], dtype=torch.float32, device="cuda")
    ori = torch.randint(oris, (grains,), generator=g, device="cuda").sort()[0]
    ends = torch.bincount(ori, minlength=oris).cumsum(0).tolist()
    N = nx * ny * nz
    if width:
        out = torch.zeros(N, oris, device="cuda")
    else:
        out = torch.empty(N, dtype=torch.int32, device="cuda")
    chunk = max(1024, (1 << 28) // grains)
    for i0 in range(0, N, chunk):
        i = torch.arange(i0, min(N, i0 + chunk), device="cuda")
        x, y, z = i % nx, i // nx % ny, i // (nx * ny)
        d = torch.cdist(torch.stack((x, y, z), 1).float() + 0.5, pts)
        if not width:
            out[i0:i0 + chunk] = ori[d.argmin(1)].int()
            continue
        near = torch.full((len(i), oris), 1e30, device="cuda")
        for o in range(oris):
            b, e = (ends[o - 1] if o else 0), ends[o]
            if e > b:
                near[:, o] = d[:, b:e].amin(1)
        s = (1.0 - (near - near.amin(1, keepdim=True)) / width).clamp_(0.0, 1.0)
        s = s * s * (3.0 - 2.0 * s)
        out[i0:i0 + chunk] = s / s.square().sum(1, keepdim=True).sqrt()
    return out


def _pool(nx, ny, nz, seed, order="zyx"):
    """A ghosted float32 temperature with a melt pool under the beam, and the
    beam's position: x, y in metres."""
    rng = np.random.default_rng(seed)
    bx, by = nx * rng.uniform(0.25, 0.45), ny * rng.uniform(0.45, 0.55)
    peak, w = rng.uniform(3000.0, 7000.0), min(45.0, 0.3 * ny)
    x, y, z = (torch.arange(m + 2, device="cuda", dtype=torch.float32) - 0.5 for m in (nx, ny, nz))
    ex, ey = torch.exp(-((x - bx) / (1.5 * w)) ** 2), torch.exp(-((y - by) / w) ** 2)
    ez = torch.exp((z - nz) / (0.6 * w)).clamp_(max=1.0)
    if order == "zyx":
        T = 300.0 + peak * ez[:, None, None] * ey[None, :, None] * ex[None, None, :]
    else:
        T = 300.0 + peak * ex[:, None, None] * ey[None, :, None] * ez[None, None, :]
    return T, bx * H, by * H


def _pf_args(c, T_liquidus, **more):
    a = dict(PF, Nx=c["nx"], Ny=c["ny"], Nz=c["nz"], num_oris=c["oris"], T_liquidus=T_liquidus,
             anisotropy=c.get("aniso", 0.0))
    a.update(more)
    return a


def _step_inputs(c, seed):
    melt = T_MELT if c["source"] == "gradient" else T_LIQUIDUS
    more = dict(bc=("periodic", "periodic", "neumann")) if c["periodic"] else {}
    if c["force"]:
        more.update(force_liquid_zero=True, liquid_shift=1.0)
    s = dict(args=_pf_args(c, melt, **more), crystal=_Crystal(c["oris"], seed))
    s["eta"] = _voronoi(c["nx"], c["ny"], c["nz"], c["oris"], c["grains"], seed, width=8.0)
    rng = np.random.default_rng(seed)
    s["t"] = float(rng.uniform(0.0, 2e-5))
    if c["source"] == "gradient":
        s["gradient"] = (melt, float(rng.uniform(5e5, 2e6)), 0.1, 0.5 * c["nz"] * H)
    elif c["source"] == "point":
        s["point"] = dict(ts=[s["t"]], xs=c["nx"] * H * rng.uniform(0.3, 0.5),
                          ys=c["ny"] * H * 0.5, zs=c["nz"] * H, dirs=(1.0, 0.0, 0.0), Q=25.0,
                          vel=0.8, T_ambient=300.0, alpha=5.2e-6, kappa=27.0, T_clip=2000.0)
    else:
        T, _, _ = _pool(c["nx"], c["ny"], c["nz"], seed)
        s["T"] = T[1:-1, 1:-1, 1:-1].reshape(-1, 1).contiguous()
        if c["source"] == "interpolated":
            s["T"] = (s["T"], (300.0 + 0.95 * (s["T"] - 300.0)).contiguous())
    return s


def _track(c, bx, by):
    """One straight track from the pool on; three of them for the raster of
    the multi-track run (30 orientations)."""
    if c["oris"] != 30:
        return [(0.0, 1.0, bx, by, bx + SPEED, by, POWER)]
    ys = [by, by + 0.2 * c["ny"] * H, by + 0.4 * c["ny"] * H]
    return raster(ys, SPEED, 250.0, bx, c["nx"] * H * 0.9)


def _laser_inputs(c, seed):
    T, bx, by = _pool(c["nx"], c["ny"], c["nz"], seed)
    return dict(args=_pf_args(c, T_LIQUIDUS), crystal=_Crystal(c["oris"], seed), T=T,
                path=_track(c, bx, by),
                eta=_voronoi(c["nx"], c["ny"], c["nz"], c["oris"], c["grains"], seed, width=8.0))


def _serve_jobs(c):
    """Sizes, orientation counts and steps of the jobs (the stream's mix)."""
    rng = np.random.default_rng(c["mix"])
    jobs = []
    for _ in range(c["jobs"]):
        j = dict(nx=int(rng.integers(32, 161)), ny=int(rng.integers(32, 161)),
                 nz=int(rng.integers(16, 65)), oris=int(rng.integers(10, 31)))
        j.update(steps=int(rng.integers(c["steps"] // 3, c["steps"] + 1)),
                 grad=float(rng.uniform(5e5, 2e6)), grains=max(2, _cells(j) // 2000))
        jobs.append(j)
    return jobs


def _job_args(j):
    return _pf_args(j, T_MELT, force_liquid_zero=True, liquid_shift=1.0)


def _job_gradient(j):
    return (T_MELT, j["grad"], 0.1, 0.5 * j["nz"] * H)


def _job_eta(j, k, seed):
    return _voronoi(j["nx"], j["ny"], j["nz"], j["oris"], j["grains"], seed * 97 + k, width=8.0)


def _adjoint_inputs(c, seed):
    T, bx, by = _pool(c["nx"], c["ny"], c["nz"], seed)
    w = np.random.default_rng(seed).random(c["oris"]).astype(np.float32)
    return dict(args=_pf_args(c, T_LIQUIDUS), crystal=_Crystal(c["oris"], seed), T=T, bx=bx, by=by,
                w=w, eta=_voronoi(c["nx"], c["ny"], c["nz"], c["oris"], c["grains"], seed,
                                  width=8.0))


def _record_inputs(c, seed):
    """A state, the one it grew from (boundaries two cells away) and T."""
    eta = _voronoi(c["nx"], c["ny"], c["nz"], c["oris"], c["grains"], seed, width=8.0)
    eta0 = eta.view(c["nz"], c["ny"], c["nx"], c["oris"]).roll(2, 2).view_as(eta)
    T, _, _ = _pool(c["nx"], c["ny"], c["nz"], seed)
    return eta, eta0, T[1:-1, 1:-1, 1:-1].reshape(-1, 1).contiguous()


def _cfd_inputs(c, seed):
    """A pool with a vortex under the beam: T, vel and their convective terms."""
    rng = np.random.default_rng(seed)
    N, d = (c["nx"], c["ny"], c["nz"]), 1e-3 / 464
    NL = [max(3, round(f * n)) for f, n in zip((0.75, 0.5, 0.4), N)]
    X0 = [N[0] * d * rng.uniform(0.2, 0.5), N[1] * d * 0.5, N[2] * d]
    args = dict(rho=8440.0, visco=7e-3, Marangoni=-2e-5, dt=1e-6, t_OFF=0.0012, speed=0.5, X0=X0,
                rb=5e-5, eta=0.43, P=100.0, T_ref=300.0, Ts=1563.0, Tl=1623.0,
                latent_heat=270000.0, heat_source=0,
                cp=cfd_am.LinearClip(0.2441, 338.39, 300.0, 1563.0),
                k=cfd_am.LinearClip(0.0163105, 4.5847, 300.0, 1563.0))
    args["mesh"] = cfd_am.mesh3d([n * d for n in N], list(N))
    args["mesh_local"] = cfd_am.mesh3d([n * d for n in NL], NL)
    x, y, z = torch.meshgrid(*((torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) * d - b
                               for n, b in zip(N, X0)), indexing="ij")
    w = min(4.5e-5, 0.35 * N[1] * d)
    T = 300.0 + rng.uniform(2200.0, 2800.0) * torch.exp(-(x * x + y * y) / w ** 2 + 2.0 * z / w)
    # curl of (0, P, 0) with P = a x z exp(-r^2 / b^2): no divergence, no flow
    # through the top
    b2 = (0.5 * w) ** 2
    e = rng.uniform(0.2, 0.4) / w * torch.exp(-(x * x + y * y + z * z) / b2)
    vel = torch.stack((-x * e * (1.0 - 2.0 * z * z / b2), torch.zeros_like(x),
                       z * e * (1.0 - 2.0 * x * x / b2)), dim=3)

    def along(f):
        return sum(v * gr for v, gr in zip(vel.unbind(3), torch.gradient(f, spacing=d)))

    return args, dict(T=T[..., None], vel=vel, conv_T=along(T)[..., None],
                      conv=torch.stack([along(f) for f in vel.unbind(3)], dim=3),
                      grad_p0=torch.zeros_like(vel),
                      solidID=((T.clamp(1563.0, 1623.0) - 1563.0) / 60.0)[..., None])


def _grain_inputs(c, seed):
    T, _, _ = _pool(c["nx"], c["ny"], c["nz"], seed)
    return (_voronoi(c["nx"], c["ny"], c["nz"], c["oris"], c["grains"], seed),
            T[1:-1, 1:-1, 1:-1].reshape(-1).contiguous())


def _table(grains, rows):
    """The grains' statistics in columns of fixed length, as a program that
    collects them over many outputs keeps them; the rest of a column is 0."""
    out = {"labels": grains["labels"], "count": len(grains["cells"])}
    for name in ("ori", "first_cell", "cells", "volumes", "aspect_ratios"):
        out[name] = np.zeros(rows, grains[name].dtype)
        out[name][:len(grains[name])] = grains[name]
    return out


_COORDINATES = {}  # a program's cell centres, made once for its grid


def _coordinates(nx, ny, nz):
    if (nx, ny, nz) not in _COORDINATES:
        _COORDINATES.clear()
        _COORDINATES[nx, ny, nz] = torch.meshgrid(
            *((torch.arange(n, device="cuda", dtype=torch.float32) + 0.5) * H
              for n in (nx, ny, nz)), indexing="ij")[:2]
    return _COORDINATES[nx, ny, nz]


# ---- one pass --------------------------------------------------------------------

def prepare(case, seed):
    c = case
    kind = c["kind"]
    if kind == "step":
        s = _step_inputs(c, seed)
        solver = PFSolver(s["args"], s["crystal"])
        if c["source"] == "gradient":
            T = Quench(*s["gradient"])
        elif c["source"] == "point":
            T = PointSource(**s["point"])
        elif c["source"] == "interpolated":
            T = InterpolatedT(*s["T"], s["t"] + 1e-6, 2e-6)
        else:
            T = s["T"]
        return dict(kind=kind, solver=solver, eta=s["eta"], t=s["t"], T=T)
    if kind == "laser":
        s = _laser_inputs(c, seed)
        run_ = HeatPFRun(PFSolver(s["args"], s["crystal"]), GAMMA, s["path"], dt=DT_LASER,
                         eta0=s["eta"], T_init=s["T"])
        run_.prepare()
        return dict(kind=kind, run=run_, eta=s["eta"], T=s["T"], steps=c["steps"])
    if kind == "heat":
        T, bx, by = _pool(c["nx"], c["ny"], c["nz"], seed, order="xyz")
        return dict(kind=kind, T=T, xl=bx, yl=by, x=_coordinates(c["nx"], c["ny"], c["nz"]))
    if kind == "record":
        eta, eta0, T = _record_inputs(c, seed)
        solver = PFSolver(_pf_args(c, T_LIQUIDUS), _Crystal(c["oris"], seed))
        return dict(kind=kind, solver=solver, eta=eta, eta0=eta0, T=T, record=c["record"])
    if kind == "serve":
        jobs = []
        for k, j in enumerate(_serve_jobs(c)):
            jobs.append(Job(_job_args(j), _Crystal(j["oris"], seed * 97 + k),
                            Quench(*_job_gradient(j)), j["steps"], DT_PF,
                            eta0=_job_eta(j, k, seed)))
        return dict(kind=kind, server=BatchServer(), jobs=jobs)
    if kind == "adjoint":
        s = _adjoint_inputs(c, seed)
        problem = LaserTrackProblem(s["args"], s["crystal"], GAMMA, s["w"], DT_LASER, c["steps"],
                                    s["bx"], s["by"], checkpoint_every=c["every"], T_init=s["T"])
        P, v = (torch.tensor(x, dtype=torch.float64, requires_grad=True) for x in (POWER, SPEED))
        return dict(kind=kind, problem=problem, P=P, v=v, eta=s["eta"].requires_grad_())
    if kind == "cfd":
        args, fields = _cfd_inputs(c, seed)
        return dict(kind=kind, sim=cfd_am.AM_3d(args), fields=fields)
    ori, T = _grain_inputs(c, seed)
    args = dict(Nx=c["nx"], Ny=c["ny"], Nz=c["nz"], h=H, num_oris=c["oris"], T_liquidus=T_LIQUIDUS)
    return dict(kind=kind, args=args, ori=ori, T=T, rows=2 * c["grains"] + 64)


def run(state):
    s = state
    kind = s["kind"]
    if kind == "step":
        _, eta = s["solver"].stepper((s["eta"], s["t"]), s["t"] + DT_PF, [s["T"]])
        return eta
    if kind == "laser":
        r = s["run"].load(s["eta"], s["T"]).run(s["steps"])
        return {"eta": r.state, "T": r.T_ghosted}
    if kind == "heat":
        return update_T(s["T"], s["xl"], s["yl"], *s["x"], POWER, H, H, H, DT_LASER, GAMMA)
    if kind == "record":
        return getattr(s["solver"], s["record"])(s["eta"], s["T"], s["eta0"])
    if kind == "serve":
        server, jobs = s["server"], [j.fresh() for j in s["jobs"]]
        for j in jobs:
            server.submit(j)
        server.run(realtime=False)
        server.done.clear()
        return [j.result for j in jobs]
    if kind == "adjoint":
        J = HeatPFObjective.apply(s["P"], s["v"], s["eta"], s["problem"])
        dP, dv, deta = torch.autograd.grad(J, (s["P"], s["v"], s["eta"]))
        return {"J": J.detach(), "dP": dP, "dv": dv, "deta": deta}
    if kind == "cfd":
        sim, f = s["sim"], s["fields"]
        sim.T, sim.t = f["T"], 0.0
        for name in ("vel", "conv", "conv_T", "grad_p0", "solidID"):
            getattr(sim, name).copy_(f[name])
        sim.time_integration()
        return {name: getattr(sim, name) for name in f}
    return _table(segment_grains(s["args"], s["ori"], s["T"]), s["rows"])


def work(case):
    """Bytes: every step's state read once and written once.  Operations: of
    the update formulas per order parameter (12, or 33 with anisotropy) and
    per cell's temperature (40)."""
    c = case
    kind = c["kind"]
    if kind == "serve":
        v = sum(_cells(j) * j["oris"] * j["steps"] for j in _serve_jobs(c))
        return {"bytes": 8 * v, "flops": 12 * v}
    N = _cells(c)
    if kind == "heat":
        return {"bytes": 8 * N, "flops": 40 * N}
    if kind == "cfd":
        box = round(0.75 * c["nx"]) * round(0.5 * c["ny"]) * round(0.4 * c["nz"])
        return {"bytes": 8 * (6 * N + 18 * box), "flops": 400 * N + 1000 * box}
    if kind == "grains":
        return {"bytes": 12 * N, "flops": 10 * N}
    per = 33 if c.get("aniso") else 12
    if kind == "step":
        T = {"array": 4, "interpolated": 8}.get(c["source"], 0)
        return {"bytes": N * (8 * c["oris"] + T), "flops": per * N * c["oris"]}
    if kind == "laser":
        return {"bytes": c["steps"] * N * (8 * c["oris"] + 8),
                "flops": c["steps"] * N * (per * c["oris"] + 40)}
    if kind == "record":
        return {"bytes": N * (4 * c["oris"] + 8), "flops": 14 * N * c["oris"]}
    # adjoint: the forward run, then per step the state and the multipliers
    return {"bytes": c["steps"] * N * (20 * c["oris"] + 24),
            "flops": c["steps"] * N * (4 * per * c["oris"] + 200)}


# ---- the same results in float64 -------------------------------------------------

def _f(x):
    """A parameter as the package holds it: float32."""
    return float(np.float32(x))


def _shift(e, axis, step, periodic):
    if periodic:
        return torch.roll(e, -step, axis)
    n = e.shape[axis]
    i = (torch.arange(n, device=e.device) + step).clamp_(0, n - 1)
    return e.index_select(axis, i)


def _pf_rhs(e, T, a, dirs, periodic):
    """d eta / dt on (nz, ny, nx, n) planes at temperature T (nz, ny, nx)."""
    h2 = _f(H) ** 2
    Tc = T.clamp(max=2000.0)[..., None]
    zeta = 0.5 * (1.0 - torch.tanh(1e10 * (Tc / _f(a["T_liquidus"]) - 1.0)))
    Lg = _f(a["L0"]) * torch.exp(-_f(a["Qg"]) / (_f(a["gas_const"]) * Tc))
    sides = [(_shift(e, ax, -1, p), _shift(e, ax, 1, p))
             for ax, p in ((2, periodic[0]), (1, periodic[1]), (0, periodic[2]))]
    lap = sum(m + p for m, p in sides).sub_(6.0 * e).div_(h2)
    if a["anisotropy"] > 0.0:
        g = [p - m for m, p in sides]
        del sides
        ee = g[0] ** 2 + g[1] ** 2 + g[2] ** 2
        top = None
        for d in dirs:  # the orientation's three cube axes, each (n, 3)
            q = (g[0] * d[:, 0] + g[1] * d[:, 1] + g[2] * d[:, 2]) ** 2
            top = q if top is None else torch.maximum(top, q)
        c2 = torch.where(ee > 0.0, top / torch.where(ee > 0.0, ee, 1.0), 1.0).clamp(max=1.0)
        lap = lap * (1.0 + _f(a["anisotropy"]) * (c2 ** 2 + (1.0 - c2) ** 2))
    S = (e * e).sum(-1, keepdim=True)
    bulk = _f(a["m_g"]) * e * (4.0 * S - 3.0 * e * e - 1.0 + 2.0 * (1.0 - zeta) ** 2)
    return Lg * (_f(a["kappa_g"]) * lap - bulk)


def _pf_step(e, T, dt, a, crystal):
    """One Euler step of (nz, ny, nx, n), a few planes at a time."""
    bc = a.get("bc", "neumann")
    px, py, pz = ((b == "periodic") for b in ((bc,) * 3 if isinstance(bc, str) else bc))
    dirs = torch.as_tensor(crystal.unique_grain_directions, device="cuda").float().double()
    nz = e.shape[0]
    per = max(1, int(2e7) // (e.shape[1] * e.shape[2] * e.shape[3]))
    out = torch.empty_like(e)
    for z0 in range(0, nz, per):
        z1 = min(nz, z0 + per)
        if pz:
            i = torch.arange(z0 - 1, z1 + 1, device="cuda") % nz
        else:
            i = torch.arange(z0 - 1, z1 + 1, device="cuda").clamp_(0, nz - 1)
        b = e.index_select(0, i)
        out[z0:z1] = e[z0:z1] + dt * _pf_rhs(b, T.index_select(0, i), a, dirs,
                                             (px, py, False))[1:-1]
    if a.get("force_liquid_zero"):
        out[T > _f(a["T_liquidus"]) + _f(a["liquid_shift"])] = 0.0
    return out


def _heat_step(Tg, xl, yl, P, dt, g=GAMMA):
    """One explicit heat step of the ghosted (nz+2, ny+2, nx+2) field."""
    d = _f(H)
    I = slice(1, -1)
    T = Tg[I, I, I]
    clip = T.clamp(300.0, _f(g["Tl"]))
    k = 0.0163 * clip + 4.5847
    cp = 0.2441 * clip + 338.39 + ((T > _f(g["Ts"])) & (T < _f(g["Tl"]))).to(T.dtype) * _f(g["L"])
    sb, T0 = _f(g["SB"]) * _f(g["eps"]), _f(g["T0"])
    x = (torch.arange(T.shape[2], dtype=T.dtype, device=T.device)) * d + _f(H / 2)
    y = (torch.arange(T.shape[1], dtype=T.dtype, device=T.device)) * d + _f(H / 2)
    r = _f(g["r"])
    beam = (2.0 * P * _f(g["eta"]) / math.pi / r ** 2
            * torch.exp(-2.0 * ((x[None, :] - xl) ** 2 + (y[:, None] - yl) ** 2) / r ** 2))
    B = Tg.clone()
    for ax in range(3):
        for end in (0, -1):
            cell = T.select(ax, end)
            face = (cell + _ghost(Tg, ax, end)) / 2.0
            q = _f(g["h"]) * (face - T0) + sb * (face ** 4 - T0 ** 4)
            if ax == 0 and end == -1:
                q = q - beam
            _ghost(B, ax, end).copy_(cell - q * d / k.select(ax, end))
    lap = 0.0
    for ax in range(3):
        n = T.shape[ax]
        view = [I, I, I]
        view[ax] = slice(0, n)
        lo = B[tuple(view)]
        view[ax] = slice(2, n + 2)
        lap = lap + (lo + B[tuple(view)] - 2.0 * T) / d ** 2
    out = B.clone()
    out[I, I, I] = T + dt * k / (_f(g["rho"]) * cp) * lap
    return out


def _ghost(Tg, ax, end):
    """The ghost face (without its edges) at one end of an axis."""
    view = [slice(1, -1)] * 3
    view[ax] = end
    return Tg[tuple(view)]


def _beam(path, t):
    for t0, t1, x0, y0, x1, y1, P in path:
        t0, t1, x0, y0, x1, y1 = (_f(v) for v in (t0, t1, x0, y0, x1, y1))
        if t0 <= t < t1:
            f = (t - t0) / (t1 - t0)
            return x0 + f * (x1 - x0), y0 + f * (y1 - y0), _f(P)
    return 0.0, 0.0, 0.0


def _planes(c, gradient, t):
    """The moving gradient's temperature, (nz, ny, nx), as the float32 array
    that the reference's driver makes of it (it can meet T_liquidus exactly)."""
    base, grad, vel, z0 = gradient
    z = 0.5 * _f(H) + _f(H) * torch.arange(c["nz"], dtype=torch.float64, device="cuda")
    T = (base + grad * (z - z0) - grad * vel * t).float().double()
    return T[:, None, None].expand(c["nz"], c["ny"], c["nx"])


def _point_T(c, p):
    x, y, z = (_f(H) * torch.arange(n, dtype=torch.float64, device="cuda") + _f(0.5 * _f(H))
               for n in (c["nx"], c["ny"], c["nz"]))
    X = (x - _f(p["xs"]))[None, None, :]
    Y = (y - _f(p["ys"]))[None, :, None]
    Z = (z - _f(p["zs"]))[:, None, None]
    R = torch.sqrt(X * X + Y * Y + Z * Z)
    ux, uy, uz = (_f(u) for u in p["dirs"])
    T = _f(p["T_ambient"]) + _f(p["Q"]) / (2.0 * math.pi * _f(p["kappa"])) / R * torch.exp(
        -_f(p["vel"]) / (2.0 * _f(p["alpha"])) * (R + X * ux + Y * uy + Z * uz))
    return T.clamp(max=_f(p["T_clip"]))


def _exact_step(c, seed):
    s = _step_inputs(c, seed)
    e = s["eta"].double().view(c["nz"], c["ny"], c["nx"], c["oris"])
    if c["source"] == "gradient":
        T = _planes(c, s["gradient"], s["t"])
    elif c["source"] == "point":
        T = _point_T(c, s["point"])
    elif c["source"] == "interpolated":
        r = (s["t"] + 1e-6 - (s["t"] + DT_PF)) / 2e-6
        T = (r * s["T"][0].double() + (1.0 - r) * s["T"][1].double()).view(e.shape[:3])
    else:
        T = s["T"].double().view(e.shape[:3])
    dt = _f((s["t"] + DT_PF) - s["t"])
    return _pf_step(e, T, dt, s["args"], s["crystal"]).view(-1, c["oris"])


def _exact_laser(c, seed):
    s = _laser_inputs(c, seed)
    e = s["eta"].double().view(c["nz"], c["ny"], c["nx"], c["oris"])
    Tg, t = s["T"].double(), 0.0
    for _ in range(c["steps"]):
        e = _pf_step(e, Tg[1:-1, 1:-1, 1:-1], DT_LASER, s["args"], s["crystal"])
        Tg = _heat_step(Tg, *_beam(s["path"], t + 0.5 * DT_LASER), DT_LASER)
        t += DT_LASER
    return {"eta": e.view(-1, c["oris"]), "T": Tg}


def _exact_heat(c, seed):
    T, bx, by = _pool(c["nx"], c["ny"], c["nz"], seed, order="xyz")
    out = _heat_step(T.double().permute(2, 1, 0), _f(bx), _f(by), POWER, DT_LASER)
    return out.permute(2, 1, 0).contiguous()


def _exact_record(c, seed):
    eta, eta0, T = _record_inputs(c, seed)
    n, shape = c["oris"], (c["nz"], c["ny"], c["nx"], c["oris"])
    T, tl = T.double().view(-1), _f(T_LIQUIDUS)
    N = len(T)
    first = torch.arange(n, 0, -1, device="cuda")  # of equal maxima the first

    def argmax(e):
        return ((e == e.amax(1, keepdim=True)) * first).amax(1)

    changed = int((argmax(eta) != argmax(eta0)).sum())
    liquid = int((T >= tl).sum())
    energy, mass = 0.0, np.zeros(n)
    if c["record"] == "diagnostics":
        zeta = 0.5 * (1.0 - torch.tanh(1e10 * (T.clamp(max=2000.0) / tl - 1.0))).view(shape[:3])
        e4, total, h = eta.view(shape), 0.0, _f(H)
        for z in range(c["nz"]):
            e, up = e4[z].double(), e4[min(z + 1, c["nz"] - 1)].double()
            e2 = e * e
            S, Q = e2.sum(-1), (e2 * e2).sum(-1)
            bulk = Q / 4.0 - S / 2.0 + S * S - Q + (1.0 - zeta[z]) ** 2 * S
            grad = ((_shift(e, 1, 1, False) - e) ** 2 + (_shift(e, 0, 1, False) - e) ** 2
                    + (up - e) ** 2).sum(-1)
            total = total + (_f(PF["m_g"]) * bulk + 0.5 * _f(PF["kappa_g"]) * grad / h ** 2).sum()
        energy = float(total) * h ** 3
        mass = eta.sum(0, dtype=torch.float64).cpu().numpy()
    return {"energy": energy, "max_T": float(T.max()), "n_cells": N, "n_ori_changed": changed,
            "n_liquid": liquid, "n_nonfinite": 0, "mass": mass,
            "pct_ori_changed": changed / N * 100.0, "pct_liquid": liquid / N * 100.0}


def _exact_serve(c, seed):
    out = []
    for k, j in enumerate(_serve_jobs(c)):
        e = _job_eta(j, k, seed).double().view(j["nz"], j["ny"], j["nx"], j["oris"])
        args, crystal = _job_args(j), _Crystal(j["oris"], seed * 97 + k)
        for step in range(j["steps"]):
            e = _pf_step(e, _planes(j, _job_gradient(j), step * DT_PF), DT_PF, args, crystal)
        out.append(e.view(-1, j["oris"]))
    return out


def _exact_adjoint(c, seed):
    from torch.utils.checkpoint import checkpoint
    s = _adjoint_inputs(c, seed)
    dirs = torch.as_tensor(s["crystal"].unique_grain_directions, device="cuda").float().double()
    P, v = (torch.tensor(x, dtype=torch.float64, device="cuda", requires_grad=True)
            for x in (POWER, SPEED))
    eta = s["eta"].double().requires_grad_()
    x_start, y = _f(s["bx"]), _f(s["by"])

    def step(e, Tg, P, v, t):
        T = Tg[1:-1, 1:-1, 1:-1]
        new = e + DT_LASER * _pf_rhs(e, T, s["args"], dirs, (False,) * 3)
        return new, _heat_step(Tg, x_start + v * (t + 0.5 * DT_LASER), y, P, DT_LASER)

    e, Tg, t = eta.view(c["nz"], c["ny"], c["nx"], c["oris"]), s["T"].double(), 0.0
    for _ in range(c["steps"]):
        e, Tg = checkpoint(step, e, Tg, P, v, t, use_reentrant=False)
        t += DT_LASER
    J = (e * e * torch.as_tensor(s["w"], device="cuda").double()).sum() / _cells(c)
    dP, dv, deta = torch.autograd.grad(J, (P, v, eta))
    return {"J": J.detach(), "dP": dP, "dv": dv, "deta": deta}


def _exact_grains(c, seed):
    """Components by propagating the smallest cell index, with pointer jumps."""
    ori, T = _grain_inputs(c, seed)
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    N = nx * ny * nz
    key = torch.where(T < _f(T_LIQUIDUS), ori.long(), -1).view(nz, ny, nx)
    lab = torch.arange(N, device="cuda")
    joins = []
    for ax in range(3):
        n = key.shape[ax]
        a, b = key.narrow(ax, 0, n - 1), key.narrow(ax, 1, n - 1)
        same = (a == b) & (a >= 0)
        i = lab.view_as(key).narrow(ax, 0, n - 1)[same]
        joins.append((i, i + (nx * ny, nx, 1)[ax]))
    while True:
        old = lab.clone()
        for i, j in joins:
            low = torch.minimum(lab[i], lab[j])
            root = torch.maximum(lab[i], lab[j])
            lab = lab.scatter_reduce(0, root, low, "amin")
        while True:
            up = lab[lab]
            if torch.equal(up, lab):
                break
            lab = up
        if torch.equal(old, lab):
            break
    key = key.view(-1)
    solid = key >= 0
    roots = torch.unique(lab[solid])
    roots = roots[torch.argsort(key[roots] * N + roots)]
    rank = torch.full((N,), -1, dtype=torch.int64, device="cuda")
    rank[roots] = torch.arange(len(roots), device="cuda")
    labels = torch.where(solid, rank[lab], -1)
    i = torch.nonzero(solid).view(-1)
    xyz = torch.stack((i % nx, i // nx % ny, i // (nx * ny))).double()
    g, K = labels[i], len(roots)
    cells = torch.bincount(g, minlength=K)
    mean = torch.stack([torch.zeros(K, dtype=torch.float64, device="cuda").index_add_(0, g, p)
                        for p in xyz]) / cells
    off = xyz - mean[:, g]
    cov = torch.zeros(K, 9, dtype=torch.float64, device="cuda").index_add_(
        0, g, (off[:, None] * off[None]).reshape(9, -1).t())
    cov = cov.view(K, 3, 3) / (cells - 1).clamp(min=1)[:, None, None]
    ln = np.sqrt(np.maximum(np.linalg.eigvalsh(cov.cpu().numpy())[:, ::-1], 0.0))
    cells = cells.cpu().numpy()
    with np.errstate(divide="ignore", invalid="ignore"):
        ratio = np.where(cells >= 5, 2.0 * ln[:, 0] / (ln[:, 1] + ln[:, 2]), 1.0)
    return _table({"labels": labels.int(), "ori": key[roots].cpu().numpy(),
                   "first_cell": roots.cpu().numpy(), "cells": cells, "volumes": cells * H ** 3,
                   "aspect_ratios": ratio}, 2 * c["grains"] + 64)


def exact(case, seed):
    if case["kind"] == "cfd":
        return None  # iterative solves: their result depends on where they stop
    return {"step": _exact_step, "laser": _exact_laser, "heat": _exact_heat,
            "record": _exact_record, "serve": _exact_serve, "adjoint": _exact_adjoint,
            "grains": _exact_grains}[case["kind"]](dict(case), seed)
