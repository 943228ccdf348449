"""The cell-per-lane step (``pf_lane.cu``) at every orientation count that has an
instance, above the cell count from which counts other than 20 take it: all five
temperature sources, with and without anisotropy, ragged tiles (nx mod 16 = 2,
13 and 14), Neumann and periodic axes, chunks of the planner's and one chunk
whose planes go round the ring of slots several times.

Against the TMA-fed kernel (variant 3) it is the same arithmetic in the same
order, so equal bit for bit, but for n = 20, whose sum of squares has an order of
its own; against the generic kernel, whose exponential, divisions and folding
differ, to 1e-5 after two steps, as the other kernels' agreement test has it."""
import numpy as np
import pytest
import torch

from tests.cases import GAMMA_DEFAULTS, pf_case

pytestmark = pytest.mark.gpu
COUNTS = (10, 12, 14, 16, 18, 20, 22, 24)
DT = 1e-8


@pytest.fixture(scope="module", autouse=True)
def _built():
    from jax_am_gb300 import _build, _lib
    _build.build()
    yield
    lib = _lib.load()
    lib.pfg_set_kernel_variant(0)
    lib.pfg_tune(3, 0)
    assert _lib.device_error() == 0, "a bounded device-side wait ran out"


def _case(n, aniso, bc, shape, force=False):
    """Random cells in the upper half, grains with exact zeros in the lower one
    (vectors that are zero across a warp are skipped)."""
    from jax_am_gb300.phase_field.allen_cahn import PFSolver
    poly, eta, T, pf_args, _, _ = pf_case(shape, n, aniso, seed=n, bc=bc, noise=0.6, force=force)
    nx, ny, nz = shape
    e = eta.reshape(nz, ny, nx, n)
    e[: nz // 2] = 0.0
    e[: nz // 2, :, : nx // 2, 1] = 1.0
    e[: nz // 2, :, nx // 2:, n - 1] = 1.0
    return (PFSolver(pf_args, poly), torch.tensor(eta, dtype=torch.float32, device="cuda"),
            torch.tensor(T, dtype=torch.float32, device="cuda"))


def _source(name, solver, T):
    from jax_am_gb300.phase_field.allen_cahn import Quench
    from jax_am_gb300.phase_field.coupling import InterpolatedT
    from jax_am_gb300.phase_field.point_source import PointSource
    if name == "array":
        return T
    if name == "quench":
        return Quench(1623.0, 2e7, 0.1, z0=0.4 * solver.params.nz * solver.params.h_z)
    if name == "point":
        return PointSource([0.0, DT], [8e-6, 8.1e-6], 9e-6, 1.4e-5, (0.6, 0.8, 0.0), 25.0, 0.8,
                           300.0, T_clip=2000.0)
    return InterpolatedT(T, T + 40.0, 3 * DT, 4 * DT)


def _steps(name, solver, eta, T, steps=2):
    """(eta, ghosted T or None) after the steps."""
    from jax_am_gb300.runner import HeatPFRun, single_track
    if name == "heat":
        p = solver.params
        Tg = torch.nn.functional.pad(T.view(1, 1, p.nz, p.ny, p.nx), (1,) * 6, mode="replicate")
        run = HeatPFRun(solver, dict(GAMMA_DEFAULTS), single_track(5e-6, 9e-6, 0.8, 200.0, 1.0),
                        dt=DT, eta0=eta, T_init=Tg, compensated=False)
        run.run(steps, graph=False)
        return run.state, run.T_ghosted
    state, t = (eta, 0.0), 0.0
    for _ in range(steps):
        t += DT
        state, _ = solver.stepper(state, t, [_source(name, solver, T)])
    return state[0], None


def _with(variant, chunks, f):
    from jax_am_gb300 import _lib
    lib = _lib.load()
    assert lib.pfg_set_kernel_variant(variant) == 0 and lib.pfg_tune(3, chunks) == 0
    try:
        return f()
    finally:
        lib.pfg_set_kernel_variant(0)
        lib.pfg_tune(3, 0)


def _geometry(n, kind):
    if kind == "neumann":
        return None, (34, 23, 17)
    if n % 4 == 0:  # whole 16-byte vectors: any nx, periodic x
        return "periodic", (45, 19, 13)
    return ("neumann", "periodic", "periodic"), (46, 19, 13)


@pytest.mark.parametrize("aniso", [0.0, 0.15])
@pytest.mark.parametrize("kind", ["neumann", "periodic"])
@pytest.mark.parametrize("n", COUNTS)
def test_lane_kernel_agrees_with_the_others(n, kind, aniso):
    from jax_am_gb300 import _lib
    bc, shape = _geometry(n, kind)
    solver, eta, T = _case(n, aniso, bc, shape, force=kind == "periodic")
    assert solver.N >= 8192
    plan = _lib.describe_plan(solver.params)
    assert plan["kernel"] == 4 and plan["vec"] == (4 if n % 4 == 0 else 2), plan
    assert _with(0, 1, lambda: _lib.describe_plan(solver.params))["planes_per_unit"] == shape[2]
    # (the fused heat step takes Neumann axes alone)
    for name in ("array", "quench", "point", "interp") + (("heat",) if bc is None else ()):
        def run():
            return _steps(name, solver, eta, T)
        got, one = _with(0, 0, run), _with(0, 1, run)
        tma, generic = _with(3, 0, run), _with(1, 0, run)
        assert bool(got[0].isfinite().all()) and float((got[0] - eta).abs().max()) > 1e-4, name
        assert torch.equal(got[0], one[0]), name
        if n == 20:
            assert float((got[0] - tma[0]).abs().max()) <= 1e-6, name
        else:
            assert torch.equal(got[0], tma[0]), name
        assert float((got[0] - generic[0]).abs().max()) <= 1e-5, name
        if name == "heat":
            assert torch.equal(got[1], one[1]) and torch.equal(got[1], tma[1])


@pytest.mark.parametrize("n", [10, 16, 18, 24])
def test_lane_kernel_non_finite_temperatures(n):
    """NaN, infinite and zero temperatures and a NaN cell: what the TMA-fed
    kernel, which skips nothing, gives."""
    solver, eta, T = _case(n, 0.15, None, (34, 23, 17))
    T = T.clone()
    T[17], T[4000], T[9000] = float("nan"), float("inf"), 0.0
    eta[6001, n // 2] = float("nan")
    got = _with(0, 0, lambda: _steps("array", solver, eta, T))[0]
    ref = _with(3, 0, lambda: _steps("array", solver, eta, T))[0]
    assert bool(ref.isnan().any())
    assert torch.equal(got.isnan(), ref.isnan())
    assert torch.equal(got.nan_to_num(), ref.nan_to_num())


@pytest.mark.parametrize("n", COUNTS)
def test_lane_kernel_starts_at_its_cell_count(n):
    """8191 cells take the TMA-fed kernel, 8192 this one (20 orientations at
    any count)."""
    from jax_am_gb300 import _lib
    for shape, kernel in (((64, 16, 8), 4), ((30, 21, 13), 4 if n == 20 else 3)):
        solver, _, _ = _case(n, 0.0, None, shape)
        assert _lib.describe_plan(solver.params)["kernel"] == kernel, shape
