"""Parity of the GPU implicit CFD solver (``jax_am_gb300.cfd.cfd_am.AM_3d``)
with the reference: the golden vectors of the reference's own ``cfd_am.py``
(``tests/golden/cfd_am3d.npz``) and, at a larger size, the FP64 oracle
(``oracle/cfd_oracle.py``), which those vectors pin.

Both sides are float64; they differ only in the summation order of the
Krylov dot products, so fields agree to far below 1e-7 of their scale after
several steps and the iteration counts agree (a solve that stops right at
its threshold may take an iteration more or less; the unpreconditioned
pressure Poisson at tol 1e-10, whose residual creeps along the threshold, up
to about a tenth more or less, with fields still within 1e-10).
"""
import os

import numpy as np
import pytest
import torch

from jax_am_gb300.cfd import cfd_am as G
from oracle import cfd_oracle as C
from tests.test_oracle_cfd import CASES, G as GOLD

pytestmark = pytest.mark.gpu

FIELDS = ("T", "vel", "conv_T", "conv", "grad_p0", "solidID")
RTOL = 1e-8


def gpu_solver(args, N, NL, h, cp, k, data_dir=None):
    a = dict(args, cp=G.LinearClip(*cp), k=G.LinearClip(*k))
    a["mesh"] = G.mesh3d([N[0] * h, N[1] * h, N[2] * h], N)
    a["mesh_local"] = G.mesh3d([NL[0] * h, NL[1] * h, NL[2] * h], NL)
    if data_dir:
        a["data_dir"], a["write_sol_interval"] = data_dir, 1
    return G.AM_3d(a)


def oracle_solver(args, N, NL, h, cp, k):
    a = dict(args, cp=C.LinClip(*cp), k=C.LinClip(*k))
    return C.AM3d(a, C.Mesh([N[0] * h, N[1] * h, N[2] * h], N),
                  C.Mesh([NL[0] * h, NL[1] * h, NL[2] * h], NL))


def close(got, ref, rtol=RTOL):
    got = got.detach().cpu().numpy().reshape(ref.shape)
    scale = max(float(np.abs(ref).max()), 1.0)
    return float(np.abs(got - ref).max()) <= rtol * scale, float(np.abs(got - ref).max()), scale


@pytest.mark.parametrize("name", sorted(CASES))
def test_am3d_golden(name):
    h = float(GOLD["h"])
    N = [int(v) for v in GOLD["grid"]]
    NL = [int(v) for v in GOLD["local"]]
    s = gpu_solver(CASES[name], N, NL, h, tuple(GOLD["cp"]), tuple(GOLD["k"]))
    for step in range(int(GOLD["steps"])):
        s.time_integration()
        torch.cuda.synchronize()
        for f in FIELDS:
            ok, err, scale = close(getattr(s, f), GOLD[f"{name}_{f}"][step])
            assert ok, (name, step, f, err, scale)
    assert float(s.T.max()) > 1623.0 and float(s.vel.abs().max()) > 1e-3


def test_am3d_oracle_larger():
    """36 x 20 x 10 cells, a 20 x 10 x 6 box, the beam crossing one cell per
    step: four steps against the oracle, fields and iteration counts."""
    h = 5e-6
    args = dict(CASES["surface"], P=60.0, speed=2.5, X0=[4e-5, 5e-5, 5e-5])
    N, NL = [36, 20, 10], [20, 10, 6]
    cp, k = (0.2441, 338.39, 300.0, 1563.0), (0.0163105, 4.5847, 300.0, 1563.0)
    s = gpu_solver(args, N, NL, h, cp, k)
    o = oracle_solver(args, N, NL, h, cp, k)
    report = []
    for step in range(4):
        s.time_integration()
        o.time_integration()
        torch.cuda.synchronize()
        rel = {}
        for f in FIELDS:
            ok, err, scale = close(getattr(s, f), getattr(o, f), 1e-7)
            rel[f] = err / scale
        it, oi = s.iterations(), o.last_iters
        report.append((step, rel, it, oi["newton"], oi["energy_lin"], oi["velocity"]))
    msg = "\n".join(str(r) for r in report)
    for step, rel, it, newton, lin, vel in report:
        assert max(rel.values()) <= 1e-7, msg
        # A BiCGSTAB stop compares |r|^2 with tol^2 |b|^2.  With another
        # summation order a solve that ends at its threshold may stop an
        # iteration earlier or later; the unpreconditioned pressure Poisson
        # at tol 1e-10 creeps along its threshold, so its count is only
        # bounded.  The fields above are the parity criterion.
        assert it["newton"] == newton, msg
        assert abs(it["energy_krylov"] - sum(lin)) <= it["newton"], msg
        assert all(abs(a - b) <= 1 for a, b in zip(it["momentum_krylov"], vel[:3])), msg
        assert abs(it["pressure_krylov"] - vel[3]) <= max(8, 0.15 * vel[3]), msg
    assert float(s.T.max()) > 1623.0


def test_coupling_transpose_and_outputs(tmp_path):
    """The coupled driver's convert_temperature on the solver's T, the VTU
    output and inspect_sol's NaN check."""
    from jax_am_gb300.phase_field.coupling import convert_temperature
    from jax_am_gb300.phase_field.vtu import read_vtu
    h = float(GOLD["h"])
    N = [int(v) for v in GOLD["grid"]]
    NL = [int(v) for v in GOLD["local"]]
    s = gpu_solver(CASES["surface"], N, NL, h, tuple(GOLD["cp"]), tuple(GOLD["k"]),
                   data_dir=str(tmp_path))
    s.time_integration()
    T_pf = convert_temperature(s.T[:, :, :, 0])
    ref = np.transpose(s.T[:, :, :, 0].cpu().numpy(), (2, 1, 0)).reshape(-1, 1)
    assert np.array_equal(T_pf.cpu().numpy(), ref.astype(np.float32))
    path = s.write_sols(1)
    data = read_vtu(path)
    assert np.allclose(data["T"].reshape(N[2], N[1], N[0]),
                       np.transpose(s.T[..., 0].cpu().numpy(), (2, 1, 0)), rtol=1e-6)
    assert data["vel"].shape == (np.prod(N), 3)
    s.inspect_sol(1, 1)
    s.T[0, 0, 0, 0] = float("nan")
    with pytest.raises(ValueError):
        s.inspect_sol(1, 1)
    assert os.path.exists(path)


def test_coupled_driver_loop_vs_oracles():
    """The coupled driver's loop (applications/phase_field/coupled/
    example.py:86-111): the CFD solver every 1e-6 s, the phase field every
    2e-7 s on the same 12 x 8 x 5 grid, fed r T_past + (1 - r) T_future
    through InterpolatedT.  The same loop with the float64 CFD oracle and the
    float64 phase-field oracle fed the same float32 interpolated fields gives
    the reference: eta within 1e-4, argmax maps exact."""
    from jax_am_gb300.phase_field.allen_cahn import PFSolver
    from jax_am_gb300.phase_field.coupling import InterpolatedT, convert_temperature
    from oracle import pf_oracle as O
    from tests.cases import f32, pf_case
    h = float(GOLD["h"])
    N = [int(v) for v in GOLD["grid"]]
    NL = [int(v) for v in GOLD["local"]]
    cfd = gpu_solver(CASES["surface"], N, NL, h, tuple(GOLD["cp"]), tuple(GOLD["k"]))
    ocfd = oracle_solver(CASES["surface"], N, NL, h, tuple(GOLD["cp"]), tuple(GOLD["k"]))
    poly, eta, _, pf_args, oargs, _ = pf_case(tuple(N), 6, 0.15, seed=11, h=(h, h, h), noise=0.3)
    pf = PFSolver(pf_args, poly)
    dt_pf, dt_cfd = 2e-7, float(CASES["surface"]["dt"])
    pf_ts = np.arange(0.0, 3e-6 + 1e-10, dt_pf)

    def fields():
        return (cfd.T[:, :, :, 0].clone(), np.float32(ocfd.T))

    T_past, oT_past = fields()
    cfd.time_integration()
    ocfd.time_integration()
    T_future, oT_future = fields()
    t_cfd = dt_cfd
    state = (torch.tensor(eta, dtype=torch.float32, device="cuda"), float(pf_ts[0]))
    e_ref = eta.astype(np.float64)
    hot = 0
    for t_pf in pf_ts[1:]:
        if t_pf > t_cfd + dt_cfd:
            cfd.time_integration()
            ocfd.time_integration()
            T_past, oT_past = T_future, oT_future
            T_future, oT_future = fields()
            t_cfd += dt_cfd
        src = InterpolatedT(convert_temperature(T_past), convert_temperature(T_future), t_cfd,
                            dt_cfd)
        t_prev = state[1]
        state, _ = pf.stepper(state, float(t_pf), [src])
        r = np.float32((t_cfd - t_pf) / dt_cfd)
        Tmix = r * oT_past + (np.float32(1.0) - r) * oT_future
        T_cells = f32(np.transpose(Tmix, (2, 1, 0)).reshape(-1, 1))
        hot = max(hot, int((T_cells > 1623.0).sum()))
        e_ref = O.explicit_euler(e_ref, t_prev, float(t_pf), T_cells, oargs,
                                 poly.unique_grain_directions)
    got = state[0].double().cpu().numpy()
    err = float(np.abs(got - e_ref).max())
    mism = int(np.sum(np.argmax(got, axis=1) != np.argmax(e_ref, axis=1)))
    assert hot > 0, "the coupled case must melt"
    assert err <= 1e-4 and mism == 0, (err, mism)


def test_am3d_local_spacing_differs():
    """The reference's CFD driver builds its flow box with a spacing that
    differs from the global grid's (applications/cfd/simple/example.py:31-33:
    0.5 of the domain over round(0.5 Ny) cells): the flow solve uses the
    box's spacing, the convective terms the global one.  Three steps against
    the oracle on 30 x 21 x 10 cells with a 15 x 10 x 4 box."""
    h = 5e-6
    N = [30, 21, 10]
    dom = [N[0] * h, N[1] * h, N[2] * h]
    NL = [round(0.5 * N[0]), round(0.5 * N[1]), round(0.4 * N[2])]
    dom_l = [0.5 * dom[0], 0.5 * dom[1], 0.4 * dom[2]]
    args = dict(CASES["surface"], P=40.0, speed=2.5, X0=[4e-5, 5e-5, 5e-5])
    cp, k = (0.2441, 338.39, 300.0, 1563.0), (0.0163105, 4.5847, 300.0, 1563.0)
    a = dict(args, cp=G.LinearClip(*cp), k=G.LinearClip(*k))
    a["mesh"], a["mesh_local"] = G.mesh3d(dom, N), G.mesh3d(dom_l, NL)
    assert a["mesh_local"].dX[1] != a["mesh"].dX[1]
    s = G.AM_3d(a)
    o = C.AM3d(dict(args, cp=C.LinClip(*cp), k=C.LinClip(*k)), C.Mesh(dom, N), C.Mesh(dom_l, NL))
    for step in range(3):
        s.time_integration()
        o.time_integration()
        torch.cuda.synchronize()
        for f in FIELDS:
            ok, err, scale = close(getattr(s, f), getattr(o, f), 1e-7)
            assert ok, (step, f, err, scale)
    assert float(s.T.max()) > 1623.0 and float(s.vel.abs().max()) > 0.0


@pytest.mark.parametrize("N,NL,heat_source", [([10, 8, 5], [10, 8, 5], 0),
                                              ([9, 7, 1], [5, 4, 1], 0),
                                              ([12, 9, 6], [12, 9, 6], 1)])
def test_am3d_edge_shapes(N, NL, heat_source):
    """A flow box equal to the whole grid (the reference's drivers allow
    mesh_local = mesh, applications/cfd/simple/example.py:30) and a single
    layer of cells (top and bottom faces on the same cells): two steps
    against the oracle."""
    h = 5e-6
    args = dict(CASES["surface"] if heat_source == 0 else CASES["body"], P=40.0, speed=2.5,
                X0=[2e-5, 2e-5, N[2] * h])
    cp, k = (0.2441, 338.39, 300.0, 1563.0), (0.0163105, 4.5847, 300.0, 1563.0)
    s = gpu_solver(args, N, NL, h, cp, k)
    o = oracle_solver(args, N, NL, h, cp, k)
    for step in range(2):
        s.time_integration()
        o.time_integration()
        torch.cuda.synchronize()
        for f in FIELDS:
            ok, err, scale = close(getattr(s, f), getattr(o, f), 1e-7)
            assert ok, (N, NL, step, f, err, scale)


@pytest.mark.parametrize("N,NL,cells_per_thread", [
    ([16, 8, 8], [16, 8, 8], 4),     # 1024 cells: one whole block
    ([18, 9, 7], [16, 9, 7], 4),     # two blocks; one block of 1008 cells
    ([17, 11, 11], [13, 11, 9], 4),  # three blocks (half a CTA idle); two
    ([17, 11, 11], [13, 11, 9], 8),  # more cells per thread: a launch per operation
])
def test_am3d_solver_block_edges(N, NL, cells_per_thread):
    """The one-launch solve at the edges of its blocks, and the launches per
    operation that larger systems take, against the oracle: two steps."""
    from jax_am_gb300 import _lib
    h = 5e-6
    args = dict(CASES["surface"], P=40.0, speed=2.5, X0=[4e-5, 3e-5, N[2] * h])
    cp, k = (0.2441, 338.39, 300.0, 1563.0), (0.0163105, 4.5847, 300.0, 1563.0)
    lib = _lib.load()
    assert lib.pfg_tune(6, cells_per_thread) == 0
    try:
        s = gpu_solver(args, N, NL, h, cp, k)
        o = oracle_solver(args, N, NL, h, cp, k)
        for step in range(2):
            s.time_integration()
            o.time_integration()
            torch.cuda.synchronize()
            for f in FIELDS:
                ok, err, scale = close(getattr(s, f), getattr(o, f), 1e-7)
                assert ok, (N, NL, step, f, err, scale)
    finally:
        lib.pfg_tune(6, 0)


def _box_case(N, NL, seed=0, **more):
    """A solver on N cells with a box of NL, a melt pool and a flow in it."""
    h = 5e-6
    args = dict(CASES["surface"], P=60.0, speed=2.5,
                X0=[0.3 * N[0] * h, 0.5 * N[1] * h, N[2] * h], **more)
    s = gpu_solver(args, N, NL, h, (0.2441, 338.39, 300.0, 1563.0),
                   (0.0163105, 4.5847, 300.0, 1563.0))
    g = torch.Generator(device="cuda").manual_seed(seed)
    x, y, z = torch.meshgrid(*((torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) * h - b
                               for n, b in zip(N, args["X0"])), indexing="ij")
    w = 0.25 * N[1] * h
    T = 300.0 + 2300.0 * torch.exp(-(x * x + y * y) / w ** 2 + 2.0 * z / w)
    s.T.copy_(T[..., None])
    s.vel.copy_(0.05 * torch.randn(s.vel.shape, generator=g, device="cuda", dtype=torch.float64) *
                (T > 1623.0)[..., None])
    return s


def _fields(s):
    return {f: getattr(s, f).clone() for f in FIELDS}


def test_timed_out_solves_leave_the_fields():
    """The wait probe makes the waits of the solves that run in one launch run
    out (10 us): an error, fields as they were, and the next step without the
    probe gives what a solver that never timed out gives.  In the second case
    the energy solve takes the launches of each iteration, which wait for
    nothing, so that the flow solves' waits run out."""
    from jax_am_gb300 import _lib
    lib = _lib.load()
    for N, NL in (([24, 14, 9], [14, 9, 6]), ([120, 60, 50], [30, 20, 12])):
        s, clean = _box_case(N, NL), _box_case(N, NL)
        clean.time_integration()
        before = _fields(s)
        assert lib.pfg_tune(8, 20000) == 0
        try:
            with pytest.raises(_lib.PFGError, match="TIMEOUT"):
                s.time_integration()
            torch.cuda.synchronize()
        finally:
            assert lib.pfg_tune(8, 0) == 0
        flow = ("vel", "conv_T", "conv", "grad_p0")
        energy_done = N[0] == 120
        for f in flow if energy_done else FIELDS:
            assert torch.equal(getattr(s, f), before[f]), f
        if energy_done:
            assert torch.equal(s.T, clean.T)
            s.T, s.solidID = before["T"], before["solidID"]
        s.time_integration()
        for f in FIELDS:
            assert torch.equal(getattr(s, f), getattr(clean, f)), f
        assert s.iterations() == clean.iterations()


@pytest.mark.parametrize("form", [1, 2], ids=["launches", "refused"])
@pytest.mark.parametrize("N,NL", [([7, 5, 3], [5, 3, 2]), ([37, 19, 13], [23, 17, 11]),
                                  ([60, 41, 15], [45, 31, 14]),
                                  ([101, 60, 50], [96, 56, 50])])
def test_both_forms_of_a_solve_agree(N, NL, form):
    """Two steps with the solves in one launch each (pfg_tune key 9 = 0) and in
    five launches an iteration, asked for (1) or because the one launch is
    refused (2): the same fields bit for bit and the same iteration counts, for
    systems of one 256-thread block to more than 256 (303,000 and 268,800
    cells)."""
    from jax_am_gb300 import _lib
    lib = _lib.load()
    a, b = _box_case(N, NL), _box_case(N, NL)
    for _ in range(2):
        a.time_integration()
        assert lib.pfg_tune(9, form) == 0
        try:
            b.time_integration()
        finally:
            assert lib.pfg_tune(9, 0) == 0
        assert a.iterations() == b.iterations()
        for f in FIELDS:
            assert torch.equal(getattr(a, f), getattr(b, f)), f
    assert a.iterations()["pressure_krylov"] > 2 and float(a.vel.abs().max()) > 1e-4


def test_solves_of_several_threads():
    """Two threads with a stream each, their solves' launches wanting every SM:
    each gives what it gives alone."""
    import threading
    N, NL = [101, 60, 50], [96, 56, 50]
    alone = [_box_case(N, NL, seed=k) for k in range(2)]
    for s in alone:
        s.time_integration()
    both = [_box_case(N, NL, seed=k) for k in range(2)]
    torch.cuda.synchronize()
    errors = []

    def work(s):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                s.time_integration()
                torch.cuda.current_stream().synchronize()
        except Exception as e:
            errors.append(e)
    threads = [threading.Thread(target=work, args=(s,)) for s in both]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for s, r in zip(both, alone):
        for f in FIELDS:
            assert torch.equal(getattr(s, f), getattr(r, f)), f
