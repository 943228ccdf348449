"""The hand-written adjoint of the fused heat + phase-field run against float64
autograd of the oracle's PyTorch restatement (the stand-in for the
reference's jax.grad) and against central finite differences at 1e-3
relative.  Tolerance: 2e-2 relative on dJ/dP and dJ/dv, 2e-2 relative
(l2) on dJ/d eta0 (the GPU forward and adjoint are float32)."""
import numpy as np
import pytest
import torch

from oracle import pf_torch as PT
from tests.cases import GAMMA_DEFAULTS, f32, pf_case

pytestmark = pytest.mark.gpu
GRAD_RTOL = 2e-2


@pytest.fixture(scope="module", autouse=True)
def _built():
    from jax_am_gb300 import _build
    _build.build()


def _setup(aniso, steps, ckpt, shape=(10, 8, 6), n=4, seed=3):
    poly, eta, _, pf_args, oargs, _ = pf_case(shape, n, aniso, seed=seed, h=(1e-6,) * 3,
                                              noise=0.6)
    nx, ny, nz = shape
    rng = np.random.default_rng(seed + 1)
    Tg = f32(rng.uniform(1000.0, 1400.0, (nz + 2, ny + 2, nx + 2)))
    g = dict(GAMMA_DEFAULTS, r=8e-6)
    w = f32(rng.random(n))
    return poly, eta, Tg, pf_args, oargs, g, w


def _torch_J(P, v, eta0, Tg, oargs, g, w, dirs, steps, dt, x_start, y, shape):
    nx, ny, nz = shape
    e = eta0.reshape(nz, ny, nx, -1)
    T = Tg
    t = 0.0
    for _ in range(steps):
        def laser(tm, P=P, v=v):
            return x_start + v * tm, y, P
        e, T = PT.coupled_step(e, T, t, dt, oargs, g, laser, dirs)
        t += dt
    return torch.mean(torch.sum(w * e.reshape(-1, e.shape[-1]) ** 2, dim=1))


@pytest.mark.parametrize("aniso,steps,ckpt", [(0.0, 12, 5), (0.15, 10, 4)])
def test_adjoint_matches_float64_autograd_and_fd(aniso, steps, ckpt):
    from jax_am_gb300.adjoint import HeatPFObjective, LaserTrackProblem
    shape = (10, 8, 6)
    poly, eta, Tg, pf_args, oargs, g, w = _setup(aniso, steps, ckpt, shape)
    dt = float(np.float32(3e-8))
    x_start, y = 2e-6, 4e-6
    P0, v0 = 2.0, 0.8
    prob = LaserTrackProblem(pf_args, poly, g, w, dt, steps, x_start, y, checkpoint_every=ckpt,
                             T_init=torch.tensor(Tg))
    # the GPU run through the autograd node
    P = torch.tensor(P0, dtype=torch.float64, requires_grad=True)
    v = torch.tensor(v0, dtype=torch.float64, requires_grad=True)
    e0 = torch.tensor(eta, dtype=torch.float32, device="cuda", requires_grad=True)
    J = HeatPFObjective.apply(P, v, e0, prob)
    J.backward()
    gP, gv, ge = P.grad.item(), v.grad.item(), e0.grad.double().cpu().numpy()

    # float64 autograd of the oracle restatement
    dirs = torch.tensor(poly.unique_grain_directions)
    Pt = torch.tensor(P0, dtype=torch.float64, requires_grad=True)
    vt = torch.tensor(v0, dtype=torch.float64, requires_grad=True)
    et = torch.tensor(eta, dtype=torch.float64, requires_grad=True)
    wt = torch.tensor(w)
    Tt = torch.tensor(Tg)
    Jt = _torch_J(Pt, vt, et, Tt, oargs, g, wt, dirs, steps, dt, x_start, y, shape)
    Jt.backward()
    rP = abs(gP - Pt.grad.item()) / abs(Pt.grad.item())
    rv = abs(gv - vt.grad.item()) / abs(vt.grad.item())
    ref_e = et.grad.numpy()
    re = np.linalg.norm(ge - ref_e) / np.linalg.norm(ref_e)
    print(f"A={aniso}: J gpu {J.item():.8e} vs f64 {Jt.item():.8e}; "
          f"dJ/dP {gP:.6e} vs {Pt.grad.item():.6e} (rel {rP:.2e}); "
          f"dJ/dv {gv:.6e} vs {vt.grad.item():.6e} (rel {rv:.2e}); dJ/deta0 rel {re:.2e}")
    assert abs(J.item() - Jt.item()) <= 1e-5 * abs(Jt.item())
    assert rP <= GRAD_RTOL and rv <= GRAD_RTOL and re <= GRAD_RTOL

    # central finite differences at 1e-3 relative on the float64 forward
    with torch.no_grad():
        def Jf(Pv, vv, ev):
            return _torch_J(torch.tensor(Pv), torch.tensor(vv), ev, Tt, oargs, g, wt, dirs, steps,
                            dt, x_start, y, shape).item()
        eps = 1e-3
        fdP = (Jf(P0 * (1 + eps), v0, torch.tensor(eta)) -
               Jf(P0 * (1 - eps), v0, torch.tensor(eta))) / (2 * eps * P0)
        fdv = (Jf(P0, v0 * (1 + eps), torch.tensor(eta)) -
               Jf(P0, v0 * (1 - eps), torch.tensor(eta))) / (2 * eps * v0)
        rng = np.random.default_rng(9)
        dirn = rng.standard_normal(eta.shape)
        he = 1e-3
        fde = (Jf(P0, v0, torch.tensor(eta + he * dirn)) -
               Jf(P0, v0, torch.tensor(eta - he * dirn))) / (2 * he)
    rfP = abs(gP - fdP) / abs(fdP)
    rfv = abs(gv - fdv) / abs(fdv)
    rfe = abs(np.sum(ge * dirn) - fde) / abs(fde)
    print(f"   FD: dJ/dP {fdP:.6e} (rel {rfP:.2e}), dJ/dv {fdv:.6e} (rel {rfv:.2e}), "
          f"directional dJ/deta0 {fde:.6e} (rel {rfe:.2e})")
    assert rfP <= GRAD_RTOL and rfv <= GRAD_RTOL and rfe <= GRAD_RTOL
    from jax_am_gb300 import _lib
    assert _lib.device_error() == 0


@pytest.mark.parametrize("shape,n,ckpt,aniso", [((13, 7, 5), 10, 3, 0.0), ((25, 6, 4), 5, 4, 0.0),
                                                ((3, 13, 9), 33, 7, 0.0), ((4, 5, 2), 64, 1, 0.0),
                                                ((9, 7, 5), 7, 3, 0.15)])
def test_adjoint_tile_edges(shape, n, ckpt, aniso):
    """Partial tiles, odd orientation counts (a lane with one orientation) and
    one cell per warp, against float64 autograd to 1e-3 relative (float32
    fields: about 1e-6); a second gradient() of the same forward(), after the
    caller has overwritten eta0, gives the same."""
    from jax_am_gb300.adjoint import LaserTrackProblem
    steps = 7
    poly, eta, Tg, pf_args, oargs, g, w = _setup(aniso, steps, ckpt, shape, n)
    dt, x_start, y, P0, v0 = float(np.float32(3e-8)), 1e-6, 2e-6, 2.0, 0.8
    prob = LaserTrackProblem(pf_args, poly, g, w, dt, steps, x_start, y, checkpoint_every=ckpt,
                             T_init=torch.tensor(Tg))
    e0 = torch.tensor(eta, dtype=torch.float32, device="cuda")
    J = prob.forward(P0, v0, e0)
    e0.zero_()
    gP, gv, ge = prob.gradient()
    gP2, gv2, ge2 = prob.gradient()
    assert torch.equal(ge, ge2) and abs(gP - gP2) <= 1e-12 * abs(gP)
    leaves = [torch.tensor(x, dtype=torch.float64, requires_grad=True) for x in (P0, v0, eta)]
    Jt = _torch_J(*leaves, torch.tensor(Tg), oargs, g, torch.tensor(w),
                  torch.tensor(poly.unique_grain_directions), steps, dt, x_start, y, shape)
    Jt.backward()
    rP, rv, re = (x.grad.numpy() for x in leaves)
    assert abs(J - Jt.item()) <= 1e-5 * abs(Jt.item())
    assert abs(gP - rP) <= 1e-3 * abs(rP) and abs(gv - rv) <= 1e-3 * abs(rv)
    assert np.linalg.norm(ge.double().cpu().numpy() - re) <= 1e-3 * np.linalg.norm(re)


@pytest.mark.parametrize("shape,n", [((1, 1, 1), 1), ((5, 3, 2), 3), ((13, 7, 5), 10),
                                     ((37, 31, 23), 64), ((80, 75, 64), 7)])
def test_objective_in_float64(shape, n):
    """J of values over float32's whole range against the exact sum; the bound
    is one rounding of 2^-53 per addition of the longest chain (a thread's
    elements, the trees, the blocks).  A diverged state's J is infinite."""
    import ctypes
    import math
    from jax_am_gb300 import _lib
    from jax_am_gb300.phase_field.allen_cahn import make_pf_params
    lib = _lib.load()
    nx, ny, nz = shape
    N = nx * ny * nz
    poly, _, _, pf_args, _, _ = pf_case(shape, n, 0.0, seed=2, h=(1e-6,) * 3)
    p = make_pf_params(pf_args, poly)
    rng = np.random.default_rng(n)
    eta, w = f32(rng.standard_normal((N, n))), f32(rng.random(n) - 0.2)
    w = np.where(np.abs(w) < 1e-3, 0.5, w)

    def J_of(eta):
        e = torch.tensor(eta, dtype=torch.float32, device="cuda")
        J = torch.zeros(1, dtype=torch.float64, device="cuda")
        lam = torch.empty_like(e)
        wd = torch.tensor(w, dtype=torch.float32, device="cuda")
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        for seed in (None, lam):
            J.zero_()
            _lib.check(lib.pfg_objective(ctypes.byref(p), _lib.ptr(e), _lib.ptr(wd), _lib.ptr(J),
                                         _lib.ptr(seed), stream), "pfg_objective")
        return J.item(), lam
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    threads = min(N * n, sms * 8 * 256) // 2
    roundings = N * n / max(1, threads) + 16 + 8 * sms
    for scale in (1.0, 1e18, 1e25, 1e-25, 1e-37):
        x = f32(eta * scale)
        J, lam = J_of(x)
        terms = (w * x * x).reshape(-1)
        exact, size = math.fsum(terms), math.fsum(np.abs(terms))
        assert abs(J - exact / N) <= roundings * 2.0 ** -53 * size / N, scale
        ref = np.float32(2) * np.float32(w) * np.float32(x) * (np.float32(1) / np.float32(N))
        with np.errstate(over="ignore"):
            np.testing.assert_array_equal(lam.cpu().numpy(), ref)
    eta[N // 2, n // 2] = np.inf
    assert J_of(eta)[0] == math.copysign(math.inf, w[n // 2])


def _adjoint_step_inputs(shape, n, aniso, force=False, seed=6):
    """One adjoint step's arguments on random fields, and the call."""
    import ctypes
    from jax_am_gb300 import _lib
    from jax_am_gb300.cfd.gamma import make_heat_params
    from jax_am_gb300.phase_field.allen_cahn import make_pf_params
    lib = _lib.load()
    nx, ny, nz = shape
    poly, eta, _, pf_args, _, _ = pf_case(shape, n, aniso, seed=seed, h=(1e-6,) * 3, force=force)
    p = make_pf_params(pf_args, poly)
    h = make_heat_params(dict(GAMMA_DEFAULTS, r=8e-6), nx, ny, nz, 1e-6, 1e-6, 1e-6,
                         path=[(0.0, 1.0, 2e-6, 3e-6, 1.0, 3e-6, 2.0)])
    g = torch.Generator(device="cuda").manual_seed(seed)
    eta = torch.tensor(eta, dtype=torch.float32, device="cuda")
    lam = torch.randn(eta.shape, generator=g, device="cuda")
    Tg = 1000.0 + 1100.0 * torch.rand((nz + 2, ny + 2, nx + 2), generator=g, device="cuda")
    Tb = torch.randn(Tg.shape, generator=g, device="cuda")
    scratch = torch.empty(int(lib.pfg_adjoint_scratch_bytes(ctypes.byref(p))), dtype=torch.uint8,
                          device="cuda")

    def step(eta, lam, lam_out, Tb_out):
        grads = torch.zeros(2, dtype=torch.float64, device="cuda")
        st = lib.pfg_adjoint_step(ctypes.byref(p), ctypes.byref(h), _lib.ptr(eta), _lib.ptr(Tg),
                                  0.0, 3e-8, _lib.ptr(lam), _lib.ptr(Tb), _lib.ptr(lam_out),
                                  _lib.ptr(Tb_out), _lib.ptr(scratch), scratch.numel(),
                                  _lib.ptr(grads), 1e-3,
                                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        _lib.check(st, "pfg_adjoint_step")
        return grads
    return eta, lam, Tg, Tb, step


@pytest.mark.parametrize("aniso", [0.0, 0.15])
@pytest.mark.parametrize("shape,n", [((33, 21, 12), 10), ((14, 9, 5), 7)])
def test_adjoint_step_in_place(shape, n, aniso):
    """lam_out in the place of lam_in or of eta against separate buffers: the
    same kernels with anisotropy, so equal; without it the one-pass kernel's
    results, whose terms (no larger than the largest result) a compiler may
    contract otherwise: 16 roundings of 2^-24."""
    eta, lam, Tg, Tb, step = _adjoint_step_inputs(shape, n, aniso)
    ref, Tref = torch.empty_like(lam), torch.zeros_like(Tb)
    gref = step(eta, lam, ref, Tref)
    for out in ("lam", "eta"):
        e, l, T = eta.clone(), lam.clone(), torch.zeros_like(Tb)
        o = l if out == "lam" else e
        grads = step(e, l, o, T)
        for got, want in ((o, ref), (T, Tref)):
            tol = 0.0 if aniso else 2.0 ** -20 * float(want.abs().max())
            assert float((got - want).abs().max()) <= tol, out
        assert torch.allclose(grads, gref, rtol=1e-12)  # the blocks' order of atomics


def test_steps_and_dt_of_a_problem_may_change():
    """``steps`` and ``dt`` are read at each run: a problem made with others and
    then changed gives what one made with them gives."""
    from jax_am_gb300.adjoint import LaserTrackProblem
    shape, n = (9, 7, 5), 4
    poly, eta, Tg, pf_args, oargs, g, w = _setup(0.0, 7, 3, shape, n)
    e0 = torch.tensor(eta, dtype=torch.float32, device="cuda")

    def problem(steps, dt):
        return LaserTrackProblem(pf_args, poly, g, w, dt, steps, 1e-6, 2e-6, checkpoint_every=3,
                                 T_init=torch.tensor(Tg))
    want, got = problem(7, 3e-8), problem(2, 1e-8)
    got.steps, got.dt, got.t_end = want.steps, want.dt, want.t_end
    res = []
    for p in (want, got):
        J = p.forward(2.0, 0.8, e0)
        res.append((J, *p.gradient()))
    a, b = res
    assert abs(a[0] - b[0]) <= 1e-14 * abs(a[0])
    assert abs(a[1] - b[1]) <= 1e-12 * abs(a[1]) and abs(a[2] - b[2]) <= 1e-12 * abs(a[2])
    assert torch.equal(a[3], b[3])


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_adjoint_step_non_finite_at_liquid_cells(value):
    """A non-finite adjoint at cells that liquid forcing zeroed stays there: the
    one-pass kernel's other cells hold what the kernels that go through
    scratch (lam_out in the place of lam_in) give, finite and equal to 16
    roundings of the largest."""
    from tests.cases import PF_DEFAULTS
    eta, lam, Tg, Tb, step = _adjoint_step_inputs((19, 13, 9), 10, 0.0, force=True)
    T = Tg[1:-1, 1:-1, 1:-1].reshape(-1)
    liquid = T > PF_DEFAULTS["T_liquidus"] + 1.0
    assert 0.2 < float(liquid.float().mean()) < 0.8
    lam[liquid, 3] = value
    out, T_out = torch.empty_like(lam), torch.zeros_like(Tb)
    step(eta, lam, out, T_out)
    ref, T_ref = lam.clone(), torch.zeros_like(Tb)
    step(eta, ref, ref, T_ref)
    assert bool(ref[~liquid].isfinite().all()) and bool(T_ref.isfinite().all())
    assert torch.equal(out.isfinite(), ref.isfinite())
    for got, want in ((out[ref.isfinite()], ref[ref.isfinite()]), (T_out, T_ref)):
        assert float((got - want).abs().max()) <= 2.0 ** -20 * float(want.abs().max())
