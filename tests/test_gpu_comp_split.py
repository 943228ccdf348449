"""The compensated fused step for orientation counts other than 20: the
compensated heat update in its own kernel (``heat_comp.cu``), then the
TMA-fed phase-field kernel with zeta from the start-of-step temperature pair
(``pfg_heat_pf_step_comp``; ``gamma.py:9-61``, ``allen_cahn.py:56-57,
106-114``).  Tolerances as the other laser cases: max |d eta| <= 1e-4,
max |dT| <= 1e-3 K against a float64 run."""
import numpy as np
import pytest
import torch

from tests.laser_parity import T_LIQ, _laser_case

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from jax_am_gb300 import _build
    _build.build()


def _variant(v):
    from jax_am_gb300 import _lib
    assert _lib.load().pfg_set_kernel_variant(v) == 0


def test_split_step_matches_the_lane_kernel():
    """n = 20: the split compensated step (kernel variant 3: the heat kernel,
    then the TMA-fed kernel) against the cell-per-lane kernel's fused one.
    The temperature pairs agree to 1e-6 K (both use the same double-float
    update; which cells take the full double-float path is decided per warp,
    and the warps group cells differently) and eta to 1e-5."""
    from jax_am_gb300.phase_field.allen_cahn import PFSolver
    from jax_am_gb300.phase_field.utils import Field
    from jax_am_gb300.runner import HeatPFRun, single_track
    from jax_am_gb300.workloads import gamma_args
    from tests.laser_parity import PF_KEYS
    pf_args = dict(PF_KEYS, Nx=64, Ny=48, Nz=24, h=1e-6, num_grains=60, num_oris=20,
                   T_liquidus=1623.0, anisotropy=0.15)
    poly = Field(pf_args, seed=8)
    s = PFSolver(pf_args, poly)
    path = single_track(5e-6, 24e-6, 0.8, 200.0, 1e-3)
    out = []
    try:
        for v in (0, 3):
            _variant(v)
            run = HeatPFRun(s, gamma_args(), path, compensated=True)
            run.run(40, graph=False)
            out.append((run.state.double(), run.T_ghosted_f64, float(run.T_ghosted.max())))
    finally:
        _variant(0)
    (e0, T0, m0), (e1, T1, m1) = out
    assert m0 > 500.0  # the beam heated the surface
    dT = float((T0 - T1).abs().max())
    de = float((e0 - e1).abs().max())
    print(f"lane vs split compensated step: max |dT| = {dT:.3e} K, max |d eta| = {de:.3e}")
    assert dT <= 1e-6
    assert de <= 1e-5


@pytest.mark.parametrize("shape,n,steps", [((40, 30, 16), 12, 40), ((48, 32, 16), 30, 40),
                                           ((44, 20, 12), 8, 30)])
def test_split_step_vs_oracle(shape, n, steps):
    from jax_am_gb300.runner import single_track
    nx, ny, nz = shape
    path = single_track(4e-6, 0.5 * ny * 1e-6, 0.8, 200.0, 1e-3)
    with torch.no_grad():
        Tmax = _laser_case(shape, n, 40, 0.15, path, steps, 3,
                           f"compensated split step {nx}x{ny}x{nz} n={n}, {steps} steps",
                           compensated=True)
    assert Tmax > 500.0


def test_multi_track_n30_long_run():
    """A reduced multi-track raster (320 x 160 x 80 cells, n = 30, A = 0.15,
    three 250 W tracks at 1 m/s) over 2000 steps.  With a float32
    temperature the same run leaves the tolerances after about 500 steps
    (1.2 K at step 500, 3.3 K and 1.6e-3 in eta at step 2000: latent-heat and
    zeta switches taken the other way); compensated it stays inside."""
    from jax_am_gb300.runner import raster
    ys = [160e-6 * f for f in (0.3, 0.5, 0.7)]
    path = raster(ys, 1.0, 250.0, 20e-6, 300e-6)
    with torch.no_grad():
        Tmax = _laser_case((320, 160, 80), 30, 1280, 0.15, path, 2000, 5,
                           "multi track 320x160x80 n=30 A=0.15, 2000 steps (compensated)",
                           compensated=True)
    assert Tmax >= T_LIQ, f"the laser never melted the surface (T max {Tmax:.1f} K)"
    torch.cuda.empty_cache()


# ---- one step's rounding -----------------------------------------------------
# Pair arithmetic in which every sum, difference, product and quotient is a
# normalised pair of its own, in NumPy float32 (a fused multiply-add is the
# longdouble value rounded once).
_f, _L = np.float32, np.longdouble


def _two_sum(a, b):
    s = a + b
    bb = s - a
    return s, (a - (s - bb)) + (b - bb)


def _fast(a, b):
    s = a + b
    return s, b - (s - a)


def _fma(a, b, c):
    return (_L(a) * _L(b) + _L(c)).astype(_f)


def _add(x, y):
    s, e = _two_sum(x[0], y[0])
    t, u = _two_sum(x[1], y[1])
    s, e = _fast(s, e + t)
    return _fast(s, e + u)


def _sub(x, y):
    return _add(x, (-y[0], -y[1]))


def _mul(x, y):
    p = x[0] * y[0]
    return _fast(p, _fma(x[0], y[1], _fma(x[1], y[0], _fma(x[0], y[0], -p))))


def _div(x, y):
    z = np.zeros_like(x[0])
    q1 = x[0] / y[0]
    r = _sub(x, _mul(y, (q1, z)))
    q = _fast(q1, r[0] / y[0])
    r = _sub(x, _mul(y, q))
    return _add(q, (r[0] / y[0], z))


def _pair(v, like=None):
    v = np.asarray(v, dtype=np.float64)
    h = v.astype(_f)
    p = h, (v - h).astype(_f)
    return p if like is None else tuple(np.broadcast_to(a, like.shape).astype(_f) for a in p)


@pytest.mark.parametrize("n", [20, 12], ids=["lane", "split"])
@pytest.mark.parametrize("lo,hi", [(400.0, 1540.0), (1575.0, 1610.0), (1640.0, 3000.0),
                                   (3000.0, 9000.0)])
def test_compensated_step_rounds_as_full_pairs(n, lo, hi):
    """One compensated heat step of random temperature pairs against extended
    precision: the root mean square and the largest error of the cells away from
    the faces are those of full pair arithmetic on the same values (2 % and a
    quarter for the sample's spread; low parts summed in float32 add a fifth to
    the former)."""
    from jax_am_gb300.phase_field.allen_cahn import PFSolver
    from jax_am_gb300.runner import HeatPFRun, single_track
    from tests.cases import GAMMA_DEFAULTS, pf_case
    nx, ny, nz = 96, 64, 48
    hx, dt = float(_f(1e-6)), float(_f(2e-8))
    poly, eta, _, pf_args, _, _ = pf_case((nx, ny, nz), n, 0.0, seed=4, h=(hx,) * 3)
    g = dict(GAMMA_DEFAULTS)
    rng = np.random.default_rng(int(lo) + n)
    base = rng.uniform(lo, hi, (nz // 8 + 1, ny // 8 + 1, nx // 8 + 1))
    T = np.kron(base, np.ones((8, 8, 8)))[: nz + 2, : ny + 2, : nx + 2]
    T = T + rng.uniform(-10.0, 10.0, T.shape)
    h, l = _pair(T)
    run = HeatPFRun(PFSolver(pf_args, poly), g, single_track(1e-6, 2e-6, 0.8, 0.0, 1.0), dt=dt,
                    eta0=torch.tensor(eta, dtype=torch.float32, device="cuda"),
                    T_init=torch.tensor(h), compensated=True)
    run.Tl[run.cur].copy_(torch.tensor(l))
    run.run(1, graph=False)
    got = run.T_ghosted_f64.cpu().numpy()[2:-2, 2:-2, 2:-2]

    def at(a, d=(0, 0, 0)):
        return a[tuple(slice(2 + k, m - 2 + k) for k, m in zip(d, a.shape))]
    dirs = [(0, 0, 1), (0, 1, 0), (1, 0, 0)]
    rho, L, Ts, Tl = (float(_f(g[k])) for k in ("rho", "L", "Ts", "Tl"))
    x = _L(h) + _L(l)
    c = at(x)
    clip = np.clip(c, 300.0, _L(Tl))
    k = _L(0.0163) * clip + _L(4.5847)
    cp = _L(0.2441) * clip + _L(338.39) + np.where((c > Ts) & (c < Tl), _L(L), _L(0))
    lap = sum((at(x, d) - c) + (at(x, tuple(-v for v in d)) - c) for d in dirs) / (_L(hx) * _L(hx))
    exact = c + k * _L(dt) / (cp * _L(rho)) * lap

    C = at(h), at(l)
    z = np.zeros_like(C[0])
    cl = tuple(np.where(clip == c, v, w) for v, w in zip(C, (clip.astype(_f), z)))
    kk = _add(_mul(_pair(0.0163, z), cl), _pair(4.5847, z))
    cc = _add(_mul(_pair(0.2441, z), cl), _pair(338.39, z))
    cm = _add(cc, _pair(L, z))
    cc = tuple(np.where((c > Ts) & (c < Tl), a, b) for a, b in zip(cm, cc))
    ll = z, z
    for d in dirs:
        m, p = ((at(h, e), at(l, e)) for e in (tuple(-v for v in d), d))
        ll = _add(ll, _mul(_add(_sub(m, C), _sub(p, C)), _pair(1.0 / (hx * hx), z)))
    coef = _div(_mul(kk, (np.full_like(z, dt), z)), _mul(cc, (np.full_like(z, rho), z)))
    full = _add(C, _mul(coef, ll))
    e_full = np.abs((_L(full[0]) + _L(full[1]) - exact).astype(np.float64))
    e_got = np.abs((_L(got) - exact).astype(np.float64))
    rms = [float(np.sqrt(np.mean(e * e))) for e in (e_got, e_full)]
    print(f"n = {n}, {lo} .. {hi} K: rms {rms[0]:.3e} (full pairs {rms[1]:.3e}), largest "
          f"{e_got.max():.3e} ({e_full.max():.3e}) K")
    assert rms[0] <= 1.02 * rms[1]
    assert e_got.max() <= 1.25 * e_full.max()
