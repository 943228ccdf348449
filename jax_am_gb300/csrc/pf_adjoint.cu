// Hand-written discrete adjoint of the fused heat + phase-field step.
//
// Forward step k (pfg_heat_pf_step): eta' = eta + dt R(eta, T) with
//   R_i = -Lg(T) (m_g/ad_hoc) g_i + Lg(T) kappa_g ad_hoc a_i(e_i) L_i,
//   g_i = eta_i (K - 3 eta_i^2), K = 4 S + 2 (1 - zeta(T))^2 - 1, S = sum eta^2,
//   L_i = sum_d w_d (eta_i(+d) + eta_i(-d) - 2 eta_i), e_i = central differences,
// and T' = H(T; P, x_laser) (explicit heat step whose ghost faces are state).
// Given the adjoints of step k+1 (lam' = dJ/d eta', Tb' = dJ/dTg' including
// the ghost faces) and the forward state of step k, the kernels below produce
// the adjoints of step k and add this step's dJ/dP and dJ/dv.
//
// Transposes used (derived for the reference's edge-replicate Neumann
// boundary, allen_cahn.py:61-66): the Laplacian term transposes to the same
// Laplacian applied to u = lam Lg kappa' a (even extension at a Neumann face);
// the anisotropy term (a depends on e = eta(+d) - eta(-d)) transposes to minus
// the central difference of v_d = lam Lg kappa' L da/de_d with an odd
// extension at a Neumann face; periodic axes wrap in both.
//
// Without anisotropy (a = 1) u at a neighbour is its lam times one number per
// cell, so one launch per cell (heat transpose and the cell coefficients) and
// one per order parameter do the step and no (N, n) field is written but
// lam_out: at 1M cells, n = 10, 128 us a step (9 + 31 + 88) against 230 us with the
// fields written and gathered.  With anisotropy, or with an output in the place of an input, the
// fields u, v and loc go through memory (kernels A, B, then C).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "pfg_device.cuh"
#include "pfg_host.h"
#include "pfg_step.cuh"

namespace pfg {

struct AdjArgs {
  int nx, ny, nz, n;
  int bcx, bcy, bcz;
  float dt;
  PFConsts pc;
  HeatConsts hc;
  float xl, yl, P, dxl_dv;  // beam at mid-step and d x_laser / d v
  int beam_on;
  const float* eta;    // forward eta at step k (nz, ny, nx, n)
  const float* Tg;     // forward ghosted T at step k
  const float* lam_in; // dJ/d eta^{k+1}
  const float* Tb_in;  // dJ/d Tg^{k+1} (ghosted)
  float* lam_out;      // dJ/d eta^k
  float* Tb_out;       // dJ/d Tg^k (ghosted; interior and faces written)
  float* u;            // (N, n)
  float* v;            // 3 x (N, n)
  float* loc;          // (N, n)
  float* muPF;         // (N) dt * sum_i lam_i dR_i/dT
  float* mask;         // (N) 0 where liquid forcing zeroed the cell, else 1
  // isotropic step, per cell: Lg kappa' (-0 where liquid), Lg m_g / ad_hoc,
  // 2 (1 - zeta)^2 (-1 where liquid) and d Lg / dT
  float* q;
  float* g;
  float* om2;
  float* dLg;
  float* alpha;        // (N) thermal diffusivity k / (rho cp)
  int tx, ty, zc, tiles_x, tiles_y;  // isotropic step: tile and planes per unit
  double* grads;       // [dJ/dP, dJ/dv]
  float dirs[3 * PFG_MAX_ORIS * 3];
};

__device__ __forceinline__ int nbr(int i, int d, int n, int periodic) {
  return bc_index(i + d, n, periodic);
}

// d zeta / dT of zeta = (1 - tanh(1e10 (T / T_liq - 1))) / 2 evaluated as the
// float32 step kernel does: the float32 tanh is exactly +-1 unless x == 0.
__device__ __forceinline__ float dzeta_dT(const PFConsts& c, float x) {
  return (x == 0.f) ? -0.5f * 1e10f / c.T_liq : 0.f;
}

// Lane layout of kernels A and B: a cell takes tpc = ceil(n / 2) lanes, each
// lane two consecutive orientations, so a warp holds 32 / tpc cells (for
// n = 10: six cells, 30 of 32 lanes busy).
struct AdjLanes {
  int tpc, cpw, cw, g;
  bool active;
};
__device__ __forceinline__ AdjLanes adj_lanes(int n) {
  AdjLanes l;
  const int lane = threadIdx.x & 31;
  l.tpc = (n + 1) >> 1;
  l.cpw = 32 / l.tpc;
  l.cw = lane / l.tpc;
  l.g = lane - l.cw * l.tpc;
  l.active = l.cw < l.cpw;
  return l;
}
// Sum of v over the tpc lanes of this lane's cell, returned to every lane of
// the cell (a guarded shfl-down tree leaves the sum in the cell's lane 0).
__device__ __forceinline__ float cell_sum(float v, const AdjLanes& l) {
  for (int o = 1; o < l.tpc; o <<= 1) {
    const float t = __shfl_down_sync(0xffffffffu, v, o);
    if (l.g + o < l.tpc) v += t;
  }
  const int lane = threadIdx.x & 31;
  return __shfl_sync(0xffffffffu, v, min(lane - l.g, 31));
}

// The temperature-only quantities of the forward step's arithmetic and their
// derivatives.
struct AdjTemp {
  float om, Lg, dLg, dz;
  bool liquid;
};
__device__ __forceinline__ AdjTemp adj_temp(const PFConsts& pc, float T) {
  AdjTemp r;
  const bool clipped = T > 2000.f;
  const float Tc = clipped ? 2000.f : T;
  const float xz = Tc / pc.T_liq - 1.f;
  const float zeta = (xz > 0.f) ? 0.f : (xz < 0.f) ? 1.f : (xz == 0.f) ? 0.5f : xz;
  r.om = 1.f - zeta;
  r.Lg = pc.L0 * expf(pc.neg_Qg_over_R / Tc);
  r.dLg = clipped ? 0.f : r.Lg * (-pc.neg_Qg_over_R) / (Tc * Tc);
  r.dz = clipped ? 0.f : dzeta_dT(pc, xz);
  r.liquid = pc.force && T > pc.liquid_limit;
  return r;
}

// ---- kernel A: u, v, the local term and the temperature sensitivity --------
__global__ void __launch_bounds__(256) adj_pf_local_kernel(const __grid_constant__ AdjArgs a) {
  const int ncell = a.nx * a.ny * a.nz;  // host checks < 2^31
  const int n = a.n;
  const AdjLanes ln = adj_lanes(n);
  const int warp_id = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int nwarps = (int)(((long long)gridDim.x * blockDim.x) >> 5);
  const float mg = a.pc.mg_ad, kap = a.pc.kappa_ad, A = a.pc.aniso;
  const int64_t Nn = (int64_t)ncell * n;
  const int xy = a.nx * a.ny;
  const int64_t sy = (int64_t)a.nx * n, sz = (int64_t)xy * n;
  const int64_t gsy = a.nx + 2, gsz = (int64_t)(a.ny + 2) * (a.nx + 2);
  for (int cb = warp_id * ln.cpw; cb < ncell; cb += nwarps * ln.cpw) {
    const int c = cb + ln.cw;
    const bool valid = ln.active && c < ncell;
    const int cc = valid ? c : 0;
    const int z = cc / xy, r = cc - z * xy, y = r / a.nx, x = r - y * a.nx;
    // temperature-only quantities (as in the forward fast kernels)
    const float T = a.Tg[(int64_t)(z + 1) * gsz + (int64_t)(y + 1) * gsy + x + 1];
    const AdjTemp tq = adj_temp(a.pc, T);
    const float om = tq.om, Lg = tq.Lg, dLg = tq.dLg, dz = tq.dz;
    const bool liquid = tq.liquid;
    const int64_t base = (int64_t)z * sz + (int64_t)y * sy + (int64_t)x * n;
    // per-cell sums
    float s = 0.f, ld = 0.f;
    if (valid) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int i = 2 * ln.g + j;
        if (i < n) {
          const float ei = a.eta[base + i], li = a.lam_in[base + i];
          s = fmaf(ei, ei, s);
          ld = fmaf(li, ei, ld);
        }
      }
    }
    s = cell_sum(s, ln);
    ld = cell_sum(ld, ln);
    const float K = 4.f * s + 2.f * om * om - 1.f;
    const int xm = nbr(x, -1, a.nx, a.bcx), xp = nbr(x, 1, a.nx, a.bcx);
    const int ym = nbr(y, -1, a.ny, a.bcy), yp = nbr(y, 1, a.ny, a.bcy);
    const int zm = nbr(z, -1, a.nz, a.bcz), zp = nbr(z, 1, a.nz, a.bcz);
    const int64_t oxm = (int64_t)z * sz + (int64_t)y * sy + (int64_t)xm * n;
    const int64_t oxp = (int64_t)z * sz + (int64_t)y * sy + (int64_t)xp * n;
    const int64_t oym = (int64_t)z * sz + (int64_t)ym * sy + (int64_t)x * n;
    const int64_t oyp = (int64_t)z * sz + (int64_t)yp * sy + (int64_t)x * n;
    const int64_t ozm = (int64_t)zm * sz + (int64_t)y * sy + (int64_t)x * n;
    const int64_t ozp = (int64_t)zp * sz + (int64_t)y * sy + (int64_t)x * n;
    float mu = 0.f;
    if (valid) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int i = 2 * ln.g + j;
        if (i >= n) continue;
        const float e = a.eta[base + i], lam = liquid ? 0.f : a.lam_in[base + i];
        const float vxm = a.eta[oxm + i], vxp = a.eta[oxp + i];
        const float vym = a.eta[oym + i], vyp = a.eta[oyp + i];
        const float vzm = a.eta[ozm + i], vzp = a.eta[ozp + i];
        const float L = a.pc.wx * ((vxp - e) + (vxm - e)) + a.pc.wy * ((vyp - e) + (vym - e)) +
                        a.pc.wz * ((vzp - e) + (vzm - e));
        float an = 1.f, dax = 0.f, day = 0.f, daz = 0.f;
        const float ex = vxp - vxm, ey = vyp - vym, ez = vzp - vzm;
        const float ee = ex * ex + ey * ey + ez * ez;
        float pbest = 0.f, m = -1.f;
        int kbest = 0;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const float* d = &a.dirs[(k * n + i) * 3];
          const float pk = d[0] * ex + d[1] * ey + d[2] * ez;
          if (pk * pk > m) { m = pk * pk; pbest = pk; kbest = k; }
        }
        const float c2 = (ee > 0.f) ? m / ee : 1.f;
        if (c2 < 1.f) {
          const float s2 = 1.f - c2;
          an = 1.f + A * (c2 * c2 + s2 * s2);
          // da/de = A (4 c2 - 2) * 2 (p* d* - c2 e) / ee
          const float f = A * (4.f * c2 - 2.f) * 2.f / ee;
          const float* d = &a.dirs[(kbest * n + i) * 3];
          dax = f * (pbest * d[0] - c2 * ex);
          day = f * (pbest * d[1] - c2 * ey);
          daz = f * (pbest * d[2] - c2 * ez);
        } else {
          an = 1.f + A;
        }
        const float gg = e * (K - 3.f * e * e);
        const float Q = Lg * kap;
        a.u[base + i] = lam * Q * an;
        a.v[base + i] = lam * Q * L * dax;
        a.v[Nn + base + i] = lam * Q * L * day;
        a.v[2 * Nn + base + i] = lam * Q * L * daz;
        a.loc[base + i] = liquid ? 0.f : -Lg * mg * (lam * (K - 9.f * e * e) + 8.f * e * ld);
        mu += lam * (dLg * (-mg * gg + kap * an * L) + Lg * mg * 4.f * om * e * dz);
      }
    }
    mu = cell_sum(mu, ln);
    if (valid && ln.g == 0) {
      a.muPF[c] = a.dt * mu;
      a.mask[c] = liquid ? 0.f : 1.f;
    }
  }
}

// ---- kernel B: the adjoint of the stencil terms, gathered per element --------
__global__ void __launch_bounds__(256) adj_pf_gather_kernel(const __grid_constant__ AdjArgs a) {
  const int ncell = a.nx * a.ny * a.nz;
  const int n = a.n;
  const AdjLanes ln = adj_lanes(n);
  const int warp_id = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int nwarps = (int)(((long long)gridDim.x * blockDim.x) >> 5);
  const int64_t Nn = (int64_t)ncell * n;
  const int xy = a.nx * a.ny;
  const int64_t sy = (int64_t)a.nx * n, sz = (int64_t)xy * n;
  for (int cb = warp_id * ln.cpw; cb < ncell; cb += nwarps * ln.cpw) {
    const int c = cb + ln.cw;
    if (!ln.active || c >= ncell) continue;  // no shuffles below
    const int z = c / xy, r = c - z * xy, y = r / a.nx, x = r - y * a.nx;
    const int64_t base = (int64_t)z * sz + (int64_t)y * sy + (int64_t)x * n;
    // neighbour offsets and the sign of v at each (odd extension at a Neumann face)
    int64_t off[6];
    float sgn[6];
    const int dims[3] = {a.nx, a.ny, a.nz};
    const int bcs[3] = {a.bcx, a.bcy, a.bcz};
    const int pos[3] = {x, y, z};
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      int q[3] = {x, y, z};
      const int ax = k >> 1, step = (k & 1) ? 1 : -1;
      const int raw = pos[ax] + step;
      q[ax] = bc_index(raw, dims[ax], bcs[ax]);
      sgn[k] = (!bcs[ax] && (raw < 0 || raw >= dims[ax])) ? -1.f : 1.f;
      off[k] = (int64_t)q[2] * sz + (int64_t)q[1] * sy + (int64_t)q[0] * n;
    }
    const float m = a.mask[c];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int i = 2 * ln.g + j;
      if (i >= n) continue;
      const float uc = a.u[base + i];
      const float lapu = a.pc.wx * (a.u[off[0] + i] + a.u[off[1] + i] - 2.f * uc) +
                         a.pc.wy * (a.u[off[2] + i] + a.u[off[3] + i] - 2.f * uc) +
                         a.pc.wz * (a.u[off[4] + i] + a.u[off[5] + i] - 2.f * uc);
      const float dvx = sgn[1] * a.v[off[1] + i] - sgn[0] * a.v[off[0] + i];
      const float dvy = sgn[3] * a.v[Nn + off[3] + i] - sgn[2] * a.v[Nn + off[2] + i];
      const float dvz = sgn[5] * a.v[2 * Nn + off[5] + i] - sgn[4] * a.v[2 * Nn + off[4] + i];
      a.lam_out[base + i] =
          m * a.lam_in[base + i] + a.dt * (a.loc[base + i] + lapu - (dvx + dvy + dvz));
    }
  }
}

// ---- the isotropic step of the order parameters --------------------------------
// A block marches a tile of tx x ty cells (12 warps: two along x, six along y;
// a warp holds 32 / tpc cells) through zc planes, with the planes below and at
// the cell in registers; the in-plane neighbours come from L1, where the block
// has just loaded them as the plane ahead.  The sums over a cell's orientations
// and every product that the two-launch form stores are rounded as there.
constexpr int kIsoThreads = 384, kIsoWarpsX = 2, kIsoWarpsY = 6;

// Two consecutive values of a cell (the second absent at the end of an odd n).
template <bool VEC>
__device__ __forceinline__ float2 load_two(const float* p, bool second) {
  if constexpr (VEC) return __ldg(reinterpret_cast<const float2*>(p));
  else return make_float2(__ldg(p), second ? __ldg(p + 1) : 0.f);
}

// VEC: n even and the fields 8-byte aligned.
template <bool VEC>
__global__ void __launch_bounds__(kIsoThreads, 2)
adj_pf_iso_kernel(const __grid_constant__ AdjArgs a) {
  const int n = a.n;
  const AdjLanes ln = adj_lanes(n);
  const int warp = threadIdx.x >> 5;
  const int per_plane = a.tiles_x * a.tiles_y;
  const int chunk = blockIdx.x / per_plane, tile = blockIdx.x - chunk * per_plane;
  const int tyi = tile / a.tiles_x, txi = tile - tyi * a.tiles_x;
  const int xr = txi * a.tx + (warp % kIsoWarpsX) * ln.cpw + ln.cw;
  const int yr = tyi * a.ty + warp / kIsoWarpsX;
  const bool valid = ln.active && xr < a.nx && yr < a.ny;
  const int x = valid ? xr : 0, y = valid ? yr : 0;  // idle lanes shadow cell (0, 0)
  const int zb = chunk * a.zc, ze = min(zb + a.zc, a.nz);
  const int i0 = valid ? 2 * ln.g : 0;
  const bool second = i0 + 1 < n;
  const int xy = a.nx * a.ny;
  const int64_t sz = (int64_t)xy * n;
  const int c0 = y * a.nx + x;
  // in-plane neighbours: cells, and elements from the cell's
  const int cxm = y * a.nx + nbr(x, -1, a.nx, a.bcx), cxp = y * a.nx + nbr(x, 1, a.nx, a.bcx);
  const int cym = nbr(y, -1, a.ny, a.bcy) * a.nx + x, cyp = nbr(y, 1, a.ny, a.bcy) * a.nx + x;
  const float mg = a.pc.mg_ad, kap = a.pc.kappa_ad;
  auto u_of = [](float2 l, float q) { return make_float2(__fmul_rn(l.x, q), __fmul_rn(l.y, q)); };
  const int64_t first = (int64_t)c0 * n + i0;
  const float* eta = a.eta + first;
  const float* lam = a.lam_in + first;
  const int zl = nbr(zb, -1, a.nz, a.bcz);
  float2 em = load_two<VEC>(eta + zl * sz, second), ec = load_two<VEC>(eta + zb * sz, second);
  float2 um = u_of(load_two<VEC>(lam + zl * sz, second), a.q[(int64_t)zl * xy + c0]);
  float2 lc = load_two<VEC>(lam + zb * sz, second);
  float2 uc = u_of(lc, a.q[(int64_t)zb * xy + c0]);
  eta += zb * sz;
  lam += zb * sz;
  // the host keeps a plane below 2^31 elements
  const int nxm = (cxm - c0) * n, nxp = (cxp - c0) * n, nym = (cym - c0) * n, nyp = (cyp - c0) * n;
  int cz = zb * xy + c0;
  for (int z = zb; z < ze; ++z, eta += sz, lam += sz, cz += xy) {
    const bool wraps = z + 1 == a.nz;  // the plane above: the next, this one or the first
    const int64_t up_at = wraps ? (a.bcz ? -(int64_t)(a.nz - 1) * sz : 0) : sz;
    const float2 ep = load_two<VEC>(eta + up_at, second), lp = load_two<VEC>(lam + up_at, second);
    float2 up = u_of(lp, a.q[cz + (wraps ? (a.bcz ? -(a.nz - 1) * xy : 0) : xy)]);
    const float2 exm = load_two<VEC>(eta + nxm, second), exp_ = load_two<VEC>(eta + nxp, second);
    const float2 eym = load_two<VEC>(eta + nym, second), eyp = load_two<VEC>(eta + nyp, second);
    const float* qz = a.q + (cz - c0);
    float2 uxm = u_of(load_two<VEC>(lam + nxm, second), qz[cxm]);
    float2 uxp = u_of(load_two<VEC>(lam + nxp, second), qz[cxp]);
    float2 uym = u_of(load_two<VEC>(lam + nym, second), qz[cym]);
    float2 uyp = u_of(load_two<VEC>(lam + nyp, second), qz[cyp]);
    const float Lgm = a.g[cz], o2 = a.om2[cz], dLg = a.dLg[cz];
    const bool liquid = o2 < 0.f;
    // per-cell sums
    float s = 0.f, ld = 0.f;
    if (valid) {
      s = fmaf(ec.x, ec.x, s);
      ld = fmaf(lc.x, ec.x, ld);
      if (second) {
        s = fmaf(ec.y, ec.y, s);
        ld = fmaf(lc.y, ec.y, ld);
      }
    }
    s = cell_sum(s, ln);
    ld = cell_sum(ld, ln);
    const float K = 4.f * s + o2 - 1.f;
    // d zeta / dT: only at T == T_liquidus exactly (1 - zeta = 1/2)
    float om = 0.f, dz = 0.f;
    if (o2 == 0.5f) {
      const AdjTemp tq = adj_temp(
          a.pc, a.Tg[((int64_t)(z + 1) * (a.ny + 2) + (y + 1)) * (a.nx + 2) + x + 1]);
      om = tq.om;
      dz = tq.dz;
    }
    float mu = 0.f;
    auto element = [&](float e, float vxm, float vxp, float vym, float vyp, float vzm, float vzp,
                       float l, float u, float u0, float u1, float u2, float u3, float u4,
                       float u5) {
      const float lamm = liquid ? 0.f : l;
      const float L = a.pc.wx * ((vxp - e) + (vxm - e)) + a.pc.wy * ((vyp - e) + (vym - e)) +
                      a.pc.wz * ((vzp - e) + (vzm - e));
      const float gg = e * (K - 3.f * e * e);
      const float loc =
          liquid ? 0.f : __fmul_rn(-Lgm, fmaf(8.f * e, ld, __fmul_rn(lamm, K - 9.f * e * e)));
      mu += lamm * (dLg * (-mg * gg + kap * L) + Lgm * 4.f * om * e * dz);
      const float lapu = a.pc.wx * (u0 + u1 - 2.f * u) + a.pc.wy * (u2 + u3 - 2.f * u) +
                         a.pc.wz * (u4 + u5 - 2.f * u);
      return fmaf(liquid ? 0.f : 1.f, l, __fmul_rn(a.dt, loc + lapu));
    };
    float2 out;
    auto both = [&] {
      mu = 0.f;
      out.x = element(ec.x, exm.x, exp_.x, eym.x, eyp.x, em.x, ep.x, lc.x, uc.x, uxm.x, uxp.x,
                      uym.x, uyp.x, um.x, up.x);
      if (second)
        out.y = element(ec.y, exm.y, exp_.y, eym.y, eyp.y, em.y, ep.y, lc.y, uc.y, uxm.y, uxp.y,
                        uym.y, uyp.y, um.y, up.y);
    };
    both();
    // A liquid cell has no u (q = -0) whatever its lam, but 0 times a non-finite
    // lam is NaN: looked at where a result shows it (as a test at every u, 85
    // -> 94 us a step at 1M cells, n = 10).
    if (!isfinite(out.x) || (second && !isfinite(out.y))) {
      auto clear = [&](float2& u, int64_t cell) {
        if (__float_as_uint(a.q[cell]) == 0x80000000u) u = make_float2(0.f, 0.f);
      };
      const int64_t below = (int64_t)nbr(z, -1, a.nz, a.bcz) * xy + c0;
      clear(uc, cz);
      clear(um, below);
      clear(up, (int64_t)nbr(z, 1, a.nz, a.bcz) * xy + c0);
      clear(uxm, cz - c0 + cxm);
      clear(uxp, cz - c0 + cxp);
      clear(uym, cz - c0 + cym);
      clear(uyp, cz - c0 + cyp);
      both();
    }
    if (valid) {
      float* o = a.lam_out + (lam - a.lam_in);
      if constexpr (VEC) {
        *reinterpret_cast<float2*>(o) = out;
      } else {
        o[0] = out.x;
        if (second) o[1] = out.y;
      }
    }
    mu = cell_sum(valid ? mu : 0.f, ln);
    if (valid && ln.g == 0) {  // on top of the heat transpose's part
      const int64_t idx = ((int64_t)(z + 1) * (a.ny + 2) + (y + 1)) * (a.nx + 2) + x + 1;
      a.Tb_out[idx] = a.Tb_out[idx] + __fmul_rn(a.dt, mu);
    }
    em = ec;
    ec = ep;
    um = uc;
    lc = lp;
    uc = up;
  }
}

// ---- kernel C: heat transpose, one thread per interior cell -------------------
// ISO: the isotropic step adds its part of dJ/dT afterwards.  The neighbours'
// diffusivities (two divisions each) come from the launch before.
struct HeatLocal {
  float k, dk, cp, dcp, alpha, dalpha;
};
__device__ __forceinline__ HeatLocal heat_local(const HeatConsts& H, float T) {
  HeatLocal r;
  const bool in = T > 300.f && T < H.Tl;
  const float Tk = fminf(fmaxf(T, 300.f), H.Tl);
  r.k = 0.0163f * Tk + 4.5847f;
  r.dk = in ? 0.0163f : 0.f;
  r.cp = 0.2441f * Tk + 338.39f + (heat_mushy(H, T) ? H.latent : 0.f);
  r.dcp = in ? 0.2441f : 0.f;
  r.alpha = r.k / H.rho / r.cp;
  r.dalpha = (r.dk * r.cp - r.k * r.dcp) / (H.rho * r.cp * r.cp);
  return r;
}

// Per-cell numbers of the step: the diffusivity, and with ISO the cell
// coefficients of the isotropic step.
template <bool ISO>
__global__ void __launch_bounds__(256) adj_cell_kernel(const __grid_constant__ AdjArgs a) {
  const int ncell = a.nx * a.ny * a.nz, xy = a.nx * a.ny;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < ncell; c += gridDim.x * blockDim.x) {
    const int z = c / xy, rem = c - z * xy, y = rem / a.nx, x = rem - y * a.nx;
    const float T = a.Tg[((int64_t)(z + 1) * (a.ny + 2) + (y + 1)) * (a.nx + 2) + x + 1];
    a.alpha[c] = heat_local(a.hc, T).alpha;
    if constexpr (ISO) {
      const AdjTemp tq = adj_temp(a.pc, T);
      a.q[c] = tq.liquid ? -0.f : tq.Lg * a.pc.kappa_ad;
      a.g[c] = tq.Lg * a.pc.mg_ad;
      a.om2[c] = tq.liquid ? -1.f : 2.f * tq.om * tq.om;
      a.dLg[c] = tq.dLg;
    }
  }
}

template <bool ISO>
__global__ void __launch_bounds__(256) adj_heat_kernel(const __grid_constant__ AdjArgs a) {
  const HeatConsts& H = a.hc;
  const int ncell = a.nx * a.ny * a.nz;  // host checks (with room for the stride)
  const int xy = a.nx * a.ny;
  const int64_t sx = 1, sy = a.nx + 2, sz = (int64_t)(a.ny + 2) * (a.nx + 2);
  const float R2 = a.hc.two_over_r2;
  double gP = 0.0, gv = 0.0;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < ncell; c += gridDim.x * blockDim.x) {
    const int z = c / xy, rem = c - z * xy, y = rem / a.nx, x = rem - y * a.nx;
    const int64_t idx = (int64_t)(z + 1) * sz + (int64_t)(y + 1) * sy + x + 1;
    const float Tc = a.Tg[idx];
    const HeatLocal hl = heat_local(H, Tc);
    const float dt = a.dt;
    const float mu_c = a.Tb_in[idx];
    // neighbours: value used in the forward Laplacian and its adjoint route
    const int64_t st[6] = {-sx, sx, -sy, sy, -sz, sz};
    const bool face[6] = {x == 0, x == a.nx - 1, y == 0, y == a.ny - 1, z == 0, z == a.nz - 1};
    const float d[6] = {H.dx, H.dx, H.dy, H.dy, H.dz, H.dz};
    const float r2[6] = {1.f / H.dx2, 1.f / H.dx2, 1.f / H.dy2, 1.f / H.dy2, 1.f / H.dz2, 1.f / H.dz2};
    float Nv[6], dGdT[6], dGdG[6], dGdB[6], B[6];
#pragma unroll
    for (int f = 0; f < 6; ++f) {
      const float Gold = a.Tg[idx + st[f]];
      dGdT[f] = dGdG[f] = dGdB[f] = 0.f;
      B[f] = 0.f;
      if (face[f]) {
        const float Tf = 0.5f * (Tc + Gold);
        const float Rf = heat_robin(H, Tf);
        const float dR = H.h + 4.f * H.sb_eps * Tf * Tf * Tf;
        float beam = 0.f;
        if (f == 5 && a.beam_on) {
          const float px = H.x_first + (float)x * H.dx - a.xl;
          const float py = H.y_first + (float)y * H.dy - a.yl;
          beam = a.P * H.beam_coef * expf(-(px * px + py * py) * R2);
          B[f] = beam;
        }
        const float q = Rf - beam;
        Nv[f] = Tc - q / hl.k * d[f];
        dGdT[f] = 1.f - d[f] * (0.5f * dR / hl.k - q * hl.dk / (hl.k * hl.k));
        dGdG[f] = -d[f] * 0.5f * dR / hl.k;
        dGdB[f] = d[f] / hl.k;
      } else {
        Nv[f] = Gold;  // an interior neighbour (old value)
      }
    }
    const float lap = (Nv[0] - 2.f * Tc + Nv[1]) * r2[0] + (Nv[2] - 2.f * Tc + Nv[3]) * r2[2] +
                      (Nv[4] - 2.f * Tc + Nv[5]) * r2[4];
    float mu = mu_c * (1.f + dt * hl.dalpha * lap -
                       2.f * dt * hl.alpha * (r2[0] + r2[2] + r2[4]));
#pragma unroll
    for (int f = 0; f < 6; ++f) {
      if (face[f]) {
        const float w = mu_c * dt * hl.alpha * r2[f] + a.Tb_in[idx + st[f]];
        mu += w * dGdT[f];
        a.Tb_out[idx + st[f]] = w * dGdG[f];
        if (f == 5 && a.beam_on) {
          // B = P coef exp(...): dB/dP = B / P, dB/dxl = B * 4 (x - xl) / r^2
          const float px = H.x_first + (float)x * H.dx - a.xl;
          gP += (double)(w * dGdB[f]) * (double)(B[f] / a.P);
          gv += (double)(w * dGdB[f]) * (double)(B[f] * 2.f * R2 * px) * (double)a.dxl_dv;
        }
      } else {
        // this cell is the neighbour m's Laplacian input with weight dt alpha_m / d^2
        const int cs[6] = {-1, 1, -a.nx, a.nx, -xy, xy};
        mu += a.Tb_in[idx + st[f]] * dt * a.alpha[c + cs[f]] * r2[f];
      }
    }
    if constexpr (ISO) {
      a.Tb_out[idx] = mu;
    } else {
      a.Tb_out[idx] = mu + a.muPF[c];
    }
  }
  // block reduction of the two gradient components, one atomic per block
  __shared__ double sP[8], sv[8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    gP += __shfl_xor_sync(0xffffffffu, gP, o);
    gv += __shfl_xor_sync(0xffffffffu, gv, o);
  }
  if (lane == 0) { sP[w] = gP; sv[w] = gv; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double tP = 0.0, tv = 0.0;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) { tP += sP[i]; tv += sv[i]; }
    atomicAdd(&a.grads[0], tP);
    atomicAdd(&a.grads[1], tv);
  }
}

// ---- objective J = mean over cells of sum_i w_i eta_i^2 and its seed ----------
// Float64 throughout.  The float64 pipe bounds this kernel (two lanes a clock an
// SM), so an element takes one instruction of it: a thread keeps to one
// orientation (the launch's threads, less a remainder, are a whole number of
// cells) and applies its weight once, and integer instructions widen the values
// (1M cells, n = 10: 28 us a launch; with conversions 46, with a product and a
// weight an element 85).

// |v| as a double, of a finite value: the exponent's bias and place change.  Far
// fields are full of denormals, which are scaled by 2^64 first.
__device__ __forceinline__ double widened_abs(float v) {
  const bool tiny = fabsf(v) < 1e-30f;
  const unsigned m = __float_as_uint(fabsf(tiny ? v * 0x1p64f : v));
  const unsigned bias = m == 0u ? 0u : tiny ? 0x34000000u : 0x38000000u;
  return __hiloint2double((int)((m >> 3) + bias), (int)(m << 29));
}

template <bool SEED>
__global__ void __launch_bounds__(256)
objective_kernel(const float* __restrict__ eta, const float* __restrict__ w, long long ncell, int n,
                 double* __restrict__ J, float* __restrict__ lam) {
  const float inv = 1.f / (float)ncell;
  const long long total = ncell * n;
  const long long stride = (long long)gridDim.x * blockDim.x / n * n;
  const long long first = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  double sum = 0.0;
  if (first < stride && first < total) {
    const float wi = __ldg(w + (int)(first % n));
    bool other = false;  // an infinite or NaN value
#pragma unroll 4
    for (long long e = first; e < total; e += stride) {
      const float v = __ldg(eta + e);
      other |= !isfinite(v);
      const double d = widened_abs(v);
      sum = fma(d, d, sum);
      if (SEED) lam[e] = 2.f * wi * v * inv;
    }
    if (other) {
      sum = 0.0;
      for (long long e = first; e < total; e += stride) {
        const double d = (double)__ldg(eta + e);
        sum = fma(d, d, sum);
      }
    }
    sum *= (double)wi;
  }
  __shared__ double s[8];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += s[k];
    atomicAdd(J, t / (double)ncell);
  }
}

}  // namespace pfg

using namespace pfg;

// Whether [a, a + na) and [b, b + nb) share an element.
static bool overlap(const float* a, int64_t na, const float* b, int64_t nb) {
  return a < b + nb && b < a + na;
}

extern "C" int64_t pfg_adjoint_scratch_bytes(const pfg_pf_params* p) {
  if (check_pf_params(p)) return -1;
  const int64_t N = (int64_t)p->nx * p->ny * p->nz;
  return (5 * N * p->num_oris + 2 * N) * (int64_t)sizeof(float);
}

extern "C" int pfg_adjoint_step(const pfg_pf_params* p, const pfg_heat_params* h,
                                const float* eta, const float* Tg, double t, float dt,
                                const float* lam_in, const float* Tb_in, float* lam_out,
                                float* Tb_out, void* scratch, int64_t scratch_bytes,
                                double* grads, float dxl_dv, void* stream) {
  int st = check_pf_params(p);
  if (st) return st;
  st = check_heat_params(h);
  if (st) return st;
  if (h->nx != p->nx || h->ny != p->ny || h->nz != p->nz) return PFG_ERR_SHAPE;
  if (!eta || !Tg || !lam_in || !Tb_in || !lam_out || !Tb_out || !scratch || !grads)
    return PFG_ERR_NULL;
  if (scratch_bytes < pfg_adjoint_scratch_bytes(p)) return PFG_ERR_CAPACITY;
  // 32-bit cell indices (with room for the grid-stride look-ahead)
  if ((int64_t)p->nx * p->ny * p->nz >= ((int64_t)1 << 31) - ((int64_t)1 << 22))
    return PFG_ERR_SHAPE;
  if (!device_info().ok) return PFG_ERR_NO_DEVICE;
  AdjArgs a{};
  a.nx = p->nx; a.ny = p->ny; a.nz = p->nz; a.n = p->num_oris;
  a.bcx = p->bc_x; a.bcy = p->bc_y; a.bcz = p->bc_z;
  a.dt = dt;
  a.pc = make_pf_consts(*p);
  a.hc = make_heat_consts(*h);
  float xl = 0.f, yl = 0.f, P = 0.f;
  // the beam at the mid-step time, as the forward step places it
  for (int s = 0; s < h->num_segments; ++s) {
    const pfg_segment& g = h->path[s];
    const double tm = t + 0.5 * (double)dt;
    if (tm >= (double)g.t0 && tm < (double)g.t1) {
      const double f = (tm - (double)g.t0) / ((double)g.t1 - (double)g.t0);
      xl = (float)((double)g.x0 + f * ((double)g.x1 - (double)g.x0));
      yl = (float)((double)g.y0 + f * ((double)g.y1 - (double)g.y0));
      P = g.power;
      break;
    }
  }
  a.xl = xl; a.yl = yl; a.P = P; a.beam_on = P != 0.f; a.dxl_dv = dxl_dv;
  a.eta = eta; a.Tg = Tg; a.lam_in = lam_in; a.Tb_in = Tb_in;
  a.lam_out = lam_out; a.Tb_out = Tb_out;
  const int64_t N = (int64_t)p->nx * p->ny * p->nz, Nn = N * p->num_oris;
  float* sc = static_cast<float*>(scratch);
  a.u = sc;
  a.v = sc + Nn;
  a.loc = sc + 4 * Nn;
  a.muPF = sc + 5 * Nn;
  a.mask = sc + 5 * Nn + N;
  a.grads = grads;
  for (int i = 0; i < 3 * p->num_oris * 3; ++i) a.dirs[i] = p->grain_dirs[i];
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const DeviceInfo& d = device_info();
  const int cpw = 32 / ((p->num_oris + 1) / 2);  // cells per warp of the element kernels
  const int cell_blocks = (int)std::min<int64_t>((N + 255) / 256, (int64_t)d.sm_count * 16);
  // The isotropic kernel reads eta and lam_in at neighbours while others write
  // lam_out, and after Tb_out is written.  Kernels A and B read lam_in at the
  // element that they write and have read eta before, and C writes Tb_out last,
  // so outputs there may take the place of eta or lam_in.
  const int64_t Ng = (int64_t)(p->nx + 2) * (p->ny + 2) * (p->nz + 2);
  const bool in_place = overlap(lam_out, Nn, lam_in, Nn) || overlap(lam_out, Nn, eta, Nn) ||
                        overlap(Tb_out, Ng, lam_in, Nn) || overlap(Tb_out, Ng, eta, Nn);
  // its in-plane offsets are 32-bit (a plane of 2^31 elements takes the others)
  if (!(a.pc.aniso > 0.f) && !in_place &&
      (int64_t)p->nx * p->ny * p->num_oris < ((int64_t)1 << 31)) {
    a.q = sc;
    a.g = sc + N;
    a.om2 = sc + 2 * N;
    a.dLg = sc + 3 * N;
    a.alpha = sc + 4 * N;
    a.tx = kIsoWarpsX * cpw;
    a.ty = kIsoWarpsY;
    a.tiles_x = (p->nx + a.tx - 1) / a.tx;
    a.tiles_y = (p->ny + a.ty - 1) / a.ty;
    // planes per unit: fewest plane times over the waves of blocks (two per SM),
    // counting two for the planes beside a unit's
    const int64_t tiles = (int64_t)a.tiles_x * a.tiles_y, slots = 2LL * d.sm_count;
    double least = 1e300;
    for (int zch = 1; zch <= p->nz && zch <= 4096; ++zch) {
      const int zc = (p->nz + zch - 1) / zch;
      const int64_t units = tiles * ((p->nz + zc - 1) / zc);
      const double cost = (double)((units + slots - 1) / slots) * (zc + 2.0);
      if (cost < least - 1e-9) {
        least = cost;
        a.zc = zc;
      }
    }
    const int64_t units = tiles * ((p->nz + a.zc - 1) / a.zc);
    if (units >= ((int64_t)1 << 31)) return PFG_ERR_SHAPE;
    adj_cell_kernel<true><<<cell_blocks, 256, 0, s>>>(a);
    adj_heat_kernel<true><<<cell_blocks, 256, 0, s>>>(a);
    const bool vec = p->num_oris % 2 == 0 &&
                     ((reinterpret_cast<uintptr_t>(eta) | reinterpret_cast<uintptr_t>(lam_in) |
                       reinterpret_cast<uintptr_t>(lam_out)) & 7u) == 0;
    if (vec) adj_pf_iso_kernel<true><<<(unsigned)units, kIsoThreads, 0, s>>>(a);
    else adj_pf_iso_kernel<false><<<(unsigned)units, kIsoThreads, 0, s>>>(a);
    return record_cuda(cudaGetLastError());
  }
  const int warps_blocks =
      (int)std::min<int64_t>((N + 8 * cpw - 1) / (8 * cpw), (int64_t)d.sm_count * 16);
  adj_pf_local_kernel<<<warps_blocks, 256, 0, s>>>(a);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return record_cuda(e);
  adj_pf_gather_kernel<<<warps_blocks, 256, 0, s>>>(a);
  e = cudaGetLastError();
  if (e != cudaSuccess) return record_cuda(e);
  a.alpha = a.u;  // u has been gathered
  adj_cell_kernel<false><<<cell_blocks, 256, 0, s>>>(a);
  adj_heat_kernel<false><<<cell_blocks, 256, 0, s>>>(a);
  return record_cuda(cudaGetLastError());
}

extern "C" int pfg_objective(const pfg_pf_params* p, const float* eta, const float* w, double* J,
                             float* lam_seed, void* stream) {
  int st = check_pf_params(p);
  if (st) return st;
  if (!eta || !w || !J) return PFG_ERR_NULL;
  if (!device_info().ok) return PFG_ERR_NO_DEVICE;
  const long long ncell = (long long)p->nx * p->ny * p->nz;
  const int blocks = (int)std::min<long long>((ncell * p->num_oris + 255) / 256,
                                              (long long)device_info().sm_count * 8);
  const cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (lam_seed) objective_kernel<true><<<blocks, 256, 0, s>>>(eta, w, ncell, p->num_oris, J, lam_seed);
  else objective_kernel<false><<<blocks, 256, 0, s>>>(eta, w, ncell, p->num_oris, J, nullptr);
  return record_cuda(cudaGetLastError());
}
