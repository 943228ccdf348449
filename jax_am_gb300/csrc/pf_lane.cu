// Cell-per-lane TMA stencil step: the fast path for even num_oris from 10 to
// 24, with 16-byte orientation vectors where num_oris % 4 == 0 and 8-byte ones
// otherwise (then nx is even and x Neumann, as in the TMA-fed kernel).  26 and
// up do not leave shared memory for two CTAs an SM.
//
// Each thread owns one cell of a TX x TY tile (TX * TY = the CTA's threads:
// one cell per thread) and marches it through a chunk of z planes.  All per-cell work is
// done by the thread that owns the cell, in registers: the sum S of eta^2,
// zeta and the Arrhenius factor, the folded coefficients and the fused heat
// update.  Nothing per cell goes through shared memory, there are no
// shuffles, and all 32 lanes of a warp update cells.
//  * Staging.  Each halo row of a plane tile is one contiguous run of cells in
//    HBM, copied by one cp.async.bulk (TMA) transfer into a ring of plane
//    slots; the ghosted temperature tile goes through 4-byte cp.async copies
//    arriving on the same mbarrier.  Warp 0 issues the copies of a plane right
//    after the per-plane barrier; there is no producer warp.
//  * z in registers.  A thread keeps its own cell's eta (all orientations)
//    of plane z-1 in registers (read when that plane was the centre), so a
//    plane needs from shared memory the cell and its four x/y neighbours in
//    plane z and the cell above (z+1).  The plane below is never read again
//    once it has been the centre, so its slot is refilled one
//    iteration earlier than a stencil that reads z-1 from shared memory.
//  * The orientation loop is unrolled: the rotated cube axes of each
//    orientation are kernel parameters, read as constant-bank operands.
// Every wait is bounded; a wait that runs out sets the device error flag,
// the CTA waits for its copies in flight (each with the full bound) and
// returns.
//
// Bound: issue slots and chains of dependent instructions at 16 warps an SM (24
// for n = 10 and 12).  Against the TMA-fed kernel, whose lanes share a cell (its per-cell work goes
// through shared memory, and no vector of zeros is skipped), a moving-gradient
// step at 128 x 128 x 64 cells, isotropic: n = 10 49 -> 31 us, 12 62 -> 25,
// 16 49 -> 39, 20 64 -> 43, 24 79 -> 49; anisotropic 51 -> 31, 69 -> 29,
// 51 -> 43, 65 -> 46, 86 -> 52.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "pfg_host.h"
#include "pfg_mbar.cuh"
#include "pfg_step.cuh"

namespace pfg {

__device__ int g_lane_device_error = 0;  // PFG_ERR_TIMEOUT once a bounded wait ran out

__device__ __forceinline__ bool lane_wait(uint64_t* bar, unsigned parity,
                                          long long cycles = kWaitCycles) {
  if (mbar_wait_for(bar, parity, cycles)) return true;
  atomicExch(&g_lane_device_error, PFG_ERR_TIMEOUT);
  return false;
}

// The moving gradient's temperature of plane z at time t
// (solidification/example.py:21-34), in float64 as the reference evaluates it.
__device__ __forceinline__ float quench_T(const StepArgs& a, int z, double t) {
  const double zc = a.q.z_first + (double)z * (double)a.h_z;
  return (float)(a.q.T_base + a.q.grad * (zc - a.q.z0) - a.q.grad * a.q.vel * t);
}

// s + lo^2 + hi^2 of a pair.
__device__ __forceinline__ float add_squares(F2 u, float s) {
  return fmaf(f2_lo(u), f2_lo(u), fmaf(f2_hi(u), f2_hi(u), s));
}

// A vector of VP pairs (16 or 8 bytes).
template <int VP>
__device__ __forceinline__ void load_pairs(F2* v, const float* p) {
  if constexpr (VP == 2) {
    const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(p);
    v[0].b = u.x;
    v[1].b = u.y;
  } else {
    v[0].b = *reinterpret_cast<const unsigned long long*>(p);
  }
}
template <int VP>
__device__ __forceinline__ void store_pairs(float* p, const F2* v) {
  if constexpr (VP == 2)
    *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(v[0].b, v[1].b);
  else
    *reinterpret_cast<unsigned long long*>(p) = v[0].b;
}

// The launch shape of an orientation count.
template <int N>
struct LanePlan {
  static constexpr int VP = N % 4 == 0 ? 2 : 1;  // pairs per vector
  static constexpr int TX = 16, NC = 256;        // 16 x 16 tiles, one cell per thread
  // cells of a staged row: with 8-byte vectors a row is copied from and to an
  // even cell (whole 16 bytes)
  static constexpr int ROWC = VP == 2 ? TX + 2 : TX + 4;
  // The lanes of one shared-memory phase (8 lanes of a 16-byte load, 16 of an
  // 8-byte one) fall on distinct banks: cells along x do by their stride unless
  // N % 8 == 0, where a phase then takes XB cells of each of 8 / XB rows; and
  // the row pitch places the phase's rows beside one another.  (Without, at
  // 1M cells, n = 16: 67 us a step against the TMA-fed kernel's 49.)
  static constexpr int XB = N % 16 == 0 ? 2 : N % 8 == 0 ? 4 : 8;
  static constexpr int row = ROWC * N;
  static constexpr int want = VP == 1 ? 16 : 4;  // the pitch's bank, where it matters
  static constexpr int pitch =
      (VP == 1 || XB < 8) ? row + ((want - row) % 32 + 32) % 32 : row;  // floats
  static constexpr size_t slot = (size_t)(NC / TX + 2) * pitch * 4;
  static constexpr int tslot = ((TX + 2) * (NC / TX + 2) + 3) / 4 * 4;
  // CTAs per SM.  Three take at most 80 registers a thread and a third of
  // shared memory: n = 10 34 -> 31 us a step at 128 x 128 x 64, n = 12 30 -> 25
  // (anisotropic 37 -> 31, 36 -> 29); n = 14 and 16 gain at some sizes and lose
  // 5 to 7 % at others, and 16 spills.
  static constexpr int CTAS = N <= 12 ? 3 : 2;
  // ring slots: four where that many CTAs then fit an SM
  static constexpr int S = 4 * (slot + 2 * tslot * 4) <= (CTAS == 3 ? 76544 : 114304) ? 4 : 3;
};
// COMP: the fused heat state is compensated (T = T + T_lo, double-float
// update).
//
// Ring: plane j (grid plane zb - 1 + j) sits in slot j % S and its copies
// complete phase (j / S) & 1 of that slot's barrier.  Iteration m (z =
// zb + m) reads plane m + 1 (the x/y neighbours) and plane m + 2 (the cell
// above); plane m was last read in iteration m - 1, so right after the
// barrier that opens iteration m its slot takes plane m + S.
template <int N, bool ANISO, int TSRC, bool COMP>
__global__ void __launch_bounds__(LanePlan<N>::NC, LanePlan<N>::CTAS)
pf_lane_kernel(const __grid_constant__ StepArgs a) {
  using LP = LanePlan<N>;
  constexpr int NC = LP::NC, TX = LP::TX, TY = NC / TX, S = LP::S;
  constexpr int VP = LP::VP, V = 2 * VP, NP = N / 2, NV = N / V;
  constexpr bool HALF = VP == 1;  // 8-byte vectors: rows start and end at even cells
  constexpr int TPX = TX + 2, TPY = TY + 2;  // staged tile with its halo
  constexpr int ROWF = LP::pitch;             // floats per staged row
  constexpr int SLOTF = TPY * ROWF;           // floats per eta slot
  constexpr int TSLOT = LP::tslot;
  constexpr bool HEAT = TSRC == kTHeat;
  static_assert(N % 2 == 0 && (S == 3 || S == 4), "pairs; 3 or 4 plane slots");
  static_assert(!COMP || HEAT, "the compensated state is the fused heat state");
  extern __shared__ __align__(128) float smem[];
  float* eta_s = smem;
  float* T_s = eta_s + S * SLOTF;
  float* TL_s = T_s + S * TSLOT;  // low parts of the compensated temperature

  // ---- work unit: (tile, z chunk), z chunk slowest
  const int per_plane = a.tiles_x * a.tiles_y;
  const int zi = blockIdx.x / per_plane;
  const int rem = blockIdx.x - zi * per_plane;
  const int byi = rem / a.tiles_x;
  const int bxi = rem - byi * a.tiles_x;
  const int x0 = bxi * TX, y0 = byi * TY;
  const int xe = min(x0 + TX, a.nx), ye = min(y0 + TY, a.ny);
  const int zb = zi * a.zc, ze = min(zb + a.zc, a.nz);
  const int txv = xe - x0, tyv = ye - y0;
  const bool tile_inner = x0 > 0 && xe < a.nx && y0 > 0 && ye < a.ny;
  const int nplanes = ze - zb + 2;  // planes zb-1 .. ze
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  __shared__ uint64_t full[S];  // the ring's barriers
  __shared__ int s_abort;
  __shared__ double s_t0;
  __shared__ long long s_step;
  __shared__ float s_beam[5];  // xl, yl, P and the low parts of xl, yl
  // moving gradient: the temperature of plane z, evaluated by one thread a
  // plane ahead (float64 arithmetic is slow on this GPU), double-buffered
  __shared__ float s_Tq[2];
  __shared__ uint64_t s_never;  // a barrier nothing arrives on (the wait probe)
  if (threadIdx.x == 0) {
    s_abort = 0;
    // expect-tx arrival of warp 0's lane 0 (+ one cp.async arrival per thread)
    for (int s = 0; s < S; ++s) mbar_init(&full[s], 1 + (HEAT ? NC : 0));
    mbar_init(&s_never, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    double t = 0.0;
    if constexpr (TSRC != kTArray) {
      t = start_time(a);
      if (blockIdx.x == 0) end_step(a, t);
    }
    s_t0 = t;
    if constexpr (TSRC == kTQuench) s_Tq[0] = quench_T(a, zb, t);
    s_step = (TSRC != kTArray) ? start_step(a) : 0;
    if constexpr (HEAT) {
      // beam centre and power at mid-step; the centre also as double-float
      double xd, yd;
      laser_at_d(a.hp, t + 0.5 * (double)a.dt, &xd, &yd, &s_beam[2]);
      s_beam[0] = (float)xd;
      s_beam[1] = (float)yd;
      s_beam[3] = (float)(xd - (double)s_beam[0]);
      s_beam[4] = (float)(yd - (double)s_beam[1]);
    }
  }
  __syncthreads();
  const double t0 = s_t0;
  pfg_point_source prec{};
  if constexpr (TSRC == kTPoint) prec = point_record(a.ps, s_step);
  float w_past = 0.f;
  if constexpr (TSRC == kTInterp) w_past = interp_weight(a.t_future, a.dt_coarse, t0 + (double)a.dt);

  // ---- staging of plane j into slot j % S: eta rows by warp 0 (TMA), the
  // ghosted temperature tile by every thread (cp.async)
  // (8-byte vectors: x0, xe and nx are even and x is Neumann (the planner))
  const int cx0 = HALF ? max(x0 - 2, 0) : max(x0 - 1, 0);
  const int cx1 = HALF ? (xe < a.nx ? xe + 2 : a.nx) : min(xe + 1, a.nx);
  const int dst_cell0 = HALF ? 0 : cx0 - (x0 - 1);
  const int pos0 = HALF ? x0 - cx0 : 1;  // staged position of cell x0
  const bool wrap_left = (x0 == 0) && a.bcx == PFG_BC_PERIODIC;
  const bool wrap_right = (xe == a.nx) && a.bcx == PFG_BC_PERIODIC;
  const int rows = tyv + 2;
  const unsigned row_bytes = (unsigned)((cx1 - cx0) * N * 4);
  const unsigned cell_bytes = (unsigned)(N * 4);
  const unsigned plane_bytes =
      (unsigned)rows * (row_bytes + (wrap_left ? cell_bytes : 0u) + (wrap_right ? cell_bytes : 0u));
  const int gsy = a.nx + 2, gsz = (a.ny + 2) * (a.nx + 2);  // ghosted strides (host checks < 2^31)
  // this thread's ghosted temperature cells of a staged plane (at most two):
  // offsets from the tile's first ghosted cell and in the slot, or -1
  int t_src[2], t_dst[2];
  if constexpr (HEAT) {
    const int tcols = txv + 2;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int i = threadIdx.x + q * NC;
      const int r = i / tcols, c = i - r * tcols;
      t_src[q] = r < rows ? r * gsy + c : -1;
      t_dst[q] = r * TPX + c;
    }
  }
  auto stage = [&](int j) {
    const int s = j % S;
    const int pz = zb - 1 + j;
    if (warp == 0) {
      const int gz = bc_index(pz, a.nz, a.bcz);
      float* es = eta_s + s * SLOTF;
      if (lane == 0) mbar_arrive_expect_tx(&full[s], plane_bytes);
      __syncwarp();
      if (lane < rows) {
        const int gy = bc_index(y0 - 1 + lane, a.ny, a.bcy);
        const float* src_row = a.eta_in + ((int64_t)gz * a.ny + gy) * a.nx * N;
        float* dst_row = es + lane * ROWF;
        tma_row(dst_row + dst_cell0 * N, src_row + (int64_t)cx0 * N, row_bytes, &full[s]);
        if (wrap_left) tma_row(dst_row, src_row + (int64_t)(a.nx - 1) * N, cell_bytes, &full[s]);
        if (wrap_right) tma_row(dst_row + (txv + 1) * N, src_row, cell_bytes, &full[s]);
      }
    }
    if constexpr (HEAT) {
      float* ts = T_s + s * TSLOT;
      const float* tplane = a.T + (int64_t)(pz + 1) * gsz + (int64_t)y0 * gsy + x0;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        if (t_src[q] >= 0) {
          cp_async<4>(ts + t_dst[q], tplane + t_src[q]);
          if constexpr (COMP)
            cp_async<4>(TL_s + s * TSLOT + t_dst[q], a.T_lo + (tplane - a.T) + t_src[q]);
        }
      }
      cp_async_mbar_arrive_noinc(&full[s]);
    }
  };

  // ---- this thread's cell
  // a warp owns an 8 x 4 block of cells (rows of 8 lanes): its cells and
  // their neighbours span fewer grains than a 16 x 2 strip, so more of its
  // orientation vectors are exact zeros (1.4 % faster than 16 x 2); a row of
  // 8 lanes at an 80-byte stride reads shared memory without bank conflicts
  constexpr int XB = LP::XB;
  const int lx = lane % XB + XB * ((lane >> 3) % (8 / XB));
  const int ly = (lane % 8) / XB + (8 / XB) * (lane / (64 / XB));
  const int tr = (warp / (TX / 8)) * 4 + ly;
  const int tc = (warp % (TX / 8)) * 8 + lx;
  const bool valid = tr < tyv && tc < txv;
  const bool warp_on = ((threadIdx.x >> 5) / (TX / 8)) * 4 < tyv;  // some row of this warp is in the tile
  const int gx = x0 + tc, gy = y0 + tr;
  const int own = (tr + 1) * ROWF + (tc + pos0) * N;  // staged offset of the cell
  // Neumann along x: the edge cell is its own neighbour (its halo is not staged)
  const int oxm = (gx == 0 && a.bcx == PFG_BC_NEUMANN) ? 0 : -N;
  const int oxp = (gx == a.nx - 1 && a.bcx == PFG_BC_NEUMANN) ? 0 : N;
  const int town = (tr + 1) * TPX + tc + 1;  // staged temperature offset
  const int g_own = (gy + 1) * gsy + gx + 1;  // ghosted index within a plane
  const int64_t cell0 = (int64_t)gy * a.nx + gx;  // cell index within a plane
  const int64_t plane_cells = (int64_t)a.ny * a.nx;

  const LapPair L = lap_pair(a.pc);
  float xl = 0.f, yl = 0.f, Pw = 0.f;
  DF xld{0.f, 0.f}, yld{0.f, 0.f};
  if constexpr (HEAT) {
    xl = s_beam[0];
    yl = s_beam[1];
    Pw = s_beam[2];
    if constexpr (COMP) {
      xld = DF{s_beam[0], s_beam[3]};
      yld = DF{s_beam[1], s_beam[4]};
    }
  }

  // ---- prologue: planes 0 .. S-1 in flight; planes 0, 1, 2 waited for
  int issued = 0;
  for (int j = 0; j < S && j < nplanes; ++j) {
    stage(j);
    issued = j + 1;
  }
  bool ok = true;
  // wait probe: a wait on a barrier that never completes runs out after
  // probe_wait cycles and takes the timeout path
  if (a.probe_wait > 0) ok = lane_wait(&s_never, 0u, a.probe_wait);
  for (int j = 0; j < 3 && ok; ++j) ok = lane_wait(&full[j], 0u);
  if (!ok) s_abort = 1;

  // The cell's eta and temperature of plane z-1 are carried in registers
  // (that plane's slot is refilled while plane z is computed); plane z's come
  // from its slot.  (Unrolling the z loop to rotate register sets instead of
  // copying them makes the loop body overflow the instruction cache.)
  F2 zm[NP], cc[NP];
  float Tzm = 0.f, Tc = 0.f;
  float Lzm = 0.f, Lc = 0.f;  // their low parts (COMP)
  if (ok) {
#pragma unroll
    for (int v = 0; v < NV; ++v) load_pairs<VP>(zm + v * VP, eta_s + 0 * SLOTF + own + v * V);
    if constexpr (HEAT) Tzm = T_s[0 * TSLOT + town];
    if constexpr (COMP) Lzm = TL_s[0 * TSLOT + town];
  }
  // per-cell temperature array: the value of the next plane is loaded one
  // plane ahead
  float Tnext = 0.f;
  if constexpr (TSRC == kTArray) {
    if (valid) Tnext = __ldg(a.T + (int64_t)zb * plane_cells + cell0);
  }
  float* out = a.eta_out + ((int64_t)zb * plane_cells + cell0) * N;

  for (int z = zb; z < ze; ++z) {
    const int m = z - zb;
    const int s1 = (m + 1) % S, s2 = (m + 2) % S;  // slots of planes z and z + 1
    if (m > 0 && ok) ok = lane_wait(&full[s2], (unsigned)(((m + 2) / S) & 1));
    if (!ok) *(volatile int*)&s_abort = 1;
    __syncthreads();  // everyone finished plane z - 1; the slot of plane m is free
    if (*(volatile int*)&s_abort) break;  // uniform across the CTA
    if (m + S < nplanes) {
      stage(m + S);
      issued = m + S + 1;
    }
    // read in the next iteration, after its barrier
    if constexpr (TSRC == kTQuench)
      if (threadIdx.x == 0 && z + 1 < ze) s_Tq[(m + 1) & 1] = quench_T(a, z + 1, t0);
    const float* e1 = eta_s + s1 * SLOTF;
    const float* e2 = eta_s + s2 * SLOTF;
#pragma unroll
    for (int v = 0; v < NV; ++v) load_pairs<VP>(cc + v * VP, e1 + own + v * V);
    float Tzp = 0.f, Lzp = 0.f;
    if constexpr (HEAT) {
      Tc = T_s[s1 * TSLOT + town];
      Tzp = T_s[s2 * TSLOT + town];
    }
    if constexpr (COMP) {
      Lc = TL_s[s1 * TSLOT + town];
      Lzp = TL_s[s2 * TSLOT + town];
    }
    if (warp_on) {
      // ---- temperature at the start of the step, and the heat update
      float Tcell;
      if constexpr (HEAT) {
        const float* t1 = T_s + s1 * TSLOT;
        const float Txm = t1[town - 1], Txp = t1[town + 1];
        const float Tym = t1[town - TPX], Typ = t1[town + TPX];
        const int idx = (z + 1) * gsz + g_own;
        const bool face_plane = !(tile_inner && z > 0 && z < a.nz - 1);  // CTA-uniform
        if constexpr (COMP) {
          const float* l1 = TL_s + s1 * TSLOT;
          const DF c{Tc, Lc};
          DF n[6] = {DF{Txm, l1[town - 1]},   DF{Txp, l1[town + 1]}, DF{Tym, l1[town - TPX]},
                     DF{Typ, l1[town + TPX]}, DF{Tzm, Lzm},         DF{Tzp, Lzp}};
          const bool on_face = face_plane && (gx == 0 || gx == a.nx - 1 || gy == 0 ||
                                              gy == a.ny - 1 || z == 0 || z == a.nz - 1);
          const float tmax = fmaxf(fmaxf(fmaxf(Tc, Txm), fmaxf(Txp, Tym)),
                                   fmaxf(fmaxf(Typ, Tzm), Tzp));
          DF Tn = c;
          // warp-uniform choice: DF arithmetic where the temperature is far
          // from ambient or the beam heats the top face
          if (__any_sync(0xffffffffu, valid && (tmax > a.hd.hot || z == a.nz - 1))) {
            if (!__any_sync(0xffffffffu, on_face && valid))
              Tn = heat_core_df(a.hc, a.hd, c, n);
            else if (valid)
              Tn = heat_update_df_accurate(a.hc, a.hd, c, n, gx, gy, z, xld, yld, Pw, a.T_out,
                                           a.T_lo_out, idx, 1, gsy, gsz);
          } else if (__any_sync(0xffffffffu, on_face && valid)) {
            if (valid)
              Tn = heat_update_df_near_ambient<true>(a.hc, c, n, gx, gy, z, xl, yl, Pw, a.dt,
                                                     a.T_out, a.T_lo_out, idx, 1, gsy, gsz);
          } else {
            Tn = heat_update_df_near_ambient<false>(a.hc, c, n, gx, gy, z, xl, yl, Pw, a.dt,
                                                    a.T_out, a.T_lo_out, idx, 1, gsy, gsz);
          }
          if (valid) {
            a.T_out[idx] = Tn.h;
            a.T_lo_out[idx] = Tn.l;
          }
        } else {
          float Tn;
          if (!face_plane)
            Tn = heat_cell_update<int, false>(a.hc, Tc, Txm, Txp, Tym, Typ, Tzm, Tzp, gx, gy, z,
                                              xl, yl, Pw, a.dt, a.T_out, idx, 1, gsy, gsz);
          else if (valid)
            Tn = heat_cell_update<int, true>(a.hc, Tc, Txm, Txp, Tym, Typ, Tzm, Tzp, gx, gy, z, xl,
                                             yl, Pw, a.dt, a.T_out, idx, 1, gsy, gsz);
          else
            Tn = 0.f;
          if (valid) a.T_out[idx] = Tn;
        }
        Tcell = Tc;
      } else if constexpr (TSRC == kTArray) {
        Tcell = Tnext;
        if (valid && z + 1 < ze) Tnext = __ldg(a.T + (int64_t)(z + 1) * plane_cells + cell0);
      } else if constexpr (TSRC == kTQuench) {
        Tcell = s_Tq[m & 1];
      } else if constexpr (TSRC == kTPoint) {
        Tcell = point_source_T(a.ps, prec, gx, gy, z);
      } else {  // kTInterp
        const int64_t ti = (int64_t)z * plane_cells + cell0;
        const float Tp = valid ? __ldg(a.T + ti) : 0.f, Tf = valid ? __ldg(a.T2 + ti) : 0.f;
        Tcell = w_past * Tp + (1.f - w_past) * Tf;
      }
      // ---- per-cell coefficients
      float s_a = 0.f, s_b = 0.f;
      if constexpr (N % 4 == 0 && N != 20) {  // the TMA-fed kernel's order
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          float& s = (v & 1) ? s_b : s_a;
          s = add_squares(cc[2 * v], add_squares(cc[2 * v + 1], s));
        }
      } else {
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          float& s = (p & 1) ? s_b : s_a;
          s = add_squares(cc[p], s);
        }
      }
      TempCoef tcf;
      if constexpr (COMP) tcf = temp_coefficients_pair(a.pc, Tcell, Lc, a.dt);
      else tcf = temp_coefficients_fast(a.pc, Tcell, a.dt);
      const float4 k = pair_fold(a.pc, tcf, s_a + s_b);
      // the skip below needs finite coefficients in every cell of the warp
      const bool kfinite = __all_sync(0xffffffffu, !valid || (isfinite(k.x) && isfinite(k.y) &&
                                                               isfinite(k.z) && isfinite(k.w)));
      const CoefPair kk = coef_pair(k);
      // ---- element updates, one vector of orientations at a time
      const float* p1 = e1 + own;
      const float* p2 = e2 + own;
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        F2 xm[VP], xp[VP], ym[VP], yp[VP], zp[VP], r[VP];
        load_pairs<VP>(xm, p1 + oxm + V * v);
        load_pairs<VP>(xp, p1 + oxp + V * v);
        load_pairs<VP>(ym, p1 - ROWF + V * v);
        load_pairs<VP>(yp, p1 + ROWF + V * v);
        load_pairs<VP>(zp, p2 + V * v);
        // Exact zeros: an orientation that is zero (+0.0) at every cell of
        // the warp and at all their six neighbours stays exactly zero
        // (gradient, Laplacian and local term vanish, and the update of +0.0
        // is +0.0 with finite coefficients), so the warp skips its
        // arithmetic.  Grain interiors and the far side of an interface are
        // such zeros.  The test is per pair of orientations (0.8 % faster
        // than per vector of four): the cells' own values (in registers)
        // first, the neighbours only when those are zero across the warp.
#pragma unroll
        for (int h = 0; h < VP; ++h) {
          const int p = v * VP + h;  // orientations 2p, 2p + 1
          bool work = !kfinite || __any_sync(0xffffffffu, (cc[p].b | zm[p].b) != 0ull);
          if (!work)
            work = __any_sync(0xffffffffu,
                              (xm[h].b | xp[h].b | ym[h].b | yp[h].b | zp[h].b) != 0ull);
          r[h] = F2{};
          if (work) {
            // the axes of the pair: the projections stay single, with their
            // constant operands from the parameters
            const float* d = a.dirs + 2 * p * 3;
            r[h] = elem_pair<ANISO>(
                L, cc[p], xm[h], xp[h], ym[h], yp[h], zm[p], zp[h], kk,
                [&](int j, F2 gx, F2 gy, F2 gz) {
                  const float* q = d + j * N * 3;
                  return f2_pack(fmaf(q[0], f2_lo(gx), fmaf(q[1], f2_lo(gy), q[2] * f2_lo(gz))),
                                 fmaf(q[3], f2_hi(gx), fmaf(q[4], f2_hi(gy), q[5] * f2_hi(gz))));
                });
          }
        }
        if (valid) store_pairs<VP>(out + V * v, r);
      }
    }
    out += plane_cells * N;
    // plane z is the next plane's z - 1
#pragma unroll
    for (int p = 0; p < NP; ++p) zm[p] = cc[p];
    Tzm = Tc;
    Lzm = Lc;
  }
  // drain: copies still in flight must land before the CTA's shared memory is
  // released (in a normal run every issued plane has been waited for
  // already); after a timeout every slot still gets its full bound
  if constexpr (HEAT) cp_async_wait(0);
  if (threadIdx.x == 0) {
    for (int j = max(0, issued - S); j < issued; ++j)
      lane_wait(&full[j % S], (unsigned)((j / S) & 1));
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

// Calls f(std::integral_constant<int, n>) for the orientation counts that have a
// kernel; false for the others.
template <class F>
static bool with_count(int n, F&& f) {
  switch (n) {
    case 10: f(std::integral_constant<int, 10>()); return true;
    case 12: f(std::integral_constant<int, 12>()); return true;
    case 14: f(std::integral_constant<int, 14>()); return true;
    case 16: f(std::integral_constant<int, 16>()); return true;
    case 18: f(std::integral_constant<int, 18>()); return true;
    case 20: f(std::integral_constant<int, 20>()); return true;
    case 22: f(std::integral_constant<int, 22>()); return true;
    case 24: f(std::integral_constant<int, 24>()); return true;
    default: return false;
  }
}

// Cells from which the counts other than 20 take this kernel: at 6,000 cells
// it and the TMA-fed kernel are level (isotropic 5.3 to 6.3 us a step against
// 5.2 to 7.8, anisotropic 5.3 to 6.2 against 5.7 to 9.7, by count), at 32,768
// it takes 5.6 to 6.5 us against 9.8 to 21, at 1M 30 to 86 against 49 to 91.
constexpr int64_t kLaneMinCells = 1 << 13;

// With a compensated heat state (comp) only 20 orientations do: the split step
// (heat kernel, then the TMA-fed kernel) is level with it for the others
// (20 steps of 200 x 100 x 50 cells: n = 12 1551 us here and 1466 split, n = 24
// 2031 and 1908, n = 10 1529 and 1565).
bool plan_lane_tiles(int nx, int ny, int nz, int n, int bcx, bool comp, int sm_count, int max_smem_per_sm,
                     int max_smem_per_block, int zchunks_override, TilePlan* out) {
  // ghosted temperature offsets are 32-bit in this kernel
  if ((int64_t)(nx + 2) * (ny + 2) * (nz + 2) >= ((int64_t)1 << 31)) return false;
  if (n != 20 && comp) return false;
  if (n != 20 && (int64_t)nx * ny * nz < kLaneMinCells) return false;
  TilePlan t{};
  int ctas = 2;
  if (!with_count(n, [&](auto c) {
        using LP = LanePlan<decltype(c)::value>;
        t.vec = 2 * LP::VP;
        t.tx = LP::TX;
        t.ty = LP::NC / LP::TX;
        t.rs = LP::NC;
        t.stages = LP::S;
        t.pitch = LP::pitch;
        t.tslot = LP::tslot;
        t.smem = LP::S * (LP::slot + 2 * LP::tslot * sizeof(float));
        ctas = LP::CTAS;
      }))
    return false;
  if (t.vec == 2 && (nx % 2 != 0 || bcx != PFG_BC_NEUMANN)) return false;
  // the CTAs of an SM: the dynamic shared memory plus the static variables and
  // the per-CTA reservation
  if (ctas * (t.smem + 1024 + 256) > (size_t)max_smem_per_sm || t.smem > (size_t)max_smem_per_block)
    return false;
  t.tpc = 1;
  t.cpw = 8;        // a warp owns 8 x 4 cells
  t.wx = t.tx / 8;
  t.rpw = 4;
  t.tiles_x = (nx + t.tx - 1) / t.tx;
  t.tiles_y = (ny + t.ty - 1) / t.ty;
  const long tiles = (long)t.tiles_x * t.tiles_y;
  int best_zc = plan_planes(tiles, nz, sm_count * ctas / 2);
  if (zchunks_override > 0) best_zc = (nz + std::min(zchunks_override, nz) - 1) /
                                      std::min(zchunks_override, nz);
  t.zc = best_zc;
  t.zchunks = (nz + t.zc - 1) / t.zc;
  t.units = tiles * t.zchunks;
  if (t.units >= (1L << 31)) return false;
  *out = t;
  return true;
}

template <int N, bool ANISO, int TSRC, bool COMP>
static cudaError_t launch_lane_t(const StepArgs& a, const TilePlan& t, cudaStream_t s) {
  using LP = LanePlan<N>;
  auto k = pf_lane_kernel<N, ANISO, TSRC, COMP>;
  // the temperature planes are staged with the fused heat state only
  const int smem = (int)(TSRC == kTHeat ? t.smem : LP::S * LP::slot);
  static int configured[64] = {0};
  const int dev = device_info().device;
  if (dev < 0 || dev >= 64 || configured[dev] < smem) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) configured[dev] = smem;
  }
  k<<<(unsigned)t.units, LP::NC, smem, s>>>(a);
  return cudaGetLastError();
}

template <int TSRC>
cudaError_t launch_lane_kernel(const StepArgs& a, const TilePlan& t, cudaStream_t s) {
  cudaError_t e = cudaErrorInvalidValue;
  with_count(a.n, [&](auto c) {
    constexpr int N = decltype(c)::value;
    if (t.tx != LanePlan<N>::TX || t.stages != LanePlan<N>::S) return;
    const bool an = a.pc.aniso > 0.f;
    if constexpr (TSRC == kTHeat) {
      if (a.T_lo) {
        if constexpr (N == 20)
          e = an ? launch_lane_t<N, true, TSRC, true>(a, t, s)
                 : launch_lane_t<N, false, TSRC, true>(a, t, s);
        return;
      }
    }
    e = an ? launch_lane_t<N, true, TSRC, false>(a, t, s)
           : launch_lane_t<N, false, TSRC, false>(a, t, s);
  });
  return e;
}

template cudaError_t launch_lane_kernel<kTArray>(const StepArgs&, const TilePlan&, cudaStream_t);
template cudaError_t launch_lane_kernel<kTHeat>(const StepArgs&, const TilePlan&, cudaStream_t);
template cudaError_t launch_lane_kernel<kTQuench>(const StepArgs&, const TilePlan&, cudaStream_t);
template cudaError_t launch_lane_kernel<kTPoint>(const StepArgs&, const TilePlan&, cudaStream_t);
template cudaError_t launch_lane_kernel<kTInterp>(const StepArgs&, const TilePlan&, cudaStream_t);

int read_lane_device_error(int clear) {
  int v = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, g_lane_device_error, sizeof(int));
  if (e != cudaSuccess) return record_cuda(e);
  if (clear && v) {
    const int zero = 0;
    e = cudaMemcpyToSymbol(g_lane_device_error, &zero, sizeof(int));
    if (e != cudaSuccess) return record_cuda(e);
  }
  return v;
}

}  // namespace pfg
