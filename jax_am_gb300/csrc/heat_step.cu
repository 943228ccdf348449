// Explicit finite-difference heat step on the ghosted field (jax_am/cfd/gamma.py:55-61).
// A thread owns one (fast, middle) position and marches kHeatChunk cells along
// the slowest axis, keeping the previous, current and next values of that axis
// in registers: per cell it loads the next value and the four in-plane
// neighbours (a neighbour across a face is the previous ghost value).  The
// field may be in either axis order; consecutive threads take consecutive
// cells of the unit-stride axis, so loads stay coalesced.  A warp whose whole
// chunk touches no domain face runs the update with the face code compiled
// out and steps pointers instead of recomputing indices.
//
// Bound: issue and load latency (128 M warp instructions, 77 % issue active, at
// 64M cells: 138 us).  Tried and slower: the column's values loaded first (153
// us), tiles of w x r columns for L1 reuse (148 - 158 us), the face fluxes in
// a launch of their own (138 + 28 us), and slabs of 8 rows fed by bulk copies
// several planes ahead (150 - 160 us: 122 M instructions at 70 %).
#include <cuda_runtime.h>

#include <type_traits>

#include "pfg_device.cuh"
#include "pfg_host.h"

namespace pfg {

constexpr int kHeatChunk = 8;  // cells marched per thread along the slowest axis

// The edge and corner ghosts carried over from one field to the other: element i
// of the list, `stride` apart.
__device__ __forceinline__ void copy_edges(int nf, int nm, int ns, const float* in, float* out,
                                           int i, int stride) {
  const int sm = nf + 2, ss = (nm + 2) * (nf + 2);
  const int nl = 4 * (nf + 2), ml = 4 * nm, sl = 4 * ns;
  for (; i < nl + ml + sl; i += stride) {
    int at;  // four lines along the fast axis with their corners, then along the others
    if (i < nl) {
      const int l = i / (nf + 2);
      at = i - l * (nf + 2) + (l & 1) * (nm + 1) * sm + (l >> 1) * (ns + 1) * ss;
    } else if (i < nl + ml) {
      const int j = i - nl, l = j / nm;
      at = (j - l * nm + 1) * sm + (l & 1) * (nf + 1) + (l >> 1) * (ns + 1) * ss;
    } else {
      const int j = i - nl - ml, l = j / ns;
      at = (j - l * ns + 1) * ss + (l & 1) * (nf + 1) + (l >> 1) * (nm + 1) * sm;
    }
    out[at] = in[at];
  }
}

// EDGES: the blocks behind the last chunk carry the edge and corner ghosts over.
template <bool XYZ, bool EDGES>
__global__ void __launch_bounds__(256, 8)
heat_step_kernel(const __grid_constant__ HeatConsts H, const float* __restrict__ Tg_in,
                 float* __restrict__ Tg_out, float xl, float yl, float P, float dt) {
  // fast / middle / slow axis extents (XYZ: z, y, x; ZYX: x, y, z)
  const int nf = XYZ ? H.nz : H.nx, nm = H.ny, ns = XYZ ? H.nx : H.nz;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;  // host keeps nf * nm < 2^31
  if (EDGES && blockIdx.y == gridDim.y - 1) {
    copy_edges(nf, nm, ns, Tg_in, Tg_out, t, gridDim.x * blockDim.x);
    return;
  }
  const bool valid = t < nf * nm;
  const int m = t / nf, f = t - m * nf;
  const int s0 = blockIdx.y * kHeatChunk;
  // The face-free update runs when no cell of the whole warp's chunk touches a
  // domain face; the vote keeps that branch warp-uniform (every lane of the
  // 256-thread block is present at the vote).
  const bool interior =
      __all_sync(0xffffffffu, !valid || (f > 0 && f < nf - 1 && m > 0 && m < nm - 1)) &&
      s0 > 0 && s0 + kHeatChunk < ns;
  if (!valid) return;
  // ghosted strides: unit along the fast axis (host keeps the ghosted size < 2^31)
  const int sm = nf + 2, ss = (nm + 2) * (nf + 2);
  int idx = (s0 + 1) * ss + (m + 1) * sm + (f + 1);
  float prev = __ldg(Tg_in + idx - ss), cur = __ldg(Tg_in + idx);
  auto cell = [&](int s, auto faces) {
    constexpr bool F = decltype(faces)::value;
    const float next = __ldg(Tg_in + idx + ss);
    const float fm = __ldg(Tg_in + idx - 1), fp = __ldg(Tg_in + idx + 1);
    const float mm = __ldg(Tg_in + idx - sm), mp = __ldg(Tg_in + idx + sm);
    const int gx = XYZ ? s : f, gy = m, gz = XYZ ? f : s;
    const int sx = XYZ ? ss : 1, sz = XYZ ? 1 : ss;
    const float Tn = XYZ ? heat_cell_update<int, F>(H, cur, prev, next, mm, mp, fm, fp, gx, gy,
                                                    gz, xl, yl, P, dt, Tg_out, idx, sx, sm, sz)
                         : heat_cell_update<int, F>(H, cur, fm, fp, mm, mp, prev, next, gx, gy,
                                                    gz, xl, yl, P, dt, Tg_out, idx, sx, sm, sz);
    Tg_out[idx] = Tn;
    prev = cur;
    cur = next;
    idx += ss;
  };
  if (interior) {  // 5 loads, no face tests; pointer steps instead of index arithmetic
    const float* p = Tg_in + idx;
    float* q = Tg_out + idx;
#pragma unroll
    for (int k = 0; k < kHeatChunk; ++k) {
      const float next = __ldg(p + ss);
      const float fm = __ldg(p - 1), fp = __ldg(p + 1);
      const float mm = __ldg(p - sm), mp = __ldg(p + sm);
      const float Tn =
          XYZ ? heat_cell_update<int, false>(H, cur, prev, next, mm, mp, fm, fp, 0, 0, 0, xl, yl,
                                             P, dt, Tg_out, 0, 0, 0, 0)
              : heat_cell_update<int, false>(H, cur, fm, fp, mm, mp, prev, next, 0, 0, 0, xl, yl,
                                             P, dt, Tg_out, 0, 0, 0, 0);
      *q = Tn;
      prev = cur;
      cur = next;
      p += ss;
      q += ss;
    }
  } else if (s0 + kHeatChunk <= ns) {  // a whole chunk: unrolled, loads issued ahead
#pragma unroll
    for (int k = 0; k < kHeatChunk; ++k) cell(s0 + k, std::true_type{});
  } else {
    for (int s = s0; s < ns; ++s) cell(s, std::true_type{});
  }
}

template <bool XYZ, bool EDGES>
static cudaError_t launch_heat(const HeatConsts& H, const float* in, float* out, float xl,
                               float yl, float power, float dt, cudaStream_t s) {
  const int nf = XYZ ? H.nz : H.nx, ns = XYZ ? H.nx : H.nz;
  const dim3 grid((unsigned)((nf * H.ny + 255) / 256),
                  (unsigned)((ns + kHeatChunk - 1) / kHeatChunk) + (EDGES ? 1u : 0u), 1);
  heat_step_kernel<XYZ, EDGES><<<grid, 256, 0, s>>>(H, in, out, xl, yl, power, dt);
  return cudaGetLastError();
}

static int heat_step(const pfg_heat_params* h, const float* Tg_in, float* Tg_out, float xl,
                     float yl, float power, float dt, bool edges, cudaStream_t s) {
  int st = check_heat_params(h);
  if (st) return st;
  if (h->layout != PFG_LAYOUT_ZYX && h->layout != PFG_LAYOUT_XYZ) return PFG_ERR_PARAM;
  if (!Tg_in || !Tg_out) return PFG_ERR_NULL;
  if (!device_info().ok) return PFG_ERR_NO_DEVICE;
  if ((int64_t)(h->nx + 2) * (h->ny + 2) * (h->nz + 2) >= ((int64_t)1 << 31)) return PFG_ERR_SHAPE;
  const HeatConsts H = make_heat_consts(*h);
  const bool xyz = h->layout == PFG_LAYOUT_XYZ;
  const int chunks = ((xyz ? h->nx : h->nz) + kHeatChunk - 1) / kHeatChunk;
  if (chunks > 65535) return PFG_ERR_SHAPE;
  cudaError_t e;
  if (edges && chunks == 65535) {  // no grid row left for the edges: the whole field first
    const size_t bytes = sizeof(float) * (h->nx + 2) * (h->ny + 2) * (h->nz + 2);
    e = cudaMemcpyAsync(Tg_out, Tg_in, bytes, cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) return record_cuda(e);
    edges = false;
  }
  if (xyz) e = edges ? launch_heat<true, true>(H, Tg_in, Tg_out, xl, yl, power, dt, s)
                     : launch_heat<true, false>(H, Tg_in, Tg_out, xl, yl, power, dt, s);
  else e = edges ? launch_heat<false, true>(H, Tg_in, Tg_out, xl, yl, power, dt, s)
                 : launch_heat<false, false>(H, Tg_in, Tg_out, xl, yl, power, dt, s);
  return record_cuda(e);
}

}  // namespace pfg

using namespace pfg;

extern "C" int pfg_heat_step(const pfg_heat_params* h, const float* Tg_in, float* Tg_out,
                             float xl, float yl, float power, float dt, void* stream) {
  return heat_step(h, Tg_in, Tg_out, xl, yl, power, dt, false, static_cast<cudaStream_t>(stream));
}

extern "C" int pfg_heat_step_whole(const pfg_heat_params* h, const float* Tg_in, float* Tg_out,
                                   float xl, float yl, float power, float dt, void* stream) {
  return heat_step(h, Tg_in, Tg_out, xl, yl, power, dt, true, static_cast<cudaStream_t>(stream));
}
