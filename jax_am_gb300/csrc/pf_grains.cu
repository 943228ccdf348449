// Grain segmentation of a phase-field state on the device.
//
// The reference's post-processing (jax_am/phase_field/utils.py:181-310)
// finds the grains of a solution by a breadth-first search on the host: two
// face-adjacent cells belong to the same grain when both are solid
// (T < T_liquidus) and have the same argmax orientation; grains are listed by
// orientation, then in the order the search meets them (increasing smallest
// cell index); each grain's volume and PCA aspect ratio follow from its cells'
// centres.
//
// Here the components come from a two-level lock-free union-find:
//  1. a block labels a tile of 32 x 8 x 8 cells in shared memory: a row's runs
//     of one orientation come from a ballot, runs of adjacent rows unite
//     (Playne and Hawick's merge: find both roots, hang the larger under the
//     smaller with atomicMin, retry if that root moved) where they first touch;
//     every cell's label is its tile root (-1 in liquid);
//  2. the cells on tile faces unite their tiles' roots in global memory;
//  3. every cell's label is replaced by its root.
// A root is therefore the smallest cell index of its component -- the cell at
// which the reference's search starts that grain.  Roots are then numbered in
// increasing index order (a block-wise scan), and one pass adds each tile's
// count and first and second coordinate moments into its grains' records
// (exact integers: per run in closed form, per tile in shared memory, then one
// 64-bit atomic per grain of the tile and moment); a thread per grain takes its
// PCA aspect ratio from the moments.  The caller orders the records by
// (orientation, first cell) to obtain the reference's order, and the volumes
// from the cell counts.
//
// Bound: latency and L2.  A cell-by-cell merge in global memory took 2306 us of
// 2946 us at 8M cells (1,500 grains: every cell of a grain chases and updates
// the same few roots); within a tile the chains are short and in shared memory:
// 357 us in all (tiles 148, shapes 49, faces 48, moments 48, roots 33).
//
// Termination: a label only ever decreases and never drops below its own
// root's index, and a non-root always points to a smaller index, so every find
// walks a strictly decreasing chain and every merge retry sees a smaller root.
#include <cuda_runtime.h>

#include <cstdint>

#include "pfg_host.h"
#include "pfg_step.cuh"

namespace pfg {

constexpr int kGrainThreads = 256;
constexpr int kScanItems = 8;                           // cells per thread in the numbering pass
constexpr int kScanChunk = kGrainThreads * kScanItems;  // cells per numbering block

struct GrainArgs {
  int nx, ny, nz;
  int T_ghosted;
  float T_liq;
  const int32_t* ori;
  const float* T;
  int32_t* L;        // labels (N)
  int32_t* id;       // grain number of each root (N; only roots are written)
  int32_t* chunk;    // roots per numbering chunk, then their exclusive offsets
  int32_t* out_of_cell;
  pfg_grain* grains;
  int64_t max_grains;
  int64_t* num_grains;
};

// Tiles: 32 cells along x (a warp's row), 8 along y and z.
constexpr int kTileX = 32, kTileY = 8, kTileZ = 8;
constexpr int kTileRows = kTileY * kTileZ, kTileCells = kTileX * kTileRows;
static_assert(kGrainThreads == kTileY * 32, "a warp takes one y of every z plane of the tile");

struct Tile {
  int x0, y0, z0;
};
__device__ __forceinline__ Tile tile_of(const GrainArgs& a, int t) {
  const int tx = (a.nx + kTileX - 1) / kTileX, ty = (a.ny + kTileY - 1) / kTileY;
  const int q = t / tx;
  return Tile{(t - q * tx) * kTileX, (q % ty) * kTileY, (q / ty) * kTileZ};
}

template <bool GLOBAL>
__device__ __forceinline__ int load_label(const int32_t* L, int x) {
  if constexpr (GLOBAL) return __ldcg(L + x);
  else return *(volatile const int32_t*)(L + x);
}

template <bool GLOBAL>
__device__ __forceinline__ int find_root(const int32_t* L, int x) {
  int y = load_label<GLOBAL>(L, x);
  while (y != x) {
    x = y;
    y = load_label<GLOBAL>(L, x);
  }
  return x;
}

template <bool GLOBAL>
__device__ __forceinline__ void merge(int32_t* L, int a, int b) {
  bool done;
  do {
    a = find_root<GLOBAL>(L, a);
    b = find_root<GLOBAL>(L, b);
    if (a < b) {
      const int old = atomicMin(L + b, a);
      done = (old == b);
      b = old;
    } else if (b < a) {
      const int old = atomicMin(L + a, b);
      done = (old == a);
      a = old;
    } else {
      done = true;
    }
  } while (!done);
}

// Labels of one tile: every cell's is the global index of its tile root.
__global__ void __launch_bounds__(kGrainThreads) grain_tile_kernel(const GrainArgs a) {
  __shared__ int32_t s_ori[kTileCells], s_L[kTileCells];
  __shared__ unsigned s_start[kTileRows];  // where a row's runs start (liquid cells too)
  const int lane = threadIdx.x & 31, yl = threadIdx.x >> 5;
  const Tile t = tile_of(a, blockIdx.x);
  const int x = t.x0 + lane, y = t.y0 + yl, xy = a.nx * a.ny;
  const bool col = x < a.nx && y < a.ny;
#pragma unroll
  for (int zl = 0; zl < kTileZ; ++zl) {
    const int z = t.z0 + zl, r = zl * kTileY + yl;
    int o = 0;
    bool solid = false;
    if (col && z < a.nz) {
      const int i = z * xy + y * a.nx + x;
      const float T = a.T_ghosted
                          ? a.T[((int64_t)(z + 1) * (a.ny + 2) + (y + 1)) * (a.nx + 2) + x + 1]
                          : a.T[i];
      o = a.ori[i];
      solid = T < a.T_liq;  // NaN T is not solid, as in the reference's compare
    }
    const int o_left = __shfl_up_sync(0xffffffffu, o, 1);
    const unsigned solids = __ballot_sync(0xffffffffu, solid);
    const bool joins = lane > 0 && solid && (solids >> (lane - 1) & 1u) && o == o_left;
    const unsigned starts = ~__ballot_sync(0xffffffffu, joins);
    const int head = 31 - __clz(starts & (0xffffffffu >> (31 - lane)));
    s_ori[r * 32 + lane] = o;
    s_L[r * 32 + lane] = solid ? r * 32 + head : -1;
    if (lane == 0) s_start[r] = starts;
  }
  __syncthreads();
  // Two rows' runs unite at the first cell of each overlap: where either run
  // starts.  First within the z planes; then, every run pointing at its plane's
  // root again (the chains stay short), across them.
  auto unite = [&](int zl, int back) {  // with the row `back` rows before
    const int r = zl * kTileY + yl, c = r * 32 + lane, d = c - 32 * back;
    if (s_L[c] >= 0 && s_L[d] >= 0 && s_ori[d] == s_ori[c] &&
        ((s_start[r] | s_start[r - back]) >> lane & 1u))
      merge<false>(s_L, c, d);
  };
  if (yl > 0)
#pragma unroll
    for (int zl = 0; zl < kTileZ; ++zl) unite(zl, 1);
  __syncthreads();
#pragma unroll
  for (int zl = 0; zl < kTileZ; ++zl) {
    const int r = zl * kTileY + yl, c = r * 32 + lane;
    if ((s_start[r] >> lane & 1u) && s_L[c] >= 0) s_L[c] = find_root<false>(s_L, c);
  }
  __syncthreads();
#pragma unroll
  for (int zl = 1; zl < kTileZ; ++zl) unite(zl, kTileY);
  __syncthreads();
#pragma unroll
  for (int zl = 0; zl < kTileZ; ++zl) {
    const int z = t.z0 + zl, c = (zl * kTileY + yl) * 32 + lane;
    if (!col || z >= a.nz) continue;
    int g = -1;
    if (s_L[c] >= 0) {
      const int q = find_root<false>(s_L, c);
      g = (t.z0 + q / (32 * kTileY)) * xy + (t.y0 + q / 32 % kTileY) * a.nx + t.x0 + q % 32;
    }
    a.L[z * xy + y * a.nx + x] = g;
  }
}

// Unite across tile faces.  Along x, a face's pairs of cells unite one by one;
// across y and z faces a pair whose left neighbours are a pair of the same two
// tile components has nothing to add.
__global__ void __launch_bounds__(kGrainThreads) grain_faces_kernel(const GrainArgs a) {
  const int xy = a.nx * a.ny;
  const int64_t fx = (int64_t)((a.nx - 1) / kTileX) * a.ny * a.nz;
  const int64_t fy = (int64_t)((a.ny - 1) / kTileY) * a.nx * a.nz;
  const int64_t fz = (int64_t)((a.nz - 1) / kTileZ) * xy;
  for (int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; f < fx + fy + fz;
       f += (int64_t)gridDim.x * blockDim.x) {
    int i, j, x;
    if (f < fz) {
      const int p = (int)(f / xy), r = (int)(f - (int64_t)p * xy);
      i = (p + 1) * kTileZ * xy + r;
      j = i - xy;
      x = r % a.nx;
    } else if (f < fz + fy) {
      const int64_t g = f - fz;
      const int row = (int)(g / a.nx), k = (a.ny - 1) / kTileY;
      x = (int)(g - (int64_t)row * a.nx);
      i = (row / k) * xy + (row % k + 1) * kTileY * a.nx + x;
      j = i - a.nx;
    } else {
      const int64_t g = f - fz - fy;
      const int k = (a.nx - 1) / kTileX, row = (int)(g / k);
      x = (int)(g - (int64_t)row * k + 1) * kTileX;
      i = row * a.nx + x;
      j = i - 1;
      x = 0;
    }
    const int li = __ldcg(a.L + i), lj = __ldcg(a.L + j);
    if (li < 0 || lj < 0 || a.ori[i] != a.ori[j]) continue;
    if (x % kTileX && __ldcg(a.L + i - 1) == li && __ldcg(a.L + j - 1) == lj) continue;
    merge<true>(a.L, li, lj);
  }
}

// exclusive prefix sum of v over the block; *total receives the block's sum
__device__ __forceinline__ int block_exclusive_scan(int v, int* total) {
  __shared__ int s_warp[kGrainThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) s_warp[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    int w = (lane < kGrainThreads / 32) ? s_warp[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += t;
    }
    if (lane < kGrainThreads / 32) s_warp[lane] = w;  // inclusive over warps
  }
  __syncthreads();
  const int before = (warp > 0) ? s_warp[warp - 1] : 0;
  *total = s_warp[kGrainThreads / 32 - 1];
  __syncthreads();  // s_warp is reused by the next call
  return before + inc - v;
}

// every cell's label becomes its root; roots per chunk of kScanChunk cells
__global__ void __launch_bounds__(kGrainThreads) grain_roots_kernel(const GrainArgs a) {
  const int N = a.nx * a.ny * a.nz;
  const int base = blockIdx.x * kScanChunk + threadIdx.x;
  int c = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    const int i = base + k * kGrainThreads;
    if (i >= N) continue;
    const int l = __ldcg(a.L + i);
    if (l < 0) continue;
    if (l == i) {
      ++c;
    } else {
      const int r = find_root<true>(a.L, l);
      if (r != l) a.L[i] = r;
    }
  }
  c = __reduce_add_sync(0xffffffffu, c);
  __shared__ int s_c[kGrainThreads / 32];
  if ((threadIdx.x & 31) == 0) s_c[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    int total = 0;
    for (int w = 0; w < kGrainThreads / 32; ++w) total += s_c[w];
    a.chunk[blockIdx.x] = total;
  }
}

// exclusive offsets of the chunk counts (one block) and the grain count
__global__ void __launch_bounds__(kGrainThreads) grain_offsets_kernel(const GrainArgs a,
                                                                      int nchunks) {
  int carry = 0;
  for (int b0 = 0; b0 < nchunks; b0 += kGrainThreads) {
    const int b = b0 + threadIdx.x;
    const int v = (b < nchunks) ? a.chunk[b] : 0;
    int total;
    const int ex = block_exclusive_scan(v, &total);
    if (b < nchunks) a.chunk[b] = carry + ex;
    carry += total;
  }
  if (threadIdx.x == 0) *a.num_grains = carry;
}

// number the roots and start their records (a thread scans consecutive cells)
__global__ void __launch_bounds__(kGrainThreads) grain_number_kernel(const GrainArgs a,
                                                                     int nchunks) {
  const int N = a.nx * a.ny * a.nz;
  const int first = a.chunk[blockIdx.x];
  const int next = (int)blockIdx.x + 1 < nchunks ? a.chunk[blockIdx.x + 1] : (int)*a.num_grains;
  if (first == next) return;  // no root here (most chunks)
  const int base = blockIdx.x * kScanChunk + threadIdx.x * kScanItems;
  int c = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    const int i = base + k;
    if (i < N && a.L[i] == i) ++c;
  }
  int total;
  int g = first + block_exclusive_scan(c, &total);
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    const int i = base + k;
    if (i < N && a.L[i] == i) {
      a.id[i] = g;
      if (g < a.max_grains) {
        pfg_grain& G = a.grains[g];
        G.first_cell = i;
        G.ori = a.ori[i];
        G.reserved = 0;
        G.cells = 0;
        for (int d = 0; d < 3; ++d) G.sum[d] = 0;
        for (int d = 0; d < 6; ++d) G.sum2[d] = 0;
      }
      ++g;
    }
  }
}

// The moments of a set of cells as sums over (1, x, y, z, xx, yy, zz, xy, xz, yz),
// moved by (X, Y, Z): the records hold whole-grid coordinates, a tile's table
// its own.
template <typename I>
__device__ __forceinline__ long long moved_moment(const I* v, int m, long long X, long long Y,
                                                  long long Z) {
  const long long c = v[0], x = v[1], y = v[2], z = v[3];
  switch (m) {
    case 0: return c;
    case 1: return x + c * X;
    case 2: return y + c * Y;
    case 3: return z + c * Z;
    case 4: return v[4] + 2 * x * X + c * X * X;
    case 5: return v[5] + 2 * y * Y + c * Y * Y;
    case 6: return v[6] + 2 * z * Z + c * Z * Z;
    case 7: return v[7] + x * Y + y * X + c * X * Y;
    case 8: return v[8] + x * Z + z * X + c * X * Z;
    default: return v[9] + y * Z + z * Y + c * Y * Z;
  }
}

// Per-cell grain numbers and the grains' moments, a tile per block.  A row's
// runs add their closed-form moments to a small table of the tile's grains in
// shared memory (tile coordinates: below 2^21, so 32 bits hold them); the
// table goes to the records with one atomic per grain and moment.  A run
// whose grain finds no place in the table adds to the record itself.
constexpr int kMoments = 10, kTable = 128, kProbes = 16;
__global__ void __launch_bounds__(kGrainThreads) grain_moments_kernel(const GrainArgs a) {
  __shared__ int s_key[kTable];
  __shared__ int s_sum[kTable][kMoments + 1];
  const int lane = threadIdx.x & 31, yl = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < kTable; i += kGrainThreads) s_key[i] = -1;
  for (int i = threadIdx.x; i < kTable * (kMoments + 1); i += kGrainThreads)
    (&s_sum[0][0])[i] = 0;
  __syncthreads();
  const Tile t = tile_of(a, blockIdx.x);
  const int x = t.x0 + lane, y = t.y0 + yl, xy = a.nx * a.ny;
  const bool col = x < a.nx && y < a.ny;
  auto record = [&](int g) { return reinterpret_cast<unsigned long long*>(&a.grains[g].cells); };
#pragma unroll
  for (int zl = 0; zl < kTileZ; ++zl) {
    const int z = t.z0 + zl;
    int g = -1;
    if (col && z < a.nz) {
      const int i = z * xy + y * a.nx + x;
      const int root = __ldcg(a.L + i);
      if (root >= 0) g = __ldg(a.id + root);
      if (a.out_of_cell) a.out_of_cell[i] = g;
    }
    const int left = __shfl_up_sync(0xffffffffu, g, 1);
    const bool start = lane == 0 || g != left;
    const unsigned starts = __ballot_sync(0xffffffffu, start);
    if (!start || g < 0 || g >= a.max_grains) continue;
    const unsigned later = lane == 31 ? 0u : starts & (0xfffffffeu << lane);
    const int end = later ? __ffs(later) - 1 : 32;  // the run is lane .. end - 1
    const int c = end - lane, b = end - 1;
    const int sx = c * (lane + b) / 2;
    const int sxx = (b * (b + 1) * (2 * b + 1) - (lane - 1) * lane * (2 * lane - 1)) / 6;
    const int v[kMoments] = {c,           sx,      c * yl,  c * zl,      sxx,
                             c * yl * yl, c * zl * zl, sx * yl, sx * zl, c * yl * zl};
    int at = (int)(((unsigned)g * 2654435761u) >> 25);  // 7 bits: the table's size
    bool placed = false;
    for (int probe = 0; probe < kProbes && !placed; ++probe) {
      const int old = atomicCAS(&s_key[at], -1, g);
      placed = old == -1 || old == g;
      if (!placed) at = (at + 1) & (kTable - 1);
    }
    if (placed) {
#pragma unroll
      for (int m = 0; m < kMoments; ++m) atomicAdd(&s_sum[at][m], v[m]);
    } else {
      for (int m = 0; m < kMoments; ++m)
        atomicAdd(record(g) + m, (unsigned long long)moved_moment(v, m, t.x0, t.y0, t.z0));
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kTable * kMoments; i += kGrainThreads) {
    const int e = i / kMoments, m = i - e * kMoments, g = s_key[e];
    if (g >= 0)
      atomicAdd(record(g) + m,
                (unsigned long long)moved_moment(s_sum[e], m, t.x0, t.y0, t.z0));
  }
}
static_assert(kTable == 128, "the table's hash takes 7 bits");

// Eigenvalues of a symmetric 3 x 3 matrix (a00, a11, a22, a01, a02, a12) by cyclic
// Jacobi rotations (Golub and Van Loan's symmetric Schur decomposition).
__device__ void eigenvalues3(double* a) {
  for (int sweep = 0; sweep < 12; ++sweep) {
    if (a[3] == 0.0 && a[4] == 0.0 && a[5] == 0.0) return;
    for (int k = 0; k < 3; ++k) {
      // rotate the plane (p, q); r is the third axis
      const int p = k == 2 ? 1 : 0, q = k == 0 ? 1 : 2, r = 3 - p - q;
      const int pq = p + q + 2, pr = p + r + 2, qr = q + r + 2;
      const double apq = a[pq];
      if (apq == 0.0) continue;
      const double tau = (a[q] - a[p]) / (2.0 * apq);
      const double t = (tau >= 0.0 ? 1.0 : -1.0) / (fabs(tau) + sqrt(1.0 + tau * tau));
      const double c = 1.0 / sqrt(1.0 + t * t), s = t * c;
      a[p] -= t * apq;
      a[q] += t * apq;
      a[pq] = 0.0;
      const double arp = a[pr], arq = a[qr];
      a[pr] = c * arp - s * arq;
      a[qr] = s * arp + c * arq;
    }
  }
}

// A grain's aspect ratio from its exact moments (utils.py:286-310): covariance
// of the cell centres (ddof = 1, numerators exact in 128-bit integers), square
// roots of its eigenvalues in descending order l0, l1, l2: 2 l0 / (l1 + l2); 1
// below 5 cells.
static_assert(sizeof(pfg_grain_shape) == 32, "four words per grain");
__global__ void __launch_bounds__(128) grain_shapes_kernel(const pfg_grain* grains,
                                                           const int64_t* num_grains,
                                                           int64_t max_grains,
                                                           pfg_grain_shape* out) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t K = *num_grains < max_grains ? *num_grains : max_grains;
  if (g >= K) return;
  const pfg_grain& G = grains[g];
  const long long c = G.cells;
  double ratio = 1.0;
  if (c >= 5) {
    const double den = (double)c * (double)(c - 1);  // exact below 2^53
    double a[6];
    const int pi[6] = {0, 1, 2, 0, 0, 1}, qi[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      const __int128 v = (__int128)c * G.sum2[m] - (__int128)G.sum[pi[m]] * G.sum[qi[m]];
      // the magnitude's two halves, one rounding (exact below 2^53)
      const unsigned __int128 u = v < 0 ? -(unsigned __int128)v : (unsigned __int128)v;
      const double d = fma((double)(unsigned long long)(u >> 64), 18446744073709551616.0,
                           (double)(unsigned long long)u);
      a[m] = (v < 0 ? -d : d) / den;
    }
    eigenvalues3(a);
    double l[3];
    for (int m = 0; m < 3; ++m) l[m] = sqrt(a[m] > 0.0 ? a[m] : 0.0);
    const double l0 = fmax(fmax(l[0], l[1]), l[2]), l2 = fmin(fmin(l[0], l[1]), l[2]);
    const double l1 = fmax(fmin(l[0], l[1]), fmin(fmax(l[0], l[1]), l[2]));
    ratio = 2.0 * l0 / (l1 + l2);  // collinear: infinite
  }
  out[g] = pfg_grain_shape{G.first_cell, G.ori, 0, c, ratio};
}

// labels[i] = rank[labels[i]] in place (-1 stays)
__global__ void __launch_bounds__(kGrainThreads) grain_relabel_kernel(int64_t N,
                                                                      const int32_t* rank,
                                                                      int32_t* labels) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int g = labels[i];
    if (g >= 0) labels[i] = __ldg(rank + g);
  }
}

static int grain_grid(int64_t N) {
  const DeviceInfo& d = device_info();
  const int64_t want = (N + kGrainThreads - 1) / kGrainThreads;
  const int64_t cap = (int64_t)d.sm_count * 8;
  return (int)(want < cap ? (want > 0 ? want : 1) : cap);
}

static int64_t chunk_count(int64_t N) { return (N + kScanChunk - 1) / kScanChunk; }

}  // namespace pfg

using namespace pfg;

// scratch: labels (N), root numbers (N), chunk counts, each 256-byte aligned
static int64_t align256(int64_t b) { return (b + 255) / 256 * 256; }

extern "C" int64_t pfg_grain_scratch_bytes(const pfg_pf_params* p) {
  if (check_pf_params(p)) return -1;
  const int64_t N = (int64_t)p->nx * p->ny * p->nz;
  return 2 * align256(N * 4) + align256(chunk_count(N) * 4);
}

extern "C" int pfg_grains(const pfg_pf_params* p, const int32_t* ori, const float* T,
                          int T_ghosted, int32_t* grain_of_cell, pfg_grain* grains,
                          int64_t max_grains, int64_t* num_grains, void* scratch,
                          int64_t scratch_bytes, void* stream) {
  int st = check_pf_params(p);
  if (st) return st;
  if (!ori || !T || !num_grains || !scratch || (max_grains > 0 && !grains)) return PFG_ERR_NULL;
  if (max_grains < 0) return PFG_ERR_PARAM;
  if (reinterpret_cast<uintptr_t>(grains) % 8 != 0) return PFG_ERR_ALIGN;
  const int64_t N = (int64_t)p->nx * p->ny * p->nz;
  // 32-bit cell labels, with room for the last block's and grid's index ranges
  if (N >= ((int64_t)1 << 31) - ((int64_t)1 << 22)) return PFG_ERR_SHAPE;
  if (scratch_bytes < pfg_grain_scratch_bytes(p)) return PFG_ERR_CAPACITY;
  if (!device_info().ok) return PFG_ERR_NO_DEVICE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  GrainArgs a{};
  a.nx = p->nx; a.ny = p->ny; a.nz = p->nz;
  a.T_ghosted = T_ghosted;
  a.T_liq = p->T_liquidus;
  a.ori = ori; a.T = T;
  char* sp = static_cast<char*>(scratch);
  a.L = reinterpret_cast<int32_t*>(sp);
  a.id = reinterpret_cast<int32_t*>(sp + align256(N * 4));
  a.chunk = reinterpret_cast<int32_t*>(sp + 2 * align256(N * 4));
  a.out_of_cell = grain_of_cell;
  a.grains = grains;
  a.max_grains = max_grains;
  a.num_grains = num_grains;
  const int grid = grain_grid(N);
  const int nchunks = (int)chunk_count(N);
  // tile counts stay below 2^31: at least one cell per tile
  const unsigned tiles = (unsigned)((p->nx + kTileX - 1) / kTileX) *
                         (unsigned)((p->ny + kTileY - 1) / kTileY) *
                         (unsigned)((p->nz + kTileZ - 1) / kTileZ);
  grain_tile_kernel<<<tiles, kGrainThreads, 0, s>>>(a);
  grain_faces_kernel<<<grid, kGrainThreads, 0, s>>>(a);
  grain_roots_kernel<<<nchunks, kGrainThreads, 0, s>>>(a);
  grain_offsets_kernel<<<1, kGrainThreads, 0, s>>>(a, nchunks);
  grain_number_kernel<<<nchunks, kGrainThreads, 0, s>>>(a, nchunks);
  grain_moments_kernel<<<tiles, kGrainThreads, 0, s>>>(a);
  return record_cuda(cudaGetLastError());
}

extern "C" int pfg_grain_shapes(const pfg_grain* grains, const int64_t* num_grains,
                                int64_t max_grains, pfg_grain_shape* out, void* stream) {
  if (max_grains < 0) return PFG_ERR_PARAM;
  if (!num_grains || (max_grains > 0 && (!grains || !out))) return PFG_ERR_NULL;
  if ((reinterpret_cast<uintptr_t>(grains) | reinterpret_cast<uintptr_t>(out)) % 8 != 0)
    return PFG_ERR_ALIGN;
  if (!device_info().ok) return PFG_ERR_NO_DEVICE;
  const int64_t blocks = (max_grains + 127) / 128;
  if (blocks > 0x7fffffff) return PFG_ERR_SHAPE;
  if (blocks)
    grain_shapes_kernel<<<(unsigned)blocks, 128, 0, static_cast<cudaStream_t>(stream)>>>(
        grains, num_grains, max_grains, out);
  return record_cuda(cudaGetLastError());
}

extern "C" int pfg_grain_relabel(int64_t num_cells, const int32_t* rank, int32_t* labels,
                                 void* stream) {
  if (num_cells < 1) return PFG_ERR_SHAPE;
  if (!rank || !labels) return PFG_ERR_NULL;
  if (!device_info().ok) return PFG_ERR_NO_DEVICE;
  grain_relabel_kernel<<<grain_grid(num_cells), kGrainThreads, 0,
                         static_cast<cudaStream_t>(stream)>>>(num_cells, rank, labels);
  return record_cuda(cudaGetLastError());
}
