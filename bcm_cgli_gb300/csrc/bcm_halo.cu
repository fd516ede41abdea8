// Ghost-layer kernels around the flux: cube-to-cube interface, the X/Y/Z
// boundary conditions and the immersed-boundary ghost cells.
//
// All three are pure data movement plus a little FP64 arithmetic; each is
// organised so one CTA or cluster owns the cells it writes and only reads cells
// that no other writes during the launch, which makes every launch race-free and
// gives the reference's results exactly.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "bcm_common.cuh"
#include "bcm_fp64_int.cuh"
#include "bcm_kernels.h"

namespace bcmg {

namespace cg = cooperative_groups;

constexpr int kHaloThreads = 256, kLayerThreads = 256;

// The cube a cluster of k_layers works on: its arrays (and the offset of its
// first value in the flat ones), the mirror's reference state, the inflow
// velocity.
struct LayerCube {
  double *U;
  float *M;  // current mirror, nullptr: none
  ptrdiff_t base;
  double r0, e0, Uin;
};

// ---------------------------------------------------------------------------
// Interface (BCM_Interface.cpp).  Same-level faces (:1745-1783 x, :2608-2642
// y, :3478-3512 z) copy the neighbour's two interior layers into this cube's
// two ghost layers over the n x n face; every read is an interior cell, every
// write a ghost cell of the task's destination cube, so all face tasks run in
// parallel.  A pass after them averages the edge ghosts in the
// reference's three ordered phases (:5640-5732): i-edges, then j-edges, then
// k-edges.
// ---------------------------------------------------------------------------
// Level-jump faces (BCM_Interface.cpp:1790-2599 x, :2651-3470 y,
// :3518-4358 z).  Sub-face slot s offsets the tangential axes (x<y<z order)
// by ((s==2||s==4) n/2, (s==3||s==4) n/2).
//  kind 1, coarse -> fine: the small cube's two ghost layers facing the big
//    cube take the big cube's adjacent interior cell (n+1 or 2 along the
//    axis, (p/2+1, q/2+1) + slot offset across it), both layers alike;
//  kind 2, fine -> coarse: the big cube's two ghost layers over the slot's
//    quadrant take 0.125 * the sum of the small cube's 2x2x2 interior cells,
//    summed in the reference's order (000,100,010,001,110,101,011,111 in i,j,k).
// With a mirror (split precision) every written value's mirror value is
// written too: injections copy the source's, averages are converted.
__device__ __forceinline__ void level_face(const LayerArgs &a, const LayerCube &z,
                                           const FaceTask &ft) {
  const int n = a.n, S = n + 4, h = n / 2, ax = ft.axis;
  // strides (values) along the face's axis and the in-face axes, x<y<z order
  const int sx = ax == 0 ? 5 * S * S : (ax == 1 ? 5 * S : 5);
  const int s0 = ax == 0 ? 5 * S : 5 * S * S, s1 = ax == 2 ? 5 * S : 5;
  const int o0 = (ft.slot == 2 || ft.slot == 4) ? h : 0;
  const int o1 = (ft.slot == 3 || ft.slot == 4) ? h : 0;
  const ptrdiff_t other = cell_index(S, ft.src, 0, 0, 0) * 5;  // the neighbour
  const double *B = a.U1_ + other;
  const float *MB = z.M ? z.M + (other - z.base) : nullptr;
  if (ft.kind == 1) {
    const int gs = (ft.side == 0 ? n + 1 : 2) * sx;
    for (int w = threadIdx.x; w < 2 * n * n * 5; w += kLayerThreads) {
      const int v = w % 5, cell = w / 5;
      const int row = cell / n, q = cell - row * n, l = row >= n, p = row - l * n;
      const int os = gs + (p / 2 + 2 + o0) * s0 + (q / 2 + 2 + o1) * s1 + v;
      const int od = (ft.side == 0 ? l : n + 2 + l) * sx + (p + 2) * s0 + (q + 2) * s1 + v;
      z.U[od] = B[os];
      if (z.M) z.M[od] = MB[os];
    }
  } else {
    for (int w = threadIdx.x; w < 2 * h * h * 5; w += kLayerThreads) {
      const int v = w % 5, cell = w / 5;
      const int row = cell / h, q = cell - row * h, l = row >= h, p = row - l * h;
      const double *x = B + (ft.side == 1 ? 2 * (l + 1) : n - 2 + 2 * l) * sx + (2 * p + 2) * s0 +
                        (2 * q + 2) * s1 + v;
      const int si = 5 * S * S, sj = 5 * S, sk = 5;
      double sum = x[0];
      sum = sum + x[si];
      sum = sum + x[sj];
      sum = sum + x[sk];
      sum = sum + x[si + sj];
      sum = sum + x[si + sk];
      sum = sum + x[sj + sk];
      sum = sum + x[si + sj + sk];
      const int od = (ft.side == 1 ? n + 2 + l : l) * sx + (p + 2 + o0) * s0 + (q + 2 + o1) * s1 + v;
      z.U[od] = 0.125 * sum;
      if (z.M) z.M[od] = mirror_value(0.125 * sum, v, z.r0, z.e0);
    }
  }
}

// One same-level face task by the threads of a CTA.  Copies move pairs of
// values (16-byte pairs of doubles, 8-byte pairs of mirror floats): S is even,
// so every row below starts at an even value and is 5n or 10 values long (n is
// a multiple of 4).  Rows are the n cells along the innermost index that both
// source and destination store contiguously (k for x and y faces); for z faces
// a row is one (i, j) column of the two ghost layers.  The mirror (split
// precision) is copied like the state: an exact copy of a value has the same
// rounding.  Source (the neighbour's interior) and destination (this cube's
// ghost layers) never overlap: a thread issues its loads for kCopyBatch items
// before storing them, so the copies are not a chain of round trips.
constexpr int kCopyBatch = 4;

__device__ __forceinline__ void face_copy(const LayerArgs &a, const LayerCube &z,
                                          const FaceTask &ft) {
  const int n = a.n, S = n + 4, ax = ft.axis;
  double2 *const D = reinterpret_cast<double2 *>(z.U);
  float2 *const DM = reinterpret_cast<float2 *>(z.M);
  const ptrdiff_t other = (ptrdiff_t)cell_index(S, ft.src, 0, 0, 0) * 5;
  // everything in pairs; source minus destination is one constant: the cubes
  // and n layers
  const int len = ax < 2 ? 5 * n / 2 : 5, rows = ax < 2 ? n : n * n;
  const int srow = ax == 0 ? 5 * S / 2 : 5 * S * S / 2;  // next row of a layer
  const int layer = ax == 0 ? 5 * S * S / 2 : 5 * S / 2;
  const int g = ft.side == 0 ? 0 : n + 2;
  const ptrdiff_t shift =
      (other - z.base) / 2 + (ft.side == 0 ? n : -n) * (ax == 0 ? 5 * S * S : (ax == 1 ? 5 * S : 5)) / 2;
  const int total = len * rows * (ax < 2 ? 2 : 1);
  auto dest = [&](int w) {
    const int row = w / len, e = w - row * len;
    if (ax == 2) {
      const int i = row / n, j = row - i * n;
      return ((i + 2) * S + j + 2) * (5 * S / 2) + 5 * g / 2 + e;
    }
    const int l = row >= n, p = row - l * n;
    return (g + l) * layer + (p + 2) * srow + 5 + e;
  };
  for (int w0 = threadIdx.x; w0 < total; w0 += kCopyBatch * kLayerThreads) {
    double2 u[kCopyBatch];
    float2 m[kCopyBatch];
    int d[kCopyBatch];
#pragma unroll
    for (int b = 0; b < kCopyBatch; ++b)
      if (w0 + b * kLayerThreads < total) {
        d[b] = dest(w0 + b * kLayerThreads);
        u[b] = D[d[b] + shift];
        if (DM) m[b] = DM[d[b] + shift];
      }
#pragma unroll
    for (int b = 0; b < kCopyBatch; ++b)
      if (w0 + b * kLayerThreads < total) {
        D[d[b]] = u[b];
        if (DM) DM[d[b]] = m[b];
      }
  }
}

// Edge fill after all face copies (BCM_Interface.cpp:5640-5732).  The
// reference fills the layer-1 edge ghosts in three ordered phases: i-edges
// (i = 2..nx), then j-edges and k-edges over the whole ghost range, so the
// last two end at the corners.  Every edge cell that is not a corner reads
// two face ghosts (cells with one ghost coordinate), which no phase writes;
// the j-edge phase's corner values are overwritten by the k-edge phase
// before anything reads them; and the k-edge phase's corner value is the
// average of the j-edge and i-edge cells next to the corner, themselves
// averages of face ghosts.  So one pass computes each edge cell from two
// face ghosts and each corner from the two edge values it averages (formed
// from four face ghosts in registers): the reference's operations, the same
// bits, one round trip to memory instead of three dependent ones.
__device__ __forceinline__ void edge_fill(const LayerArgs &a, const LayerCube &z, int first,
                                          int stride) {
  const int n = a.n, S = n + 4, s0 = 5 * S * S, s1 = 5 * S, s2 = 5;
  // an edge cell at offset o: its inward neighbours across its ghost axes
  auto edge = [&](int o, int da, int db) { return 0.5 * (z.U[o + da] + z.U[o + db]); };
  const int nedge = 12 * n, items = 5 * (nedge + 8);
#pragma unroll 2
  for (int w = first; w < items; w += stride) {
    const int v = w % 5, cell = w / 5;
    double r;
    int o;
    if (cell < nedge) {
      // edge family f (free coordinate i, j or k = 2..nx), its two ghost axes
      // a, b (a < b) and their sides
      const int f = cell / (4 * n), rem = cell - f * 4 * n, pos = 2 + (rem >> 2);
      const int sa = f == 0 ? s1 : s0, sb = f == 2 ? s1 : s2, sf = f == 0 ? s0 : (f == 1 ? s1 : s2);
      const int ua = rem & 1, ub = rem >> 1 & 1;
      o = pos * sf + (ua ? n + 2 : 1) * sa + (ub ? n + 2 : 1) * sb + v;
      r = edge(o, ua ? -sa : sa, ub ? -sb : sb);
    } else {
      // corner: the k-edge phase's average of the j-edge cell and the i-edge
      // cell next to it
      const int q = cell - nedge, d0 = q & 1 ? -s0 : s0, d1 = q & 2 ? -s1 : s1,
                d2 = q & 4 ? -s2 : s2;
      o = (q & 1 ? n + 2 : 1) * s0 + (q & 2 ? n + 2 : 1) * s1 + (q & 4 ? n + 2 : 1) * s2 + v;
      const double xj = edge(o + d1, d0, d2), yi = edge(o + d0, d1, d2);
      r = 0.5 * (xj + yi);
    }
    z.U[o] = r;
    if (z.M) z.M[o] = mirror_value(r, v, z.r0, z.e0);
  }
}

// ---------------------------------------------------------------------------
// Halo exchange of cube-sharded runs: the face bands a remote rank's face
// tasks read, gathered from this rank's cubes into a buffer, or scattered
// from a buffer into the proxy slots that stand for the remote cubes.  One
// CTA per band; a band's cells go in (layer, first in-face index, second)
// order, the in-face axes in x<y<z order.  Pure copies, so the proxies hold
// the remote cells bit for bit.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kHaloThreads)
    k_halo(double *U, Mirror mir, const int *bands, const long long *offs, long long total_cells,
           int n, double *bufU, int unpack) {
  float *M = mirror_current(mir);  // split precision: the current mirror too
  const int b = blockIdx.x;
  const int c = bands[4 * b], ax = bands[4 * b + 1], side = bands[4 * b + 2],
            L = bands[4 * b + 3];
  const int S = n + 4;
  const int t0 = ax == 0 ? 1 : 0, t1 = ax == 2 ? 1 : 2;
  const int l0 = side == 1 ? n + 2 - L : 2;  // first layer along the axis
  const long long o0 = offs[b];
  float *bufM = M ? reinterpret_cast<float *>(bufU + 5 * total_cells) : nullptr;
  const int cells = L * n * n;
  for (int w = threadIdx.x; w < cells * 5; w += blockDim.x) {
    const int v = w % 5, cell = w / 5;
    const int l = cell / (n * n), p = (cell / n) % n, q = cell % n;
    int x[3];
    x[ax] = l0 + l;
    x[t0] = 2 + p;
    x[t1] = 2 + q;
    const size_t g = 5 * cell_index(S, c, x[0], x[1], x[2]) + v;
    const size_t h = 5 * (size_t)(o0 + cell) + v;
    if (unpack) {
      U[g] = bufU[h];
      if (M) M[g] = bufM[h];
    } else {
      bufU[h] = U[g];
      if (M) bufM[h] = M[g];
    }
  }
}

cudaError_t launch_halo(double *U, const Mirror &mir, const int *bands, const long long *offs,
                        int nband, long long total_cells, int n, void *buf, int unpack,
                        cudaStream_t s) {
  if (nband <= 0) return cudaSuccess;
  k_halo<<<nband, kHaloThreads, 0, s>>>(U, mir, bands, offs, total_cells, n,
                                        static_cast<double *>(buf), unpack);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Boundary conditions (BCM_X/Y/Z_boundary_condition.cpp) in one pass.  The
// reference fills the x faces (j, k interior: inflow from cell 2, zero
// gradient from cell nx), then the y faces over every i (zero gradient from
// row 2 / nx, interior k), then the z faces over every i, j (slip with w
// negated from plane 2, zero gradient from plane nx), in that order
// (main.cpp:1161-1165), so a y face's x-ghost rows copy values the x phase
// wrote and a z face copies both.  Each value a phase reads is, through at
// most two earlier phases, a copy or the inflow formula of a cell no phase
// writes: read() follows that chain.  So every ghost position is formed
// directly, with the reference's operations, in one pass with no barrier:
// the same bits (checked on the CPU against the ordered phases for every
// mask and axis subset, and by the GPU parity tests).  `axes` limits the
// pass to the faces of one twin call (the others' ghosts are then read as
// they are).
// ---------------------------------------------------------------------------
// The inflow's total energy: pressure of the cell next to it, velocity (Uin, 0,
// 0).  A call: inlined at each of a thread's items its three divisions made
// the kernel wait for instructions.
__device__ __noinline__ double inflow_energy(const double *q, double Uin) {
  const double rho = q[0];
  const double Uu = Uin, Vv = 0., Ww = 0;
  const double U0 = q[1] / rho, V0 = q[2] / rho, W0 = q[3] / rho;
  double VV = U0 * U0 + V0 * V0 + W0 * W0;
  const double P = (q[4] - 0.5 * rho * VV) * (BCMG_K - 1);
  VV = Uu * Uu + Vv * Vv + Ww * Ww;
  return P / (BCMG_K - 1) + 0.5 * rho * VV;
}

constexpr int kBcBatch = 2;

// cover: boundary faces (bits as in m) that a same-level face task also fills
// (a periodic box's boundary lists name such faces): over their interior n x n
// positions the opening interface call would put the neighbour's cells back
// before anything reads them, so nothing is written there and the layers stay
// as the last interface call, or this launch's full one, leaves them.
__device__ __forceinline__ void bc_fill(const LayerArgs &a, const LayerCube &z, int m, int cover,
                                        int first, int stride) {
  const int n = a.n, S = n + 4, nx = n + 1, nxx = n + 2;
  const int mx = (a.axes & 1) ? (m & 3) : 0, my = (a.axes & 2) ? ((m >> 2) & 3) : 0,
            mz = (a.axes & 4) ? ((m >> 4) & 3) : 0;
  double *const U = z.U;
  // Split precision: the mirror values of every write, into both mirror
  // buffers.  The flux kernel writes the next buffer's interior cells and
  // same-level ghost layers, and the interface call after it the level-jump
  // layers and edges; the boundary layers are written here only, so the
  // next buffer takes them now and equals the state's rounding in every
  // cell once it becomes current.
  float *const M = z.M;
  float *const Mo = M ? (mirror_index(a.mir) ? a.mir.buf[0] : a.mir.buf[1]) + z.base : nullptr;
  const double Uin = z.Uin;
  // ghost positions: x faces n^2 each, y faces S n each, z faces S^2 each
  // (covered faces: none, the 4 n and the 8 n + 16 outside n x n); each
  // position fills both ghost layers with one value.  Items are (position,
  // component), component fastest, so a warp's loads and stores run over
  // whole cells in a row.
  auto count = [&](int f) -> int {  // positions of face f
    if (!((f < 2 ? mx : (f < 4 ? my : mz)) >> (f & 1) & 1)) return 0;
    const bool cov = cover >> f & 1;
    return f < 2 ? (cov ? 0 : n * n) : (f < 4 ? (cov ? 4 : S) * n : (cov ? 8 * n + 16 : S * S));
  };
  int end[6];
#pragma unroll
  for (int f = 0; f < 6; ++f) end[f] = count(f) + (f ? end[f ? f - 1 : 0] : 0);
  const int items = 5 * end[5];
  auto ghost = [&](int g) { return g < 2 ? g : n + g; };
  // Item w: the cell its value comes from as the reference's order of phases
  // leaves it there (offset in the cube), whether that is the inflow formula
  // of the cell, and its first destination (the second is `step` further).
  auto item = [&](int w, int &src, int &v, bool &infl, bool &neg, int &dst, int &step) {
    v = w % 5;
    int q = w / 5, f = 0, before = 0;
#pragma unroll
    for (int g = 0; g < 5; ++g)
      if (q >= end[g]) { f = g + 1; before = end[g]; }
    q -= before;
    const int ax = f >> 1, up = f & 1;
    const bool cov = cover >> f & 1;
    // (p, r): the position's in-face indices, x<y<z order
    int p, r;
    if (ax < 2) {
      p = q / n;
      r = 2 + q - p * n;
      p = ax == 0 ? p + 2 : (cov ? ghost(p) : p);
    } else if (!cov || q < 4 * S) {
      p = q / S;
      r = q - p * S;
      if (cov) p = ghost(p);
    } else {
      q -= 4 * S;
      p = 2 + (q >> 2);
      r = ghost(q & 3);
    }
    const int in = up ? nx : 2;
    int i = ax == 0 ? in : p, j = ax == 0 ? p : (ax == 1 ? in : r), k = ax == 2 ? in : r;
    const int g = up ? nxx : 1;
    dst = ax == 0 ? (g * S + j) * S + k : (ax == 1 ? (i * S + g) * S + k : (i * S + j) * S + g);
    step = (ax == 0 ? S * S : (ax == 1 ? S : 1)) * (up ? 1 : -1);
    infl = ax == 0 && !up;
    neg = ax == 2 && !up;  // slip wall: rho*w negated (:42-65)
    if (ax == 2) {  // rows the y phase wrote
      if ((my & 1) && j <= 1) j = 2;
      else if ((my & 2) && j >= nxx) j = nx;
    }
    if (ax > 0 && mx && j >= 2 && j <= nx) {  // and the x phase
      if ((mx & 1) && i <= 1) { i = 2; infl = true; }
      else if ((mx & 2) && i >= nxx) i = nx;
    }
    src = (i * S + j) * S + k;
  };
  // kBcBatch items per round, all loaded before any is stored
  for (int w0 = first; w0 < items; w0 += kBcBatch * stride) {
    double x[kBcBatch];
    int src[kBcBatch], v[kBcBatch], dst[kBcBatch], step[kBcBatch];
    bool infl[kBcBatch], neg[kBcBatch];
#pragma unroll
    for (int b = 0; b < kBcBatch; ++b)
      if (w0 + b * stride < items) {
        item(w0 + b * stride, src[b], v[b], infl[b], neg[b], dst[b], step[b]);
        x[b] = U[5 * src[b] + (infl[b] && v[b] < 4 ? 0 : v[b])];
      }
#pragma unroll
    for (int b = 0; b < kBcBatch; ++b)
      if (w0 + b * stride < items) {
        if (infl[b]) {  // rho and p from the cell, u = Uin, v = w = 0 (:43-80)
          if (v[b] == 1) x[b] = x[b] * Uin;
          else if (v[b] == 2 || v[b] == 3) x[b] = x[b] * 0.0;
          else if (v[b] == 4) x[b] = inflow_energy(U + 5 * src[b], Uin);
        }
        if (neg[b] && v[b] == 3) x[b] = -x[b];
        const int d1 = 5 * dst[b] + v[b], d0 = d1 + 5 * step[b];
        U[d1] = x[b];
        U[d0] = x[b];
        if (M) {
          const float mv = mirror_value(x[b], v[b], z.r0, z.e0);
          M[d1] = mv; M[d0] = mv; Mo[d1] = mv; Mo[d0] = mv;
        }
      }
  }
}

// ---------------------------------------------------------------------------
// The ghost layers of a cube by a cluster of CTAs.  Each of the up to five
// passes writes ghost cells of its cube only and reads the cube's own cells
// and other cubes' interior cells, which no pass writes: so passes depend on
// each other within a cube only, and barriers of its cluster order them.
// That replaces four or five launches a stage (closing faces, closing edges,
// boundary conditions, opening faces, opening edges), each of 8 to 45 us, most
// of it launch and dependent round trips, whatever the number of cubes: 512
// periodic cubes of 24^3 about 110 -> 34 us a stage, and with the mirror flag's
// and E normalisation's launches gone too, a step of 10 sub-iterations of 8
// cubes of 8^3 1.21 -> 0.80 ms.  What bounds it now: the passes' dependent
// loads (4 CTAs of 64 registers on an SM).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kLayerThreads, 4) k_layers(LayerArgs a) {
  const cg::cluster_group cl = cg::this_cluster();
  const int size = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int q = blockIdx.x / size;
  const int c = a.cubes ? a.cubes[q] : q + 1;
  if (!case_active(a.bt, c)) return;  // converged case (the whole cluster)
  const int flags = a.flags ? a.flags[a.cubes ? q : c] : 0;
  const int first = rank * kLayerThreads + threadIdx.x, stride = size * kLayerThreads;
  LayerCube z;
  z.base = (ptrdiff_t)cell_index(a.n + 4, c, 0, 0, 0) * 5;
  z.U = a.U1_ + z.base;
  z.M = mirror_current(a.mir);
  z.r0 = z.e0 = 0;
  if (z.M) {
    mirror_base(a.mir, a.bt, c, z.r0, z.e0);
    z.M += z.base;
  }
  z.Uin = a.bt.cube_case ? a.bt.cases[a.bt.cube_case[c]].Uin : a.Uin;
  bool wrote = false;
  auto order = [&]() {  // after the passes so far (uniform over the cluster)
    if (wrote) {
      if (size == 1) __syncthreads(); else cl.sync();
    }
    wrote = true;
  };
#pragma unroll 1
  for (int r = 0; r < 2; ++r) {
    if (r == 1 && a.axes && (flags & 63)) {
      order();
      bc_fill(a, z, flags, a.cover ? flags >> kLayerCover : 0, first, stride);
    }
    const int *off = r ? a.off[1] : a.off[0];
    if (off && off[c + 1] > off[c]) {
      order();
      const FaceTask *tasks = r ? a.tasks[1] : a.tasks[0];
      for (int t = off[c] + rank; t < off[c + 1]; t += size) {
        const FaceTask ft = tasks[t];
        if (ft.kind == 0) face_copy(a, z, ft); else level_face(a, z, ft);
      }
    }
    const int e = r ? a.edges[1] : a.edges[0];
    if (e == 1 || (e == 2 && (flags & kLayerEdge))) {
      order();
      edge_fill(a, z, first, stride);
    }
  }
}

cudaError_t launch_layers(const LayerArgs &a, int ncubes, cudaStream_t s) {
  if (ncubes <= 0) return cudaSuccess;
  // Four CTAs a cube while that leaves the chip room, else two (a step's stage,
  // us, by clusters of 1, 2 and 4: 8 cubes of 8^3 31.4 29.6 26.8, 64 of 16^3 in
  // FP64 535 528 525, 216 of 24^3 473 467 467, 216 of 12^3 87.9 84.9 87.2, 512
  // of 24^3 1026 1020 1024, 2,744 of 16^3 1516 1523 1541).
  const int size = ncubes <= 64 || (ncubes <= 304 && a.n >= 16) ? 4 : 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ncubes * size);
  cfg.blockDim = dim3(kLayerThreads);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = size;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_layers, a);
}

// ---------------------------------------------------------------------------
// IBM ghost cells (BCM_Ghostcell_minus.cpp:72-489; _plus is identical).  The
// host orders the entries in dependency levels: within a level no entry reads
// a cell another entry of the level writes, and every read sees exactly the
// value the reference's serial loop sees.  A CTA runs the levels of one group
// of entries, a barrier between them; groups share no cube.  A sphere of
// 2,792 entries in 32 cubes takes 21 levels, the later ones of some 40
// entries: launches of a level each took 230 us (under ncu; 21 x 10.9), the
// group's levels 74.  A stage of a step of that sphere among 416 cubes of 16^3,
// split: 490 -> 374 us, among 92 cubes in FP64: 1057 -> 952.
//
// Eight lanes per entry, one stencil cell each, the next entry's indices and
// weights loaded ahead.  The FP64 pipe (73 cycles an instruction of a warp)
// bounds a level's chain: the cells' divisions go to the integer pipes, each
// lane forms its cell's weighted terms, and lanes 0..4 sum one quantity each
// in the reference's order (000,100,010,001,110,101,011,111) and form one
// component of the ghost cell each: 34 FP64 instructions in a row.
// ---------------------------------------------------------------------------
__device__ __noinline__ double ghost_quotient(double x, double y) { return x / y; }

constexpr int kGhostThreads = 8 * kGhostPer;

__global__ void __launch_bounds__(kGhostThreads) k_ghost(GhostArgs a) {
  // per entry: the stencil cells' weighted terms, the results; of a ghost
  // inside its own stencil that cell's density and pressure
  __shared__ double term[kGhostPer][8][5], val[kGhostPer][5], raw[kGhostPer][2];
  const int g = threadIdx.x >> 3, m = threadIdx.x & 7;
  const int S = a.n + 4;
  // cell m of the stencil, order 000,100,010,001,110,101,011,111 (:81-145)
  const int oi = (m == 1 || m == 4 || m == 5 || m == 7), oj = (m == 2 || m == 4 || m == 6 || m == 7),
            ok = (m == 3 || m == 5 || m == 6 || m == 7);
  const unsigned cell = (oi * S + oj) * S + ok;
  float *const M = mirror_current(a.mir);
  int l = a.groups[blockIdx.x];
  const int l1 = a.groups[blockIdx.x + 1];
  if (l >= l1) return;
  int e0 = a.levels[l], e1 = a.levels[l + 1], e2 = l + 1 < l1 ? a.levels[l + 2] : e1;
  GhostEntry nxt;
  double wn = 0;
  auto load = [&]() {
    nxt.cube = 0;  // none
    if (e0 + g < e1) {
      nxt = a.entries[e0 + g];
      wn = a.weights[8 * (size_t)(e0 + g) + m];
      if (!case_active(a.bt, nxt.cube)) nxt.cube = 0;
    }
  };
  load();
  for (bool more = true; more;) {
    const GhostEntry e = nxt;
    const double w = wn;
    bool level_ends = false;
    e0 += kGhostPer;
    if (e0 >= e1) {
      level_ends = true;
      more = ++l < l1;
      e0 = e1;
      e1 = e2;
      if (l + 1 < l1) e2 = a.levels[l + 2];  // in time for the level after this
    }
    if (more) load();
    const bool act = e.cube != 0, self = e.self < 8;
    double rho0 = a.rho0, P0 = a.P0, ws = 0;
    IntFp os;
    Recip ks = {};
    if (act) {
      if (a.bt.cube_case) {  // the case of the stencil's cube
        const CaseConst &cq = a.bt.cases[a.bt.cube_case[e.cube]];
        rho0 = cq.rho0;
        P0 = cq.P0;
      }
      const double *q = a.U1_ + 5 * (size_t)(e.stencil + cell);
      const double rh = q[0], q1 = q[1], q2 = q[2], q3 = q[3], q4 = q[4];
      // (while the loads are on their way) the divisor of a ghost in its stencil
      if (self) {
        ws = __shfl_sync(0xffu << (threadIdx.x & 24), w, (threadIdx.x & 24) + e.self);
        ks = os.recip((m < 2 ? 1. : 2.) - ws);
      }
      IntFp o;
      const Recip k = o.recip(rh);
      double Uu = o.div(q1, k), Vv = o.div(q2, k), Ww = o.div(q3, k);
      if (!o.ok) {
        Uu = ghost_quotient(q1, rh);
        Vv = ghost_quotient(q2, rh);
        Ww = ghost_quotient(q3, rh);
      }
      const double VV = Uu * Uu + Vv * Vv + Ww * Ww;
      const double Pp = (q4 - 0.5 * rh * VV) * (BCMG_K - 1);
      double *t = term[g][m];
      t[0] = w * (rh - rho0);
      t[1] = w * (Pp - P0);
      t[2] = w * Uu;
      t[3] = w * Vv;
      t[4] = w * Ww;
      if (m == e.self) {
        double *r = raw[g];
        r[0] = rh; r[1] = Pp;
      }
    }
    __syncwarp();
    if (act && m < 5) {
      const double base = m == 0 ? rho0 : P0;
      double acc = -0.0;  // -0 + t is t
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (c != e.self) acc = acc + term[g][c][m];
      if (self) {
        if (m < 2 && ws > 0.9999) {
          acc = raw[g][m];
        } else {
          const double q = os.div(acc, ks);
          acc = os.ok ? q : ghost_quotient(acc, (m < 2 ? 1. : 2.) - ws);
          if (m < 2) acc = acc + base;
        }
      } else if (m < 2) {
        acc = acc + base;
      }
      val[g][m] = acc;
    }
    __syncwarp();
    if (act && m < 5) {
      const double rho = val[g][0], hr = 0.5 * rho;
      double o;
      if (m == 0) {
        o = rho;
      } else if (m < 4) {
        o = (self ? rho : hr) * val[g][m + 1];
      } else {
        const double P = val[g][1], U = val[g][2], V = val[g][3], W = val[g][4];
        const double VV = U * U + V * V + W * W;
        IntFp op;
        double p = op.div(P, RecipConst<__builtin_bit_cast(uint64_t, (double)(BCMG_K - 1))>::get());
        if (!op.ok) p = ghost_quotient(P, BCMG_K - 1);
        o = p + (self ? hr : hr * 0.25) * VV;
      }
      const size_t go = 5 * (size_t)e.ghost + m;
      a.U1_[go] = o;
      if (M) {
        double r0, e0_;
        mirror_base(a.mir, a.bt, e.ghost_cube, r0, e0_);
        M[go] = mirror_value(o, m, r0, e0_);
      }
    }
    if (level_ends && more) __syncthreads(); else __syncwarp();
  }
}

cudaError_t launch_ghost(const GhostArgs &a, int groups, cudaStream_t s, int priority) {
  if (groups <= 0) return cudaSuccess;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(groups);
  cfg.blockDim = dim3(kGhostThreads);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributePriority;
  at[0].val.priority = priority;
  cfg.attrs = at;
  cfg.numAttrs = priority != 0;
  return cudaLaunchKernelEx(&cfg, k_ghost, a);
}

}  // namespace bcmg
