// Split-precision LU-SGS sub-iteration: the sweeps in FP32, the update and
// norm sums in FP64.  Same scheme and parallel form as the FP64 kernels
// (bcm_lusgs.cu): coefficients first, then forward and backward sweeps over
// the planes i+j+k = const by a cluster of CTAs per cube, then the update.
// The sweep is a preconditioner of the dual-time iteration (the FP32 residual
// it is fed decides the converged state), so its coefficients come from the
// FP32 mirror of the state: deltas from the case's reference state (rho0, 0,
// 0, 0, P0/(K-1)), pressure p = P0 + p'.  The increment is added to the FP64
// state and the change norms are formed from the FP32 increments and summed
// in FP64, as in the split RK path.
//
// Plane order.  Between the kernels a cube's values lie value-major in the
// order of the sweep (the cells of plane h, i then j ascending, the rows of a
// cluster's CTAs one after the other), so the
// threads of a plane read and write consecutive words; k_lus_pack and
// k_lus_update change between that order and the memory order slab by slab
// (i fixed) through shared memory, where the cells of an anti-diagonal j + k
// of the slab are a run of the plane order.
//
// A sub-iteration less its flux stage (ms), against one kernel that packed,
// swept and updated a cube in one CTA and formed the coefficients in the chain
// of planes: 216 cubes of 24^3 0.88 -> 0.49, 8 of 24^3 0.53 -> 0.19, 512 of
// 32^3 5.20 -> 3.18, 512 of 16^3 0.53 -> 0.37, 512 of 12^3 0.29 -> 0.23, 512 of
// 8^3 0.143 -> 0.115.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "bcm_common.cuh"
#include "bcm_kernels.h"
#include "bcm_split_cell.cuh"

namespace bcmg {

namespace {

namespace cg = cooperative_groups;

// Cell coefficients U, V, W, VV, H, r_x, r_y, r_z, nu, dg from the FP32
// deltas m (rho' = m0, rho u = m1.., E' = m4).
__device__ __forceinline__ void luf_coef(const float *m, float rho0, float P0, float T0,
                                         float mu_L, float idx, float dT, float cfl,
                                         float omega, float *k) {
  const float rho = rho0 + m[0];
  const float ir = 1.0f / rho;
  const float U = m[1] * ir, V = m[2] * ir, W = m[3] * ir;
  const float VV = U * U + V * V + W * W;
  const float P = P0 + (m[4] - 0.5f * rho * VV) * 0.4f;
  const float c = sqrtf(1.4f * P * ir);
  const float H = (m[4] + 2.5f * P0 + P) * ir;
  const float r0 = fabsf(U) + c, r1 = fabsf(V) + c, r2 = fabsf(W) + c;
  const float T = P * ir * (1.0f / 287.0f);
  const float temp = T / T0;
  const float mu = mu_L * temp * sqrtf(temp) * (T0 + 110.f) / (T + 110.f);
  const float nu = mu * (float)(BCMG_K / BCMG_PR) * ir;
  const float rs = r0 + r1 + r2;
  float dg = 1.5f / dT + omega * rs * idx + 6.0f * nu * idx * idx;
  if (cfl > 0) dg += rs * idx / cfl;
  k[0] = U; k[1] = V; k[2] = W; k[3] = VV; k[4] = H;
  k[5] = r0; k[6] = r1; k[7] = r2; k[8] = nu; k[9] = dg;
}

// Off-diagonal terms of a cell (coefficients k, increment dq) for its
// neighbours across the faces of the three directions; LOWER: the A+ parts
// (forward sweep), else A-.
template <bool LOWER, typename Store>
__device__ __forceinline__ void luf_terms(const float *k, float idx, float omega, const float *dq,
                                          Store store) {
  const float U = k[0], V = k[1], W = k[2], VV = k[3], H = k[4];
#pragma unroll
  for (int D = 0; D < 3; ++D) {
    const float un = D == 0 ? U : (D == 1 ? V : W);
    const float dp =
        0.4f * (dq[4] - (U * dq[1] + V * dq[2] + W * dq[3]) + 0.5f * VV * dq[0]);
    const float t = dq[1 + D] - un * dq[0];
    float a[5];
    a[0] = dq[1 + D];
    a[1] = un * dq[1] + U * t;
    a[2] = un * dq[2] + V * t;
    a[3] = un * dq[3] + W * t;
    a[1 + D] += dp;
    a[4] = un * (dq[4] + dp) + H * t;
    const float h = 0.5f * idx, w = omega * k[5 + D], v = k[8] * idx * idx;
    float t5[5];
#pragma unroll
    for (int m = 0; m < 5; ++m)
      t5[m] = LOWER ? h * (a[m] + w * dq[m]) + v * dq[m] : h * (a[m] - w * dq[m]) - v * dq[m];
    store(D, t5);
  }
}

// Scratch of a cube: four words of four values per cell, word-major
// [kWords][n^3] in plane order: U V W VV, H r_x r_y r_z, nu dg flags R4 and R0 ..
// R3 (the residual, then the forward sweep's increment).  Flags: bit 0 fluid;
// bits 1..3 the lower x, y, z neighbour inside the cube is fluid, bits 4..6 the
// upper; i, j, k from bits 7, 12 and 17.
constexpr int kWords = 4;

// Position of the first cell of row i in plane h, and the row's first j.
__device__ __forceinline__ int jlo_of(int h, int i, int n) {
  const int x = h - i - (n - 1);
  return x > 0 ? x : 0;
}
// cells of planes 0 .. h-1
__device__ __forceinline__ int plane_start(int h, int n) {
  // planes up to n-1 are triangles, the last n-1 too, between them the cube's
  // count less both
  auto tet = [](int x) { return x * (x + 1) * (x + 2) / 6; };  // sum of x triangles
  int c = tet(h);
  if (h > n) c -= 3 * tet(h - n);
  if (h > 2 * n) c += 3 * tet(h - 2 * n);
  return c;
}
__device__ __forceinline__ int row_cells(int h, int i, int n) {
  const int lo = jlo_of(h, i, n), hi = min(n - 1, h - i);
  return hi >= lo ? hi - lo + 1 : 0;
}
// cells of plane h ahead of row i: of its CTA's rows (i mod size alike) the
// lower ones, and all of the CTAs before
__device__ __forceinline__ int row_start(int h, int i, int n, int size) {
  int c = 0;
  for (int r = 0; r <= i % size; ++r)
    for (int l = r; l < (r < i % size ? n : i); l += size) c += row_cells(h, l, n);
  return c;
}

// Cell t of a slab in anti-diagonal order: d = j + k ascending, then j.
__device__ __forceinline__ void slab_cell(const unsigned short *start, int n, int t, int &j,
                                          int &k) {
  int lo = 0, hi = 2 * n - 1;  // the last diagonal that starts at or before t
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (start[mid] <= t) lo = mid; else hi = mid;
  }
  j = max(0, lo - (n - 1)) + t - start[lo];
  k = lo - j;
}
__device__ __forceinline__ void slab_starts(unsigned short *start, int n) {
  for (int d = threadIdx.x; d < 2 * n - 1; d += blockDim.x)
    start[d] = (unsigned short)(d <= n ? d * (d + 1) / 2
                                       : n * n - (2 * n - 1 - d) * (2 * n - d) / 2);
}

// The constants of a cube's case.
struct LusConst {
  float dT, mu_L, rho0, P0, T0;
  double rho0d, E0d;  // mirror reference state (FP64)
};
__device__ __forceinline__ LusConst lus_const(const LusgsSplitArgs &a, int cube) {
  LusConst z = {a.dTf, a.mu_Lf, a.rho0f, a.P0f, a.T0f, a.mir.rho0, a.mir.E0};
  if (a.bt.cube_case) {
    const CaseConst *q = a.bt.cases + a.bt.cube_case[cube];
    z = {q->dTf, q->mu_Lf, q->rho0f, q->P0f, q->T0f, q->rho0, q->E0};
  }
  return z;
}

// One slab (cube, i) per CTA: coefficients, residual and flags into plane
// order.  (The mirror is read here and updated in k_lus_update: its interior
// cells belong to one cube each.)
// NT threads: a compile-time stride, so that the loads of several turns are in
// flight (run-time strides made a step of 216 cubes of 24^3 4.7% slower).
template <int NT>
__global__ void __launch_bounds__(NT) k_lus_pack(LusgsSplitArgs a, int size) {
  extern __shared__ float4 stage[];  // [kWords][n^2]
  __shared__ unsigned short start[64];
  __shared__ int place[64];  // of the slab's cells of anti-diagonal d
  const int n = a.ph.n, S = n + 4, nn = n * n;
  const int cube = 1 + blockIdx.x / n, i = blockIdx.x % n;
  if (!case_active(a.bt, cube)) return;  // converged case
  const LusConst z = lus_const(a, cube);
  const float idx = a.inv_dx[cube];
  const float *const Mc = mirror_current(a.mir);
  slab_starts(start, n);
  for (int d = threadIdx.x; d < 2 * n - 1; d += NT)
    place[d] = plane_start(i + d, n) + row_start(i + d, i, n, size) - jlo_of(i + d, i, n);
  for (int jk = threadIdx.x; jk < nn; jk += NT) {
    const int j = jk / n, k = jk - j * n;
    const size_t o = cell_index(S, cube, i + 2, j + 2, k + 2);
    float m[5], kc[10];
#pragma unroll
    for (int v = 0; v < 5; ++v) m[v] = Mc[5 * o + v];
    luf_coef(m, z.rho0, z.P0, z.T0, z.mu_L, idx, z.dT, a.cflf, a.omegaf, kc);
    float R[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) R[v] = a.R32[5 * o + v];
    const int *F = a.FWS + o;
    int f = F[0] == kFluid ? 1 : 0;
    if (i > 0 && F[-S * S] == kFluid) f |= 2;
    if (j > 0 && F[-S] == kFluid) f |= 4;
    if (k > 0 && F[-1] == kFluid) f |= 8;
    if (i + 1 < n && F[S * S] == kFluid) f |= 16;
    if (j + 1 < n && F[S] == kFluid) f |= 32;
    if (k + 1 < n && F[1] == kFluid) f |= 64;
    f |= i << 7 | j << 12 | k << 17;
    stage[jk] = make_float4(kc[0], kc[1], kc[2], kc[3]);
    stage[nn + jk] = make_float4(kc[4], kc[5], kc[6], kc[7]);
    stage[2 * nn + jk] = make_float4(kc[8], kc[9], __int_as_float(f), R[4]);
    stage[3 * nn + jk] = make_float4(R[0], R[1], R[2], R[3]);
  }
  __syncthreads();
  float4 *const scr = reinterpret_cast<float4 *>(a.scr) + (size_t)(cube - 1) * kWords * nn * n;
  for (int t = threadIdx.x; t < nn; t += NT) {
    int j, k;
    slab_cell(start, n, t, j, k);
    float4 *dst = scr + place[j + k] + j;
#pragma unroll
    for (int v = 0; v < kWords; ++v) dst[(size_t)v * nn * n] = stage[v * nn + j * n + k];
  }
}

// Shared memory of a sweeping CTA: the terms its cells add, [2 planes][3
// directions][rows * n] of the first four and after them the fifth, then the
// place of its part of each plane and its size.
__host__ __device__ inline int lus_rows(int n, int size) { return (n + size - 1) / size; }
__host__ __device__ inline size_t lus_smem(int n, int size) {
  return sizeof(float) * 30 * lus_rows(n, size) * n + 2 * sizeof(int) * (3 * n - 2);
}

// Two CTAs on an SM hide each other's barriers (65536 registers / 896).
constexpr int kSweepThreads = 448;

// A cell is moved by 16-byte words throughout: four loads and six reads and six
// writes of shared memory, where single values took 16, 15 and 15, each with
// its address, and its place comes from its flags, where a search of the row
// tables took a third of a plane's instructions: 216 cubes of 24^3 325 ->
// 247 us.
struct LusCell {
  float4 w[kWords];
  int pos;  // < 0: none
};

template <bool LOWER, int SIZE>
__device__ __forceinline__ void lus_sweep(const LusgsSplitArgs &a, cg::cluster_group cl,
                                          float4 *slots, const int *place, const int *cells,
                                          float4 *scr, float *inc, float idx) {
  const int n = a.ph.n, S = n + 4, n3 = n * n * n, np = 3 * n - 2;
  const int rank = SIZE == 1 ? 0 : (int)cl.block_rank();
  const int cols = lus_rows(n, SIZE) * n;
  float *const fifth = reinterpret_cast<float *>(slots + 6 * cols);
  auto load = [&](int p, int t, LusCell &z) {
    z.pos = -1;
    if (p < 0 || p >= np || t >= cells[p]) return;
    z.pos = place[p] + t;
#pragma unroll
    for (int v = 0; v < kWords; ++v) z.w[v] = scr[z.pos + (size_t)v * n3];
  };
  auto cell = [&](int p, const LusCell &z) {
    const int fl = __float_as_int(z.w[2].z);
    if (z.pos < 0 || !(fl & 1)) return;
    const int i = fl >> 7 & 31, j = fl >> 12 & 31, k = fl >> 17 & 31;
    const int col = (i / SIZE) * n + j, in = (p & 1) * 3 * cols;
    const int nb = LOWER ? fl >> 1 : fl >> 4;
    const float r[5] = {z.w[3].x, z.w[3].y, z.w[3].z, z.w[3].w, z.w[2].w};
    float s[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) s[m] = LOWER ? r[m] : 0.f;
#pragma unroll
    for (int D = 0; D < 3; ++D)
      if (nb & (1 << D)) {
        const float4 x = slots[in + D * cols + col];
        s[0] += x.x; s[1] += x.y; s[2] += x.z; s[3] += x.w;
        s[4] += fifth[in + D * cols + col];
      }
    const float c[10] = {z.w[0].x, z.w[0].y, z.w[0].z, z.w[0].w, z.w[1].x,
                         z.w[1].y, z.w[1].z, z.w[1].w, z.w[2].x, z.w[2].y};
    const float idg = 1.0f / c[9];
    float dq[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) dq[m] = LOWER ? s[m] * idg : r[m] - s[m] * idg;
    if (LOWER) {
      scr[z.pos + (size_t)3 * n3] = make_float4(dq[0], dq[1], dq[2], dq[3]);
      scr[z.pos + (size_t)2 * n3].w = dq[4];
    } else {
      float *q = inc + 5 * (((i + 2) * S + (j + 2)) * S + k + 2);
#pragma unroll
      for (int m = 0; m < 5; ++m) q[m] = dq[m];
    }
    const int d = LOWER ? 1 : -1, out = ((p + d) & 1) * 3 * cols;
    const bool wi = LOWER ? i + 1 < n : i > 0, wj = LOWER ? j + 1 < n : j > 0,
               wk = LOWER ? k + 1 < n : k > 0;
    luf_terms<LOWER>(c, idx, a.omegaf, dq, [&](int D, const float *x) {
      if (!(D == 0 ? wi : (D == 1 ? wj : wk))) return;
      const int at = out + D * cols + (D == 0 ? ((i + d) / SIZE) * n + j : (D == 1 ? col + d : col));
      float4 *q = slots + at;
      float *f = fifth + at;
      if (SIZE > 1 && D == 0) {
        q = cl.map_shared_rank(q, (rank + d + SIZE) % SIZE);
        f = cl.map_shared_rank(f, (rank + d + SIZE) % SIZE);
      }
      *q = make_float4(x[0], x[1], x[2], x[3]);
      *f = x[4];
    });
  };
  LusCell cur, nxt;
  const int p0 = LOWER ? 0 : np - 1, d = LOWER ? 1 : -1;
  load(p0, threadIdx.x, nxt);
  for (int s = 0, p = p0; s < np; ++s, p += d) {
    cur = nxt;
    load(p + d, threadIdx.x, nxt);
    // Clusters have fewer warps an SM to hide the loads: the plane after next
    // starts towards L2 (512 cubes of 32^3 3.31 -> 3.25 ms of a sub-iteration;
    // a CTA a cube, 8 of 24^3: 0.187 -> 0.204, so not there).
    if (SIZE > 1) {
      const int q = p + 2 * d;
      if (q >= 0 && q < np && threadIdx.x < cells[q]) {
#pragma unroll
        for (int v = 0; v < kWords; ++v) prefetch_l2(scr + place[q] + threadIdx.x + (size_t)v * n3);
      }
    }
    // (one copy of the cell's code: two may contract their products unlike)
#pragma unroll 1
    for (int t = threadIdx.x;;) {
      cell(p, cur);
      t += blockDim.x;
      if (t >= cells[p]) break;
      load(p, t, cur);
    }
    if (SIZE == 1) __syncthreads(); else cl.sync();
  }
}

template <int SIZE>
__global__ void __launch_bounds__(kSweepThreads, 2) k_lus_sweep(LusgsSplitArgs a) {
  extern __shared__ float4 slots[];
  const cg::cluster_group cl = cg::this_cluster();
  const int n = a.ph.n, np = 3 * n - 2;
  const int rank = SIZE == 1 ? 0 : (int)cl.block_rank();
  const int cube = 1 + blockIdx.x / SIZE;
  if (!case_active(a.bt, cube)) return;  // converged case (the whole cluster)
  int *place = reinterpret_cast<int *>(reinterpret_cast<float *>(slots) +
                                       30 * lus_rows(n, SIZE) * n);
  int *cells = place + np;
  for (int p = threadIdx.x; p < np; p += blockDim.x) {
    int sum = 0;
    for (int i = rank; i < n; i += SIZE) sum += row_cells(p, i, n);
    place[p] = plane_start(p, n) + row_start(p, rank, n, SIZE);
    cells[p] = sum;
  }
  // every CTA of the cluster has started before any writes into its memory
  if (SIZE == 1) __syncthreads(); else cl.sync();
  float4 *const scr = reinterpret_cast<float4 *>(a.scr) + (size_t)(cube - 1) * kWords * n * n * n;
  float *const inc = a.R32 + 5 * cell_index(n + 4, cube, 0, 0, 0);
  const float idx = a.inv_dx[cube];
  // dq* = (R + sum of lower A+ terms) / dg, then dq = dq* - (sum of upper A-
  // terms) / dg
  lus_sweep<true, SIZE>(a, cl, slots, place, cells, scr, inc, idx);
  lus_sweep<false, SIZE>(a, cl, slots, place, cells, scr, inc, idx);
}

// Q += dq on fluid cells (FP64), one slab (i fixed) per CTA; change norms of
// p, u, v, w, T from the FP32 increment (the split RK path's third-stage
// formulas) and the force integrands of the non-fluid cells (fluid cells
// have none).  The FP64 pipe bounds it (12 additions per cell and the warps'
// sums), so the conversions go to the integer pipes: 216 cubes of 24^3
// 232 -> 170 us, with four CTAs of 64 registers an SM 165.
struct LusState {
  size_t o;
  bool fluid;
  double u[5];
  float m[5], dq[5];
};

constexpr int kUpdThreads = 256;

__global__ void __launch_bounds__(kUpdThreads, 4) k_lus_update(LusgsSplitArgs a) {
  __shared__ double red[kUpdThreads / 32][7];
  const int n = a.ph.n, S = n + 4, nn = n * n, NT = blockDim.x, tid = threadIdx.x;
  const int cube = 1 + blockIdx.x / n, i = blockIdx.x % n;
  if (!case_active(a.bt, cube)) return;  // converged case
  const LusConst z = lus_const(a, cube);
  // The mirror of the state is updated in place with it: this block writes
  // its own cells of it and (same-level pushes) other cubes' ghost cells,
  // which no block of this launch reads.
  float *const Mc = mirror_current(a.mir);
  auto load = [&](int jk, LusState &s) {
    if (jk >= nn) return;
    const int j = jk / n, k = jk - j * n;
    s.o = cell_index(S, cube, i + 2, j + 2, k + 2);
    s.fluid = a.FWS[s.o] == kFluid;
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      s.u[v] = a.U1_[5 * s.o + v];
      s.m[v] = Mc[5 * s.o + v];
      s.dq[v] = a.R32[5 * s.o + v];
    }
  };
  LusState s;
  double e[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int jk = tid; jk < nn; jk += NT) {
    load(jk, s);
    if (!s.fluid) {
      e[5] += a.Residual1[5 * s.o + 0];
      e[6] += a.Residual1[5 * s.o + 1];
      continue;
    }
    const int j = jk / n, k = jk - j * n;
    const float *const dq = s.dq;
    const float rf = z.rho0 + s.m[0];
    const float m1 = s.m[1], m2 = s.m[2], m3 = s.m[3];
    const float mm = m1 * m1 + m2 * m2 + m3 * m3;
    const float Pc = z.P0 + (s.m[4] - 0.5f * mm / rf) * 0.4f;
    double un[5];
    float mn[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      un[v] = s.u[v] + to_double_int(dq[v]);
      a.U1_[5 * s.o + v] = un[v];
      mn[v] = to_float_int(v == 0 ? un[v] - z.rho0d : (v == 4 ? un[v] - z.E0d : un[v]));
      Mc[5 * s.o + v] = mn[v];
    }
    // Same-level interface copy of this cell (state and mirror), done
    // here: no block reads another cube's cells during the sweep.
    if (a.push && (i < 2 || i >= n - 2 || j < 2 || j >= n - 2 || k < 2 || k >= n - 2)) {
      push_same_level(a.U1_, a.push, n, cube, i + 2, j + 2, k + 2, un);
      push_same_level(Mc, a.push, n, cube, i + 2, j + 2, k + 2, mn);
    }
    const float dr = dq[0], e1 = dq[1], e2 = dq[2], e3 = dq[3], dE = dq[4];
    const float den = 1.0f / (rf * (rf + dr));
    const float dU = (e1 * rf - m1 * dr) * den;
    const float dVv = (e2 * rf - m2 * dr) * den;
    const float dW = (e3 * rf - m3 * dr) * den;
    const float dKE =
        0.5f * ((2.f * (m1 * e1 + m2 * e2 + m3 * e3) + e1 * e1 + e2 * e2 + e3 * e3) * rf - mm * dr) * den;
    const float dP = 0.4f * (dE - dKE);
    const float dTt = (dP * rf - Pc * dr) * den;
    e[0] += to_double_int(dP * dP);
    e[1] += to_double_int(dU * dU);
    e[2] += to_double_int(dVv * dVv);
    e[3] += to_double_int(dW * dW);
    e[4] += to_double_int(dTt * dTt);
  }
  const int m = norm_exchange(e, tid & 31);
  if ((tid & 31) < 8 && m < 7) red[tid >> 5][m] = e[0];
  __syncthreads();
  if (tid < 7) {
    double x = 0;
    for (int w = 0; w < NT / 32; ++w) x += red[w][tid];
    a.partials[(size_t)blockIdx.x * 7 + tid] = x;
  }
}

// The most cells of a plane in one CTA of a cluster.
int lus_plane_cells(int n, int size) {
  int most = 0;
  for (int p = 0; p <= 3 * n - 3; ++p)
    for (int r = 0; r < size; ++r) {
      int c = 0;
      for (int i = r; i < n; i += size) {
        const int lo = std::max(0, p - i - (n - 1)), hi = std::min(n - 1, p - i);
        if (hi >= lo) c += hi - lo + 1;
      }
      most = std::max(most, c);
    }
  return most;
}

}  // namespace

int lusgs_split_blocks(int n) { return n; }
int lusgs_split_launches() { return 3; }

// CTAs that sweep a cube.
static int lus_size(int n) { return lus_plane_cells(n, 1) <= kSweepThreads ? 1 : 4; }

// Threads for the widest plane of a cube, and of a sweeping CTA, in whole warps.
int lusgs_split_most_threads(int n) { return (lus_plane_cells(n, 1) + 31) / 32 * 32; }
int lusgs_split_plane_threads(int n) {
  return (lus_plane_cells(n, lus_size(n)) + 31) / 32 * 32;
}

cudaError_t launch_lusgs_split(const LusgsSplitArgs &a, int ncubes, cudaStream_t s) {
  if (ncubes <= 0) return cudaSuccess;
  const int n = a.ph.n, nn = n * n;
  if (nn > 1024) return cudaErrorInvalidValue;
  if (a.threads > 0 && (a.threads % 32 != 0 || a.threads > lusgs_split_most_threads(n)))
    return cudaErrorInvalidValue;
  cudaError_t e;
  // A thread a cell of a slab, up to 256 (256 whatever the slab took 25 us more for
  // 4,096 cubes of 4^3, 36 for 1,728 of 8^3).
  const auto pack = nn <= 32 ? k_lus_pack<32> : nn <= 64 ? k_lus_pack<64>
                  : nn <= 160 ? k_lus_pack<160> : k_lus_pack<256>;
  const int pack_threads = nn <= 32 ? 32 : nn <= 64 ? 64 : nn <= 160 ? 160 : 256;
  e = cudaFuncSetAttribute(pack, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)sizeof(float4) * kWords * 1024);  // the largest edge's
  if (e != cudaSuccess) return e;
  // One CTA per cube while the widest plane fits it (up to edge 24): the planes
  // are a chain, and a barrier of the CTA is cheaper than one of a cluster (216
  // cubes of 24^3, the rest of a sub-iteration as above, before the words of 16
  // bytes: 0.63 ms, by clusters of two 0.69; 8 cubes 0.29 and 0.30).  Wider
  // planes go to clusters of four: 64 cubes of 32^3 0.62 ms, by one CTA of 768
  // threads 0.74; now by clusters of two, four and eight 0.58, 0.56 and 0.58.
  const int size = lus_size(n);
  pack<<<ncubes * n, pack_threads, sizeof(float4) * kWords * nn, s>>>(a, size);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  int threads = lusgs_split_plane_threads(n);
  if (a.threads > 0) threads = std::min(threads, a.threads);  // wide planes take several passes
  const size_t smem = lus_smem(n, size);
  const auto sweep = size == 1 ? k_lus_sweep<1> : k_lus_sweep<4>;
  e = cudaFuncSetAttribute(sweep, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ncubes * size);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = size;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = size > 1;  // (clusters of one start slowly: 4,096 cubes of 4^3 66 us, now 34)
  if ((e = cudaLaunchKernelEx(&cfg, sweep, a)) != cudaSuccess) return e;
  // Three cells per thread or so, six of large slabs: a warp's norm sums take 9
  // FP64 additions a turn on top of the 12 of each cell (n = 16, three and six:
  // 0.369 and 0.379 ms of a sub-iteration of 512 cubes; n = 24 0.503 and 0.494;
  // n = 32 3.22 and 3.18).
  const int ut = std::min(kUpdThreads, (nn / (n < 24 ? 3 : 6) + 31) / 32 * 32);
  k_lus_update<<<ncubes * n, ut, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace bcmg
