// LU-SGS dual-time sub-iteration (FP64).  No counterpart in the reference:
// BCM_LUSGS.h only re-declares an older BCM_Interface.  The scheme is a
// matrix-free lower-upper symmetric Gauss-Seidel step for the same discrete
// residual as the RK path (BDF2 source + inviscid + viscous), with the
// Jameson-Turkel split Jacobians A+- = (A +- omega r I)/2 (r = |u_d| + c), a
// scalar viscous term nu = mu K/(Pr rho) and an optional local pseudo-time
// term (cfl > 0).  Per cube, cube faces and non-fluid cells carry no
// increment (block Jacobi across cubes, like the interface treats cubes).
//
// Parallel form.  A cell's forward value needs only its three lower
// neighbours (i-1, j-1, k-1) and its backward value only its three upper
// neighbours, so every plane i+j+k = h of a cube is independent.  What the
// planes' chain does not need is kept out of it:
//  * k_lu_coef forms every cell's coefficients (they depend on the state
//    only) in one pass over all cells;
//  * k_lu_sweep walks the planes.  A cell that has its increment forms the
//    three off-diagonal terms its neighbours of the next plane will add (they
//    share the pressure and viscous parts) and stores each where that
//    neighbour reads it, so a cell adds three vectors and divides.  The
//    cells of a plane go to consecutive threads; the next plane's
//    coefficients are loaded a plane ahead.  A cube is swept by a cluster of
//    CTAs (row i by CTA i mod size; only the i terms cross CTAs, through
//    distributed shared memory, with one cluster barrier per plane), since
//    few cubes would leave most of the FP64 pipes idle;
//  * k_lu_update applies Q += dq and sums the change norms of p, u, v, w, T
//    and the force integrands per cube, like the RK path's third stage
//    (BCM_Flux_XYZ_Viscous_Runge_kutta.cpp:2530-2650).
// Divisions and roots run on the integer pipes (bcm_fp64_int.cuh); products
// stay on the FP64 pipe (a plane is a few warps: the integer sequences'
// latency made the sweep 15-20% slower).  64 cubes of 24^3: 5.3 -> 1.29 ms for
// the three kernels (the sweep 1.09 ms, 7.8 us a plane: bound by the FP64
// pipe's throughput and latency over the chain of 2 x 70 planes).  Every cell's arithmetic is the same as the serial
// lexicographic sweep's, so the result is bit-identical to it (built with
// --fmad=false).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "bcm_common.cuh"
#include "bcm_fp64_int.cuh"
#include "bcm_kernels.h"

namespace bcmg {

namespace {

namespace cg = cooperative_groups;

constexpr int kLuThreads = 512;

// The constants of a cube's case.
struct LuConst {
  double dT, mu_L, T0, dx;
};
__device__ __forceinline__ LuConst lu_const(const LusgsArgs &a, int cube) {
  double dT = a.dT, mu_L = a.ph.mu_L, rho0 = a.ph.rho0, P0 = a.ph.P0;
  if (a.bt.cube_case) {
    const CaseConst *q = a.bt.cases + a.bt.cube_case[cube];
    dT = q->dT; mu_L = q->mu_L; rho0 = q->rho0; P0 = q->P0;
  }
  return {dT, mu_L, P0 / rho0 / BCMG_R, a.cube_size[cube] / a.ph.n};
}

// The FP64 pipe's own division and root, in IntFp's form.
struct PipeFp {
  __device__ static double recip(double b) { return b; }
  __device__ static double div(double a, double b) { return a / b; }
  __device__ static double root(double x) { return sqrt(x); }
};

// Cell coefficients: U, V, W, VV, H, then omega r_x, omega r_y, omega r_z,
// nu / dx^2 and the diagonal.
template <typename Fp>
__device__ __forceinline__ void lu_coef(Fp &f, const double *q, const LuConst &z, double cfl,
                                        double omega, double *k) {
  const double rho = q[0];
  const auto kr = f.recip(rho);
  const double U = f.div(q[1], kr), V = f.div(q[2], kr), W = f.div(q[3], kr);
  const double VV = U * U + V * V + W * W;
  const double P = (q[4] - 0.5 * rho * VV) * (BCMG_K - 1);
  const double c = f.root(f.div(BCMG_K * P, kr));
  const double H = f.div(q[4] + P, kr);
  const double r0 = fabs(U) + c, r1 = fabs(V) + c, r2 = fabs(W) + c;
  const double T = f.div(f.div(P, kr), f.recip((double)BCMG_R));
  const double temp = f.div(T, f.recip(z.T0));
  const double mu = f.div(z.mu_L * temp * f.root(temp) * (z.T0 + 110.), f.recip(T + 110.));
  const double nu = f.div(mu * (BCMG_K / BCMG_PR), kr);
  const double rs = r0 + r1 + r2;
  const auto kx = f.recip(z.dx), kx2 = f.recip(z.dx * z.dx);
  double dg = f.div(1.5, f.recip(z.dT)) + f.div(omega * rs, kx) + f.div(6.0 * nu, kx2);
  if (cfl > 0) dg = dg + f.div(rs, f.recip(cfl * z.dx));
  k[0] = U; k[1] = V; k[2] = W; k[3] = VV; k[4] = H;
  k[5] = omega * r0; k[6] = omega * r1; k[7] = omega * r2; k[8] = f.div(nu, kx2); k[9] = dg;
}

__device__ __noinline__ void lu_coef_ref(const double *q, const LuConst &z, double cfl,
                                         double omega, double *k) {
  PipeFp f;
  lu_coef(f, q, z, cfl, omega, k);
}

constexpr int kCoefThreads = 256;

__global__ void __launch_bounds__(kCoefThreads) k_lu_coef(LusgsArgs a) {
  const int n = a.ph.n, S = n + 4, nn = n * n;
  const int blocks = (nn * n + kCoefThreads - 1) / kCoefThreads;  // of a cube
  const int cube = 1 + blockIdx.x / blocks;
  if (!case_active(a.bt, cube)) return;  // converged case
  const int r = (blockIdx.x % blocks) * kCoefThreads + threadIdx.x;
  if (r >= nn * n) return;
  const size_t o = cell_index(S, cube, 2 + r / nn, 2 + (r / n) % n, 2 + r % n);
  if (a.FWS[o] != kFluid) return;
  const LuConst z = lu_const(a, cube);
  double q[5], k[10];
#pragma unroll
  for (int m = 0; m < 5; ++m) q[m] = a.U1_[5 * o + m];
  IntFp f;
  lu_coef(f, q, z, a.cfl, a.omega, k);
  if (!f.ok) {
    double qr[5], kk[10];
    for (int m = 0; m < 5; ++m) qr[m] = q[m];
    const LuConst zr = z;
    lu_coef_ref(qr, zr, a.cfl, a.omega, kk);
    for (int m = 0; m < 10; ++m) k[m] = kk[m];
  }
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    a.coefA[5 * o + m] = k[m];
    a.coefB[5 * o + m] = k[5 + m];
  }
}

// Off-diagonal terms of a cell (coefficients k, increment dq) for its
// neighbours across the faces of the three directions; LOWER: the A+ parts
// (forward sweep), else A-.  h is 0.5 / dx.
template <bool LOWER, typename Store>
__device__ __forceinline__ void lu_terms(const double *k, double h, const double *dq,
                                         Store store) {
  const double U = k[0], V = k[1], W = k[2], VV = k[3], H = k[4];
  const double dp = (BCMG_K - 1) * fma64(0.5, VV * dq[0], dq[4] - (U * dq[1] + V * dq[2] + W * dq[3]));
  const double e = dq[4] + dp;
  double v[5];
#pragma unroll
  for (int m = 0; m < 5; ++m) v[m] = k[8] * dq[m];
#pragma unroll
  for (int D = 0; D < 3; ++D) {
    const double un = D == 0 ? U : (D == 1 ? V : W);
    const double t = dq[1 + D] - un * dq[0];
    double a[5];
    a[0] = dq[1 + D];
    a[1] = un * dq[1] + U * t;
    a[2] = un * dq[2] + V * t;
    a[3] = un * dq[3] + W * t;
    a[1 + D] = a[1 + D] + dp;
    a[4] = un * e + H * t;
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      const double w = k[5 + D] * dq[m];
      store(D, m, LOWER ? h * (a[m] + w) + v[m] : h * (a[m] - w) - v[m]);
    }
  }
}

// Rows of a plane that a CTA of the cluster sweeps, and a cell of a plane.
struct LuCell {
  int i, j, k;  // k < 0: none
  size_t o;
  int fl;       // bit 0 fluid, bits 1..3 the neighbour this sweep adds is fluid
  double r[5], c[10];
};

// Shared memory of a CTA: the terms its cells add, value-major
// [2 planes][3 directions][5][rows * n], and per plane the first cell of each
// of its rows.
__host__ __device__ inline int lu_rows(int n, int size) { return (n + size - 1) / size; }
__host__ __device__ inline size_t lu_smem(int n, int size) {
  const size_t rows = lu_rows(n, size);
  return 30 * sizeof(double) * rows * n + sizeof(unsigned short) * (3 * n - 2) * (rows + 1);
}

template <bool LOWER>
__device__ __forceinline__ void lu_sweep(const LusgsArgs &a, cg::cluster_group cl, double *slots,
                                         const unsigned short *first, int cube, double h) {
  const int n = a.ph.n, S = n + 4, np = 3 * n - 2;
  const int size = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int rows = lu_rows(n, size), cols = rows * n;
  const size_t cb = cell_index(S, cube, 0, 0, 0);
  const int *F = a.FWS;
  const int si = S * S, sj = S;
  // cell t of the CTA's part of plane p (i + j + k)
  auto load = [&](int p, int t, LuCell &z) {
    z.k = -1;
    const unsigned short *f = first + p * (rows + 1);
    if (p < 0 || p >= np || t >= f[rows]) return;
    int lo = 0, hi = rows;  // the last row that starts at or before t
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (f[mid] <= t) lo = mid; else hi = mid;
    }
    z.i = lo * size + rank;
    z.j = max(0, p - z.i - (n - 1)) + t - f[lo];
    z.k = p - z.i - z.j;
    z.o = cb + ((size_t)(z.i + 2) * S + (z.j + 2)) * S + (z.k + 2);
    const int d = LOWER ? -1 : 1;
    z.fl = F[z.o] == kFluid ? 1 : 0;
    if (LOWER ? z.i > 0 : z.i + 1 < n) z.fl |= F[(ptrdiff_t)z.o + d * si] == kFluid ? 2 : 0;
    if (LOWER ? z.j > 0 : z.j + 1 < n) z.fl |= F[(ptrdiff_t)z.o + d * sj] == kFluid ? 4 : 0;
    if (LOWER ? z.k > 0 : z.k + 1 < n) z.fl |= F[(ptrdiff_t)z.o + d] == kFluid ? 8 : 0;
    if (z.fl & 1) {
#pragma unroll
      for (int m = 0; m < 5; ++m) {
        z.r[m] = a.Rku1[5 * z.o + m];
        z.c[m] = a.coefA[5 * z.o + m];
        z.c[5 + m] = a.coefB[5 * z.o + m];
      }
    }
  };
  auto cell = [&](int p, const LuCell &z) {
    if (z.k < 0 || !(z.fl & 1)) return;
    const int col = (z.i / size) * n + z.j;
    const double *in = slots + (p & 1) * 15 * cols + col;
    double s[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) s[m] = LOWER ? z.r[m] : 0;
#pragma unroll
    for (int D = 0; D < 3; ++D)
      if (z.fl & (2 << D)) {
#pragma unroll
        for (int m = 0; m < 5; ++m) s[m] = s[m] + in[(5 * D + m) * cols];
      }
    IntFp f;
    const Recip kd = f.recip(z.c[9]);
    double dq[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) dq[m] = f.div(s[m], kd);
    if (!f.ok) {
#pragma unroll
      for (int m = 0; m < 5; ++m) dq[m] = s[m] / z.c[9];
    }
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      if (!LOWER) dq[m] = z.r[m] - dq[m];
      a.Rku1[5 * z.o + m] = dq[m];
    }
    const int d = LOWER ? 1 : -1;
    const bool wi = LOWER ? z.i + 1 < n : z.i > 0, wj = LOWER ? z.j + 1 < n : z.j > 0,
               wk = LOWER ? z.k + 1 < n : z.k > 0;
    double *const out = slots + ((p + d) & 1) * 15 * cols;
    double *oi = out;
    if (wi) oi = size == 1 ? out : cl.map_shared_rank(out, (z.i + d) % size);
    oi += wi ? ((z.i + d) / size) * n + z.j : 0;
    lu_terms<LOWER>(z.c, h, dq, [&](int D, int m, double x) {
      if (D == 0) { if (wi) oi[m * cols] = x; }
      else if (D == 1) { if (wj) out[(5 + m) * cols + col + d] = x; }
      else { if (wk) out[(10 + m) * cols + col] = x; }
    });
  };
  LuCell cur, nxt;
  const int p0 = LOWER ? 0 : np - 1, d = LOWER ? 1 : -1;
  load(p0, threadIdx.x, nxt);
  for (int s = 0, p = p0; s < np; ++s, p += d) {
    cur = nxt;
    load(p + d, threadIdx.x, nxt);
    cell(p, cur);
    for (int t = threadIdx.x + blockDim.x; t < first[p * (rows + 1) + rows]; t += blockDim.x) {
      load(p, t, cur);
      cell(p, cur);
    }
    if (size == 1) __syncthreads(); else cl.sync();
  }
}

__global__ void __launch_bounds__(kLuThreads) k_lu_sweep(LusgsArgs a) {
  extern __shared__ double slots[];
  const cg::cluster_group cl = cg::this_cluster();
  const int n = a.ph.n, np = 3 * n - 2;
  const int size = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int cube = 1 + blockIdx.x / size;
  if (!case_active(a.bt, cube)) return;  // converged case (the whole cluster)
  const int rows = lu_rows(n, size);
  unsigned short *first = reinterpret_cast<unsigned short *>(slots + 30 * rows * n);
  for (int p = threadIdx.x; p < np; p += blockDim.x) {
    int sum = 0;
    for (int l = 0; l < rows; ++l) {
      const int i = l * size + rank;
      first[p * (rows + 1) + l] = (unsigned short)sum;
      const int jlo = max(0, p - i - (n - 1)), jhi = min(n - 1, p - i);
      if (i < n && jhi >= jlo) sum += jhi - jlo + 1;
    }
    first[p * (rows + 1) + rows] = (unsigned short)sum;
  }
  // every CTA of the cluster has started before any writes into its memory
  if (size == 1) __syncthreads(); else cl.sync();
  const double h = 0.5 / (a.cube_size[cube] / n);
  lu_sweep<true>(a, cl, slots, first, cube, h);   // dq* = (R + sum of lower A+ terms) / dg
  lu_sweep<false>(a, cl, slots, first, cube, h);  // dq = dq* - (sum of upper A- terms) / dg
}

// Q += dq on fluid cells and the partial sums of a cube, by a cluster of
// kUpdParts CTAs (the parts' sums added in order).
constexpr int kUpdThreads = 256, kUpdParts = 4;

// p, u, v, w, T of a state (p/rho for T) as the norms form them.
template <typename Div>
__device__ __forceinline__ void lu_prim(const double *q, double *p, Div div) {
  p[1] = div(q[1]); p[2] = div(q[2]); p[3] = div(q[3]);
  const double VV = p[1] * p[1] + p[2] * p[2] + p[3] * p[3];
  p[0] = (q[4] - 0.5 * q[0] * VV) * (BCMG_K - 1);
  p[4] = div(p[0]);
}

__global__ void __cluster_dims__(kUpdParts) __launch_bounds__(kUpdThreads)
    k_lu_update(LusgsArgs a) {
  __shared__ double red[kUpdThreads / 32][7];
  __shared__ double sums[7];
  const cg::cluster_group cl = cg::this_cluster();
  const int n = a.ph.n, S = n + 4, nn = n * n;
  const int cube = 1 + blockIdx.x / kUpdParts, part = blockIdx.x % kUpdParts;
  if (!case_active(a.bt, cube)) return;  // converged case (the whole cluster)
  double e[7] = {0, 0, 0, 0, 0, 0, 0};
  for (int r = part * kUpdThreads + threadIdx.x; r < nn * n; r += kUpdParts * kUpdThreads) {
    const size_t o = cell_index(S, cube, 2 + r / nn, 2 + (r / n) % n, 2 + r % n);
    e[5] += a.Residual1[5 * o + 0];
    e[6] += a.Residual1[5 * o + 1];
    if (a.FWS[o] != kFluid) continue;
    double q[5], x[5], p0[5], p1[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      q[m] = a.U1_[5 * o + m];
      x[m] = q[m] + a.Rku1[5 * o + m];
      a.U1_[5 * o + m] = x[m];
    }
    IntFp f;
    const Recip k0 = f.recip(q[0]), k1 = f.recip(x[0]);
    lu_prim(q, p0, [&](double y) { return f.div(y, k0); });
    lu_prim(x, p1, [&](double y) { return f.div(y, k1); });
    if (!f.ok) {
      lu_prim(q, p0, [&](double y) { return y / q[0]; });
      lu_prim(x, p1, [&](double y) { return y / x[0]; });
    }
#pragma unroll
    for (int m = 0; m < 5; ++m) e[m] += (p1[m] - p0[m]) * (p1[m] - p0[m]);
  }
#pragma unroll
  for (int m = 0; m < 7; ++m) {
    double v = e[m];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][m] = v;
  }
  __syncthreads();
  if (threadIdx.x < 7) {
    double v = 0;
    for (int w = 0; w < kUpdThreads / 32; ++w) v += red[w][threadIdx.x];
    sums[threadIdx.x] = v;
  }
  cl.sync();
  if (part == 0 && threadIdx.x < 7) {
    double v = 0;
    for (int w = 0; w < kUpdParts; ++w) v += cl.map_shared_rank(sums, w)[threadIdx.x];
    a.partials[(size_t)(cube - 1) * 7 + threadIdx.x] = v;
  }
  cl.sync();  // the parts stay until they are read
}

// The most cells of a plane in one CTA of a cluster.
int lu_plane_cells(int n, int size) {
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

int lusgs_launches() { return 3; }

cudaError_t launch_lusgs(const LusgsArgs &a, int ncubes, cudaStream_t s) {
  if (ncubes <= 0) return cudaSuccess;
  const int n = a.ph.n;
  if (n > 32) return cudaErrorInvalidValue;
  k_lu_coef<<<(n * n * n + kCoefThreads - 1) / kCoefThreads * ncubes, kCoefThreads, 0, s>>>(a);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  // Cluster size: two CTAs fit an SM's shared memory (24^3 cubes, 216 of them:
  // 2.48 ms against 3.00 for whole cubes per CTA), then larger while every
  // CTA can have an SM of its own and planes have cells enough for the
  // sub-partitions of more (8 cubes of 24^3: sizes 1, 2, 4, 8 take 1.61, 1.14,
  // 0.96, 0.93 ms; 64 cubes of 16^3, 96 cells a plane at size 2: 0.66, 0.61,
  // 0.62 ms; 216 cubes of 8^3: 0.30, 0.32 ms).
  int size = 1;
  while (lu_smem(n, size) > 113 * 1024) size *= 2;
  while (size < 8 && ncubes * size * 2 <= 152 && lu_plane_cells(n, size) > 96) size *= 2;
  const size_t smem = lu_smem(n, size);
  const int threads = std::min(kLuThreads, (lu_plane_cells(n, size) + 31) / 32 * 32);
  e = cudaFuncSetAttribute(k_lu_sweep, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
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
  cfg.numAttrs = 1;
  e = cudaLaunchKernelEx(&cfg, k_lu_sweep, a);
  if (e != cudaSuccess) return e;
  k_lu_update<<<ncubes * kUpdParts, kUpdThreads, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace bcmg
