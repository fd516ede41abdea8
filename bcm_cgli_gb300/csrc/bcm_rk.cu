// RK stage combination, change norms and force sums.
//
// BCM_Flux_XYZ_Viscous_Runge_kutta.cpp:2417-2652.  Fluid cells only are
// updated; at stage 3 the L2 change norms of p, u, v, w, T over fluid cells
// and the force sums over all interior cells are formed.  The reference sums
// serially (its OpenMP accumulation at :2523 is unsynchronised); here each
// block sums a fixed contiguous range of cells in a fixed tree order and one
// cluster adds the block sums in a fixed order, so the result is run-to-run
// reproducible and equal to the serial sum within rounding.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "bcm_common.cuh"
#include "bcm_fp64_int.cuh"
#include "bcm_kernels.h"

namespace bcmg {

namespace cg = cooperative_groups;

constexpr int kRkThreads = 256;

// p, u, v, w, T (p/rho) of a state as the norms form them.
template <typename Div>
__device__ __forceinline__ void norm_prim(const double *q, double *p, Div div) {
  p[1] = div(q[1]); p[2] = div(q[2]); p[3] = div(q[3]);
  const double VV = p[1] * p[1] + p[2] * p[2] + p[3] * p[3];
  p[0] = (q[4] - 0.5 * q[0] * VV) * (BCMG_K - 1);
  p[4] = div(p[0]);
}
__device__ __noinline__ void norm_prim_ref(const double *q, double *p) {
  norm_prim(q, p, [&](double y) { return y / q[0]; });
}
__device__ __noinline__ void third_stage_ref(const double *q, const double *p2, const double *rk,
                                             double *x) {
  for (int v = 0; v < 5; ++v)
    x[v] = 1.0 / 3.0 * q[v] + 2.0 / 3.0 * p2[v] + 2.0 / 3.0 * rk[v];
}

// Bound by the FP64 pipe at stage 3 (73 cycles an operation of a warp, a
// division 584): the eight divisions and the fifteen products of the
// combination go to the integer pipes, and a warp's sums take 9 additions
// instead of 35: 262,144 cells of stage 3 94 -> 39 us, 393,216 with ghost and
// solid ones 120 -> 53.
__global__ void __launch_bounds__(kRkThreads) k_rk(RkArgs a, long long total, long long chunk) {
  const int n = a.ph.n, S = n + 4;
  long long beg = (long long)blockIdx.x * chunk;
  long long end = min(total, beg + chunk);
  if (a.blk_beg) {  // batches: the block's range lies inside one case
    beg = a.blk_beg[blockIdx.x];
    end = a.blk_beg[blockIdx.x + 1];
  }
  if (beg < end && !case_active(a.bt, 1 + (int)(beg / ((long long)n * n * n)))) return;
  double s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (long long t = beg + threadIdx.x; t < end; t += kRkThreads) {
    const int c = 1 + (int)(t / ((long long)n * n * n));
    const int r = (int)(t % ((long long)n * n * n));
    const int i = 2 + r / (n * n), j = 2 + (r / n) % n, k = 2 + r % n;
    const size_t o = cell_index(S, c, i, j, k);
    double *q = a.U1_ + 5 * o;
    const double *rk = a.Rku1 + 5 * o;
    const bool fluid = a.FWS[o] == kFluid;
    if (a.RK == 1) {
      if (fluid) {
#pragma unroll
        for (int v = 0; v < 5; ++v) {
          double x = q[v] + rk[v];
          q[v] = x;
          a.U1p1[5 * o + v] = x;
        }
      }
    } else if (a.RK == 2) {
      if (fluid) {
#pragma unroll
        for (int v = 0; v < 5; ++v) {
          double x = 0.75 * q[v] + 0.25 * a.U1p1[5 * o + v] + 0.25 * rk[v];
          q[v] = x;
          a.U1p2[5 * o + v] = x;
        }
      }
    } else {
      if (fluid) {
        IntFp f;
        double x[5], p0[5], p1[5];
        const Factor third = const_factor<__builtin_bit_cast(uint64_t, 1.0 / 3.0)>(),
                     thirds = const_factor<__builtin_bit_cast(uint64_t, 2.0 / 3.0)>();
        const double *p2 = a.U1p2 + 5 * o;
#pragma unroll
        for (int v = 0; v < 5; ++v)
          x[v] = f.mul(third, q[v]) + f.mul(thirds, p2[v]) + f.mul(thirds, rk[v]);
        if (!f.ok) {
          third_stage_ref(q, p2, rk, x);
          f.ok = true;
        }
        const Recip k0 = f.recip(q[0]), k1 = f.recip(x[0]);
        norm_prim(q, p0, [&](double y) { return f.div(y, k0); });
        norm_prim(x, p1, [&](double y) { return f.div(y, k1); });
        if (!f.ok) {
          norm_prim_ref(q, p0);
          norm_prim_ref(x, p1);
        }
#pragma unroll
        for (int v = 0; v < 5; ++v) {
          q[v] = x[v];
          s[v] += (p1[v] - p0[v]) * (p1[v] - p0[v]);
        }
      }
      s[5] += a.Residual1[5 * o + 0];
      s[6] += a.Residual1[5 * o + 1];
    }
  }
  if (a.RK != 3) return;
  // Fixed-shape block reduction: warp exchanges, then the warps in order.
  __shared__ double red[kRkThreads / 32][7];
  const int m = norm_exchange(s, threadIdx.x & 31);
  if ((threadIdx.x & 31) < 8 && m < 7) red[threadIdx.x >> 5][m] = s[0];
  __syncthreads();
  if (threadIdx.x < 7) {
    double v = 0;
    for (int w = 0; w < kRkThreads / 32; ++w) v += red[w][threadIdx.x];
    a.partials[(size_t)blockIdx.x * 7 + threadIdx.x] = v;
  }
}

// Deterministic sum of partials[b][0..6] over blocks [b0, b1) into tot[7]
// (shared) of the cluster's first CTA.  CTA r of the cluster takes the r-th of
// kNormCtas equal ranges; in it kNormWarps warps per quantity; lane l of warp w
// takes blocks 32 w + l, then every 32 kNormWarps-th, into four accumulators in
// turn (loads in flight), combined as (v0 + v1) + (v2 + v3); a fixed shuffle
// tree per warp, the warps' results in warp order and the CTAs' in theirs.
// The order depends only on b1 - b0, never on timing, so a batch's case and
// the same case alone sum identically.  Launch with 7 * kNormWarps warps.
// One CTA alone is bound by what it can keep in flight (7,776 blocks: 24 us;
// the cluster takes 13 for 18,432).
constexpr int kNormWarps = 4, kNormCtas = 8;
__device__ void sum_partials(const double *partials, int b0, int b1, double *tot) {
  __shared__ double part[7][kNormWarps];
  const cg::cluster_group cl = cg::this_cluster();
  const int each = (b1 - b0 + kNormCtas - 1) / kNormCtas;
  b0 += (int)cl.block_rank() * each;
  b1 = min(b1, b0 + each);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m = w / kNormWarps, sub = w % kNormWarps;
  constexpr int kStride = 32 * kNormWarps;
  if (m < 7) {
    double v0 = 0, v1 = 0, v2 = 0, v3 = 0;
    int b = b0 + sub * 32 + lane;
    for (; b + 3 * kStride < b1; b += 4 * kStride) {
      v0 += partials[(size_t)b * 7 + m];
      v1 += partials[(size_t)(b + kStride) * 7 + m];
      v2 += partials[(size_t)(b + 2 * kStride) * 7 + m];
      v3 += partials[(size_t)(b + 3 * kStride) * 7 + m];
    }
    for (; b < b1; b += kStride) v0 += partials[(size_t)b * 7 + m];
    double v = (v0 + v1) + (v2 + v3);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    if (lane == 0) part[m][sub] = v;
  }
  __syncthreads();
  if (threadIdx.x < 7) {
    double t = part[threadIdx.x][0];
    for (int q = 1; q < kNormWarps; ++q) t += part[threadIdx.x][q];
    tot[threadIdx.x] = t;
  }
  cl.sync();
  if (cl.block_rank() == 0 && threadIdx.x < 7) {
    double t = tot[threadIdx.x];
    for (int r = 1; r < kNormCtas; ++r) t += *cl.map_shared_rank(tot + threadIdx.x, r);
    tot[threadIdx.x] = t;
  }
  cl.sync();  // no CTA leaves while its sums are read
}

// er[1..5] = L2 change norms / (MPI_Ncube n^3), er[6], er[7] = force sums /
// (0.5 rho0 U0^2 2.602) (BCM_Flux...cpp:2628-2650); thread m forms the m-th.
// With emax (the end of a sub-iteration, main.cpp:1249-1259): E_k = max(E_k,
// er_k); er_k /= E_k.
__device__ void write_norms(int n, int mpi_ncube, double rho0, double U0, const double *tot,
                            double *er, double *emax) {
  const int m = threadIdx.x;
  if (m == 0) er[0] = 0;
  if (m < 5) {
    double DN = 1. / (mpi_ncube * n * n * n);
    double x = sqrt(tot[m]) * DN;
    if (emax) {
      const double E = emax[1 + m] > x ? emax[1 + m] : x;
      emax[1 + m] = E;
      x = x / E;
    }
    er[1 + m] = x;
  } else if (m < 7) {
    er[1 + m] = tot[m] / (0.5 * rho0 * U0 * U0 * 2.602);
  }
}

__global__ void k_norms(Phys ph, const double *partials, int nblocks, double *er,
                        const int *active, double *emax) {
  if (active && !active[0]) return;  // the whole cluster
  __shared__ double tot[7];
  sum_partials(partials, 0, nblocks, tot);
  if (blockIdx.x == 0) write_norms(ph.n, ph.mpi_ncube, ph.rho0, ph.U0, tot, er, emax);
}

// Cube-sharded runs: the raw sums of this rank's blocks (the ranks' sums are
// then added, as the reference's MPI_Allreduce does, BCM_Flux...cpp
// :2641-2652), and the norms from the summed values.
__global__ void k_norm_sums(const double *partials, int nblocks, double *sums,
                            const int *active) {
  if (active && !active[0]) return;
  __shared__ double tot[7];
  sum_partials(partials, 0, nblocks, tot);
  if (blockIdx.x == 0 && threadIdx.x < 7) sums[threadIdx.x] = tot[threadIdx.x];
}

__global__ void k_norm_final(Phys ph, const double *sums, double *er, const int *active,
                             double *emax) {
  if (active && !active[0]) return;
  write_norms(ph.n, ph.mpi_ncube, ph.rho0, ph.U0, sums, er, emax);
}

// One cluster per case of a batch.
__global__ void k_norms_batch(int n, const CaseConst *cases, const int *case_blk,
                              const double *partials, double *er, const int *active,
                              double *emax) {
  __shared__ double tot[7];
  const int q = blockIdx.x / kNormCtas;
  if (active && !active[q]) return;
  sum_partials(partials, case_blk[q], case_blk[q + 1], tot);
  if (blockIdx.x % kNormCtas == 0) {
    const CaseConst &c = cases[q];
    write_norms(n, c.mpi_ncube, c.rho0, c.U0, tot, er + 8 * (size_t)q,
                emax ? emax + 6 * (size_t)q : nullptr);
  }
}

static void rk_geometry(const RkArgs &a, long long &total, long long &chunk, int &nb) {
  const long long n3 = (long long)a.ph.n * a.ph.n * a.ph.n;
  total = (long long)(a.ncube - 1) * n3;
  nb = (int)((total + 4 * kRkThreads - 1) / (4 * kRkThreads));
  if (nb > 152 * 16) nb = 152 * 16;
  if (nb < 1) nb = 1;
  chunk = (total + nb - 1) / nb;
}

int rk_partial_blocks(const RkArgs &a) {
  long long total, chunk;
  int nb;
  rk_geometry(a, total, chunk, nb);
  return nb;
}

cudaError_t launch_rk(const RkArgs &a, int *nblocks_out, cudaStream_t s) {
  long long total, chunk;
  int nb;
  rk_geometry(a, total, chunk, nb);
  if (nblocks_out) *nblocks_out = nb;
  if (total <= 0) return cudaSuccess;
  k_rk<<<nb, kRkThreads, 0, s>>>(a, total, chunk);
  return cudaGetLastError();
}

template <typename... P, typename... A>
static cudaError_t launch_sums(void (*k)(P...), int clusters, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(clusters * kNormCtas);
  cfg.blockDim = dim3(7 * 32 * kNormWarps);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kNormCtas;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, static_cast<P>(args)...);
}

cudaError_t launch_norms(const Phys &ph, const double *partials, int nblocks, double *er,
                         cudaStream_t s, const int *active, double *emax) {
  return launch_sums(k_norms, 1, s, ph, partials, nblocks, er, active, emax);
}

cudaError_t launch_norm_sums(const double *partials, int nblocks, double *sums, cudaStream_t s,
                             const int *active) {
  return launch_sums(k_norm_sums, 1, s, partials, nblocks, sums, active);
}

cudaError_t launch_norm_final(const Phys &ph, const double *sums, double *er, cudaStream_t s,
                              const int *active, double *emax) {
  k_norm_final<<<1, 32, 0, s>>>(ph, sums, er, active, emax);
  return cudaGetLastError();
}

cudaError_t launch_norms_batch(int n, const CaseConst *cases, const int *case_blk, int ncase,
                               const double *partials, double *er, cudaStream_t s,
                               const int *active, double *emax) {
  if (ncase <= 0) return cudaSuccess;
  return launch_sums(k_norms_batch, ncase, s, n, cases, case_blk, partials, er, active, emax);
}

cudaError_t launch_rk_table(const RkArgs &a, int nblocks, cudaStream_t s) {
  if (nblocks <= 0 || !a.blk_beg) return cudaErrorInvalidValue;
  k_rk<<<nblocks, kRkThreads, 0, s>>>(a, 0, 0);
  return cudaGetLastError();
}

}  // namespace bcmg

namespace bcmg {

// Stage combination with a caller-chosen chunk (cells per block) and block
// count; partials must hold nblocks * 7 doubles.
cudaError_t launch_rk_chunked(const RkArgs &a, long long chunk, int nblocks, cudaStream_t s) {
  const long long n3 = (long long)a.ph.n * a.ph.n * a.ph.n;
  const long long total = (long long)(a.ncube - 1) * n3;
  if (total <= 0 || nblocks <= 0) return cudaSuccess;
  k_rk<<<nblocks, kRkThreads, 0, s>>>(a, total, chunk);
  return cudaGetLastError();
}

}  // namespace bcmg
