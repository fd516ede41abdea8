// Immersed-boundary preprocessing on the GPU (BCM_Immersed_boundary.cpp
// :127-1081), a setup step: for every IBM ghost cell of the finest cubes it
// finds the boundary point on the body's surface triangles, the image point
// in the fluid and the trilinear weights of the image point's 8 surrounding
// cells, which the ghost fill uses every stage (BCM_Ghostcell_minus.cpp).
//
// The reference loops ghost cells x triangles on one core.  Here:
//  * k_ibm_keep: one thread per triangle tests its three vertices against
//    every cube's box widened by 1.5 cells (k_ibm_cube_box, :330-430);
//  * k_ibm_tri_prep: the ray invariants of every kept triangle, once;
//  * k_ibm_ray_part / k_ibm_ray_combine: ghost cells x triangle ranges
//    (triangles staged through shared memory, read by every thread of the
//    CTA), then per cell the first closest hit of a ray along each
//    triangle's normal over all ranges (:686-720, :1409-1450);
//  * k_ibm_closest_part / k_ibm_closest_combine: the same split for the
//    cells without any hit, the last closest point (:1290-1405);
//  * the side test of a cell uses the dotp of the last hit cell at or before
//    it in the reference's (cube, i, j, k) order, because the reference never
//    resets it; that carry is a short sequential pass on the host;
//  * both searches leave out the pairs that an FP32 filter with a rigorous
//    margin shows to miss, so the FP64 tests, and with them every result, are
//    those of the full search;
//  * k_ibm_place: one thread per ghost cell forms the boundary and image
//    points, the distance test and the image point's base cell;
//    k_ibm_weights: 16 lanes per cell the inverse of the 8x8 Vandermonde matrix
//    (Gauss-Jordan with partial pivoting) and the eight weights (:759-1040).
// Every step keeps the reference's operation order and the translation unit
// is built with --fmad=false, so the tables equal the reference's.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/bcm_gb300.h"
#include "bcm_common.cuh"
#include "bcm_kernels.h"
#include "bcm_trace.h"

namespace bcmg {
namespace {

constexpr double kMinimum = 0.0000001;  // prm.h `minimum`
constexpr double kBig = 100000000;       // prm.h `MAX`
constexpr int kTriChunk = 128;           // triangles staged per CTA pass

// Box of every cube widened by 1.5 cells, box[c*6 + 0..5] = x lo, x hi,
// y lo, y hi, z lo, z hi (the reference's bounds expressions, :330-430).
__global__ void k_ibm_cube_box(int ncube, int n, const double *__restrict__ cube_size,
                               const double *__restrict__ X, const double *__restrict__ Y,
                               const double *__restrict__ Z, double *__restrict__ box) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncube) return;
  const double dx = cube_size[c] / n;
  double *b = box + 6 * (size_t)c;
  b[0] = X[c] - 1.5 * dx; b[1] = X[c] + cube_size[c] + 1.5 * dx;
  b[2] = Y[c] - 1.5 * dx; b[3] = Y[c] + cube_size[c] + 1.5 * dx;
  b[4] = Z[c] - 1.5 * dx; b[5] = Z[c] + cube_size[c] + 1.5 * dx;
}

// The order of the doubles as integers (NaN excluded, -0 as 0): comparisons
// on the integer pipes instead of 73 cycles a warp each on the FP64 pipe.
__device__ __forceinline__ long long sort_key(double x) {
  const long long b = __double_as_longlong(x == 0.0 ? 0.0 : x);
  return b < 0 ? b ^ 0x7fffffffffffffffll : b;
}

// keep[t] = 1 when a vertex of triangle t lies in some cube's widened box
// (cubes 1..ncube-1, staged through shared memory).
constexpr int kBoxChunk = 512, kKeepThreads = 128;
__global__ void __launch_bounds__(kKeepThreads) k_ibm_keep(int ntri,
                                                           const double *__restrict__ tri,
                                                           int ncube,
                                                           const double *__restrict__ box,
                                                           int *__restrict__ keep) {
  __shared__ long long sb[kBoxChunk * 6];
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  long long v[9];
  bool num[3] = {true, true, true};
  for (int e = 0; e < 9; ++e) {
    const double x = t < ntri ? tri[9 * (size_t)t + e] : 0.0;
    v[e] = sort_key(x);
    num[e / 3] &= x == x;
  }
  int k = 0;
  for (int c0 = 1; c0 < ncube; c0 += kBoxChunk) {
    const int cnt = min(kBoxChunk, ncube - c0);
    __syncthreads();
    for (int e = threadIdx.x; e < cnt * 6; e += blockDim.x) {
      const double x = box[6 * (size_t)c0 + e];
      // no number lies above a NaN lower or below a NaN upper bound
      sb[e] = x == x ? sort_key(x) : (e & 1 ? LLONG_MIN : LLONG_MAX);
    }
    __syncthreads();
    if (k || t >= ntri) continue;
    for (int c = 0; c < cnt && !k; ++c) {
      const long long *b = sb + 6 * c;
#pragma unroll
      for (int q = 0; q < 3; ++q)
        if (num[q] && v[3 * q] >= b[0] && v[3 * q] <= b[1] && v[3 * q + 1] >= b[2] &&
            v[3 * q + 1] <= b[3] && v[3 * q + 2] >= b[4] && v[3 * q + 2] <= b[5])
          k = 1;
    }
  }
  if (t < ntri) keep[t] = k;
}

// Closest point of a triangle (:1290-1405), with the interior weight formed
// as the reference forms it.
__device__ __noinline__ void closest(const double *v, double x, double y, double z,
                                        double *p) {
  const double *a = v, *b = v + 3, *c = v + 6;
  const double ab[3] = {b[0] - a[0], b[1] - a[1], b[2] - a[2]};
  const double ac[3] = {c[0] - a[0], c[1] - a[1], c[2] - a[2]};
  const double bc[3] = {c[0] - b[0], c[1] - b[1], c[2] - b[2]};
  const double ap[3] = {x - a[0], y - a[1], z - a[2]};
  const double d1 = ab[0] * ap[0] + ab[1] * ap[1] + ab[2] * ap[2];
  const double d2 = ac[0] * ap[0] + ac[1] * ap[1] + ac[2] * ap[2];
  if (d1 <= 0. && d2 <= 0.) { p[0] = a[0]; p[1] = a[1]; p[2] = a[2]; return; }
  const double bp[3] = {x - b[0], y - b[1], z - b[2]};
  const double d3 = ab[0] * bp[0] + ab[1] * bp[1] + ab[2] * bp[2];
  const double d4 = ac[0] * bp[0] + ac[1] * bp[1] + ac[2] * bp[2];
  if (d3 >= 0. && d4 <= d3) { p[0] = b[0]; p[1] = b[1]; p[2] = b[2]; return; }
  const double vc = d1 * d4 - d3 * d2;
  if (vc <= 0. && d1 >= 0. && d3 <= 0.) {
    const double w = d1 / (d1 - d3);
    p[0] = a[0] + w * ab[0]; p[1] = a[1] + w * ab[1]; p[2] = a[2] + w * ab[2];
    return;
  }
  const double cp[3] = {x - c[0], y - c[1], z - c[2]};
  const double d5 = ab[0] * cp[0] + ab[1] * cp[1] + ab[2] * cp[2];
  const double d6 = ac[0] * cp[0] + ac[1] * cp[1] + ac[2] * cp[2];
  if (d6 >= 0. && d5 <= d6) { p[0] = c[0]; p[1] = c[1]; p[2] = c[2]; return; }
  const double vb = d5 * d2 - d1 * d6;
  if (vb <= 0. && d2 >= 0. && d6 <= 0.) {
    const double w = d2 / (d2 - d6);
    p[0] = a[0] + w * ac[0]; p[1] = a[1] + w * ac[1]; p[2] = a[2] + w * ac[2];
    return;
  }
  const double va = d3 * d6 - d5 * d4;
  if (va <= 0. && (d4 - d3) >= 0. && (d5 - d6) >= 0.) {
    const double w = (d4 - d3) / ((d4 - d3) + (d5 - d6));
    p[0] = b[0] + w * bc[0]; p[1] = b[1] + w * bc[1]; p[2] = b[2] + w * bc[2];
    return;
  }
  const double denom = 1. / (va + vb + vc);
  const double vv = vb * denom;
  const double w = vc + denom;
  p[0] = a[0] + ab[0] * vv + ac[0] * w;
  p[1] = a[1] + ab[1] * vv + ac[1] * w;
  p[2] = a[2] + ab[2] * vv + ac[2] * w;
}

// Ray invariants of one kept triangle (computed once; the same values the
// reference recomputes for every ghost cell): v0, e1 = v1 - v0, e2 = v2 - v0,
// the normal nu = e1 x e2, dir = -nu / |nu|, p = dir x e2, det = e1 . p,
// 1 / det and dir . dir.
//
// And an FP32 filter: the search tests every ghost cell against every
// triangle, and nearly all pairs miss by far.  In coordinates o' = o - org
// relative to the ghost cells' box (centre org, half extents ext), f[0] and
// f[1] give u / det and w / det of the ray test as affine functions, each
// raised by a bound m on the error of evaluating it in FP32 (at most 8 roundings
// of 2^-24 of A = |p|.ext + |c| + 1; m = 2^-18 A also covers the FP64 test's own
// rounding) and scaled so that a hit has f0 >= 0, f1 >= 0 and f0 + f1 <= 1
// for certain.  f[2] is a sphere around the triangle (centre, radius widened
// in the same way).  Where m is not small (thin or far triangles, NaN), every
// pair passes.
constexpr int kRec = 22;
struct GhostBox {
  double org[3], ext[3];
};
__global__ void k_ibm_tri_prep(int ntri, const double *__restrict__ tri, GhostBox gb,
                               double *__restrict__ rec, float4 *__restrict__ filter) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ntri) return;
  const double *v = tri + 9 * (size_t)t;
  double *r = rec + kRec * (size_t)t;
  const double e1[3] = {v[3] - v[0], v[4] - v[1], v[5] - v[2]};
  const double e2[3] = {v[6] - v[0], v[7] - v[1], v[8] - v[2]};
  const double nu[3] = {e1[1] * e2[2] - e1[2] * e2[1], e1[2] * e2[0] - e1[0] * e2[2],
                        e1[0] * e2[1] - e1[1] * e2[0]};
  const double dis = sqrt(nu[0] * nu[0] + nu[1] * nu[1] + nu[2] * nu[2]);
  const double dir[3] = {-nu[0] / dis, -nu[1] / dis, -nu[2] / dis};
  const double pp[3] = {dir[1] * e2[2] - dir[2] * e2[1], dir[2] * e2[0] - dir[0] * e2[2],
                        dir[0] * e2[1] - dir[1] * e2[0]};
  const double det = e1[0] * pp[0] + e1[1] * pp[1] + e1[2] * pp[2];
  for (int q = 0; q < 3; ++q) {
    r[q] = v[q];
    r[3 + q] = e1[q];
    r[6 + q] = e2[q];
    r[9 + q] = dir[q];
    r[12 + q] = pp[q];
    r[15 + q] = nu[q];
  }
  r[18] = det;
  r[19] = 1.0 / det;
  r[20] = dir[0] * dir[0] + dir[1] * dir[1] + dir[2] * dir[2];
  r[21] = 0.0;
  const double ed[3] = {e1[1] * dir[2] - e1[2] * dir[1], e1[2] * dir[0] - e1[0] * dir[2],
                        e1[0] * dir[1] - e1[1] * dir[0]};
  double cu = 0, cw = 0, au = 1, aw = 1, ctr[3], far = 0, reach = 0;
  for (int q = 0; q < 3; ++q) {
    cu += (gb.org[q] - v[q]) * pp[q] / det;
    cw += (gb.org[q] - v[q]) * ed[q] / det;
    au += fabs(pp[q] / det) * gb.ext[q];
    aw += fabs(ed[q] / det) * gb.ext[q];
    ctr[q] = (v[q] + v[3 + q] + v[6 + q]) / 3.0;
    reach += gb.ext[q] + fabs(ctr[q] - gb.org[q]);
  }
  const double m = ldexp(fmax(au + fabs(cu), aw + fabs(cw)), -18), sc = 1.0 / (1.0 + 3.0 * m);
  // (a NaN in a term fails the comparison or shows in the sum)
  const bool use = m < 0.25 && au + aw + cu + cw < 1e30;
  float4 *f = filter + 3 * (size_t)t;
  f[0] = f[1] = make_float4(0.f, 0.f, 0.f, 0.25f);
  if (use) {
    const double ku = sc / det;
    f[0] = make_float4((float)(pp[0] * ku), (float)(pp[1] * ku), (float)(pp[2] * ku),
                       (float)((cu + m) * sc));
    f[1] = make_float4((float)(ed[0] * ku), (float)(ed[1] * ku), (float)(ed[2] * ku),
                       (float)((cw + m) * sc));
  }
  for (int e = 0; e < 3; ++e) {
    double d2 = 0;
    for (int q = 0; q < 3; ++q) d2 += (v[3 * e + q] - ctr[q]) * (v[3 * e + q] - ctr[q]);
    far = d2 > far || !(d2 == d2) ? d2 : far;
  }
  f[2] = make_float4((float)(ctr[0] - gb.org[0]), (float)(ctr[1] - gb.org[1]),
                     (float)(ctr[2] - gb.org[2]),
                     (float)(sqrt(far) * (1 + 1e-6) + ldexp(reach, -20)));
}

// False where the pair surely misses: o' outside the triangle's prism.
__device__ __forceinline__ bool may_hit(const float *o, float4 a, float4 b) {
  const float u = __fmaf_rn(o[0], a.x, __fmaf_rn(o[1], a.y, __fmaf_rn(o[2], a.z, a.w)));
  const float w = __fmaf_rn(o[0], b.x, __fmaf_rn(o[1], b.y, __fmaf_rn(o[2], b.z, b.w)));
  return !(fminf(fminf(u, w), 1.0f - u - w) < 0.f);
}

// Ray test of ghost centre o against triangle record r (Moller-Trumbore,
// :1409-1450: det below 1e-7 rejected, both directions accepted); on a hit
// returns 1 with tt = t.
__device__ __noinline__ int ray_hit(const double *o, const double *r, double *tt) {
  if (r[18] < kMinimum) return 0;
  const double tv[3] = {o[0] - r[0], o[1] - r[1], o[2] - r[2]};
  const double u = tv[0] * r[12] + tv[1] * r[13] + tv[2] * r[14];
  if (u < 0.0 || u > r[18]) return 0;
  const double q[3] = {tv[1] * r[5] - tv[2] * r[4], tv[2] * r[3] - tv[0] * r[5],
                       tv[0] * r[4] - tv[1] * r[3]};
  const double w = r[9] * q[0] + r[10] * q[1] + r[11] * q[2];
  if (w < 0.0 || u + w > r[18]) return 0;
  *tt = (r[6] * q[0] + r[7] * q[1] + r[8] * q[2]) * r[19];
  return 1;
}

// Search over the kept triangles, split over CTAs: blockIdx.x picks 128
// ghost cells, blockIdx.y one of gridDim.y contiguous triangle ranges.  Per
// (range, ghost): the number of ray hits and the first triangle with the
// smallest |t| (dir . dir), the reference's strict `<` over its serial loop.
// Cells are a list (cell < 0: skipped) so the closest-point pass below can
// reuse the layout.
// The FP32 filter leaves one or two triangles a cell for the FP64 test: 5,984
// cells by 20,480 triangles took 1,996 us with the FP64 test on every pair (its
// first dot product alone takes six slots of 73 cycles a warp), 57 with the
// filter.
constexpr int kGhostBlock = 128;
__global__ void __launch_bounds__(kGhostBlock)
    k_ibm_ray_part(int ng, const double *__restrict__ cen, GhostBox gb, int ntri, int per,
                   const double *__restrict__ rec, const float4 *__restrict__ filter,
                   int *__restrict__ hits_p, int *__restrict__ best_p,
                   double *__restrict__ nd_p) {
  __shared__ float4 sf[kTriChunk][2];
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  const bool has = g < ng;
  double o[3] = {0, 0, 0};
  if (has) { o[0] = cen[3 * g]; o[1] = cen[3 * g + 1]; o[2] = cen[3 * g + 2]; }
  float of[3];
  for (int q = 0; q < 3; ++q) of[q] = (float)(o[q] - gb.org[q]);
  const int t0 = blockIdx.y * per, t1 = min(ntri, t0 + per);
  int hits = 0, best = -1;
  double dmin = kBig;
  for (int base = t0; base < t1; base += kTriChunk) {
    const int cnt = min(kTriChunk, t1 - base);
    __syncthreads();
    for (int e = threadIdx.x; e < cnt * 2; e += blockDim.x)
      sf[e >> 1][e & 1] = filter[3 * ((size_t)base + (e >> 1)) + (e & 1)];
    __syncthreads();
    if (!has) continue;
#pragma unroll 4
    for (int t = 0; t < cnt; ++t) {
      if (!may_hit(of, sf[t][0], sf[t][1])) continue;
      const double *r = rec + kRec * ((size_t)base + t);
      double tt;
      if (!ray_hit(o, r, &tt)) continue;
      const double nd = fabs(tt) * r[20];
      ++hits;
      if (nd < dmin) { dmin = nd; best = base + t; }
    }
  }
  if (!has) return;
  const size_t at = (size_t)blockIdx.y * ng + g;
  hits_p[at] = hits;
  best_p[at] = best;
  nd_p[at] = dmin;
}

// Per ghost cell: total hits; of the closest hit (smallest |t| dir.dir, the
// lowest triangle on ties) |t|, direction and dotp = nu . (v0 - centre),
// recomputed from that triangle with the same arithmetic.  out[g*8 + 0..5] =
// hits, |t|, d0, d1, d2, dotp.
// One warp per cell: its lanes take the ranges in turn.
__global__ void k_ibm_ray_combine(int ng, int nsplit, const double *__restrict__ cen,
                                  const double *__restrict__ rec,
                                  const int *__restrict__ hits_p, const int *__restrict__ best_p,
                                  const double *__restrict__ nd_p, double *__restrict__ out) {
  const int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (g >= ng) return;
  int hits = 0, best = INT_MAX;
  double dmin = kBig;
  for (int sp = lane; sp < nsplit; sp += 32) {
    const size_t at = (size_t)sp * ng + g;
    hits += hits_p[at];
    const int b = best_p[at];
    if (b >= 0 && nd_p[at] < dmin) { dmin = nd_p[at]; best = b; }
  }
  for (int d = 16; d > 0; d >>= 1) {
    hits += __shfl_xor_sync(0xffffffffu, hits, d);
    const double nd = __shfl_xor_sync(0xffffffffu, dmin, d);
    const int b = __shfl_xor_sync(0xffffffffu, best, d);
    if (b != INT_MAX && (best == INT_MAX || nd < dmin || (nd == dmin && b < best))) {
      dmin = nd;
      best = b;
    }
  }
  if (lane) return;
  if (best == INT_MAX) best = -1;
  double tmin = kBig, d0 = 0, d1 = 0, d2 = 0, dotp = 0;
  if (best >= 0) {
    const double o[3] = {cen[3 * g], cen[3 * g + 1], cen[3 * g + 2]};
    const double *r = rec + kRec * (size_t)best;
    double tt = 0;
    ray_hit(o, r, &tt);
    tmin = fabs(tt);
    d0 = r[9]; d1 = r[10]; d2 = r[11];
    dotp = r[15] * (r[0] - o[0]) + r[16] * (r[1] - o[1]) + r[17] * (r[2] - o[2]);
  }
  double *w = out + 8 * (size_t)g;
  w[0] = hits; w[1] = tmin; w[2] = d0; w[3] = d1; w[4] = d2; w[5] = dotp;
}

// Closest-point search for the ghost cells without any hit (list[m] ghost
// numbers), split like the ray search: per (range, cell) the LAST triangle
// with the smallest squared distance (the reference's `<=`).
// The closest point lies in the triangle, so a triangle whose sphere is
// farther than the best so far is left out, unless the cell may lie in the
// triangle's prism: there the interior weight (as the reference forms it) puts
// the point anywhere.  5,874 cells: 455 us with every pair in FP64, 193 with each
// range's own best, 65 with a first pass for an upper bound.
__global__ void __launch_bounds__(kGhostBlock)
    k_ibm_closest_part(int m, const int *__restrict__ list, const double *__restrict__ cen,
                       GhostBox gb, int ntri, int per, const double *__restrict__ tri,
                       const float4 *__restrict__ filter, unsigned *__restrict__ bound,
                       int *__restrict__ best_p, double *__restrict__ nd_p) {
  __shared__ float4 sf[kTriChunk][3];
  const int e0 = blockIdx.x * blockDim.x + threadIdx.x;
  const bool has = e0 < m;
  double o[3] = {0, 0, 0};
  if (has) {
    const int g = list[e0];
    o[0] = cen[3 * g]; o[1] = cen[3 * g + 1]; o[2] = cen[3 * g + 2];
  }
  float of[3];
  for (int q = 0; q < 3; ++q) of[q] = (float)(o[q] - gb.org[q]);
  const int t0 = blockIdx.y * per, t1 = min(ntri, t0 + per);
  int best = -1;
  double dmin = kBig;
  float rmin = 1e4f * (1 + 1e-6f);  // no less than the closest point's distance
  // first pass: the smallest upper bound of the range, shared by all ranges
  // (whichever of them a range sees, it leaves out only triangles that are
  // farther than some other's point)
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    for (int base = t0; base < t1; base += kTriChunk) {
      const int cnt = min(kTriChunk, t1 - base);
      __syncthreads();
      for (int e = threadIdx.x; e < cnt * 3; e += blockDim.x)
        sf[e / 3][e % 3] = filter[3 * (size_t)base + e];
      __syncthreads();
      if (!has) continue;
      for (int t = 0; t < cnt; ++t) {
        const float4 c = sf[t][2];
        const float x = of[0] - c.x, y = of[1] - c.y, z = of[2] - c.z;
        const float d2 = __fmaf_rn(x, x, __fmaf_rn(y, y, z * z));
        if (pass == 0) {
          const float far = sqrtf(d2) * (1 + 1e-6f) + c.w;
          if (far < rmin && !may_hit(of, sf[t][0], sf[t][1])) rmin = far;
          continue;
        }
        const float r = c.w + rmin;
        if (d2 > r * r * (1 + 1e-6f) && !may_hit(of, sf[t][0], sf[t][1])) continue;
        double p[3];
        closest(tri + 9 * ((size_t)base + t), o[0], o[1], o[2], p);
        const double nd = (p[0] - o[0]) * (p[0] - o[0]) + (p[1] - o[1]) * (p[1] - o[1]) +
                          (p[2] - o[2]) * (p[2] - o[2]);
        if (nd <= dmin) {
          dmin = nd;
          best = base + t;
          rmin = fminf(rmin, sqrtf((float)nd) * (1 + 1e-6f) + 1e-18f);
        }
      }
    }
    if (pass == 0 && has) {
      const unsigned mine = __float_as_uint(rmin);  // positive: ordered as integers
      rmin = __uint_as_float(min(mine, atomicMin(bound + e0, mine)));
    }
  }
  if (!has) return;
  const size_t at = (size_t)blockIdx.y * m + e0;
  best_p[at] = best;
  nd_p[at] = dmin;
}

// The closest point of those cells (the highest triangle on ties) into
// out[g*8 + 2..4]; 0 when no triangle is within the search distance.  One warp
// per cell.
__global__ void k_ibm_closest_combine(int m, int nsplit, const int *__restrict__ list,
                                      const double *__restrict__ cen,
                                      const double *__restrict__ tri,
                                      const int *__restrict__ best_p,
                                      const double *__restrict__ nd_p, double *__restrict__ out) {
  const int e0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (e0 >= m) return;
  int best = -1;
  double dmin = kBig;
  for (int sp = lane; sp < nsplit; sp += 32) {
    const size_t at = (size_t)sp * m + e0;
    const int b = best_p[at];
    if (b >= 0 && nd_p[at] <= dmin) { dmin = nd_p[at]; best = b; }
  }
  for (int d = 16; d > 0; d >>= 1) {
    const double nd = __shfl_xor_sync(0xffffffffu, dmin, d);
    const int b = __shfl_xor_sync(0xffffffffu, best, d);
    if (b >= 0 && (best < 0 || nd < dmin || (nd == dmin && b > best))) {
      dmin = nd;
      best = b;
    }
  }
  if (lane) return;
  const int g = list[e0];
  double p[3] = {0, 0, 0};
  if (best >= 0) closest(tri + 9 * (size_t)best, cen[3 * g], cen[3 * g + 1], cen[3 * g + 2], p);
  double *w = out + 8 * (size_t)g;
  w[2] = p[0]; w[3] = p[1]; w[4] = p[2];
}

// Triangle ranges per ghost block so that a search launch fills the GPU
// (about 8 CTAs per SM), each range at least 64 triangles.
int sm_count() {
  int dev = 0, sms = 152;
  if (cudaGetDevice(&dev) == cudaSuccess)
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}
int ibm_splits(int nblocks, int ntri) {
  const int want = (8 * sm_count() + nblocks - 1) / nblocks;
  const int most = (ntri + 63) / 64;
  return std::max(1, std::min(want, most));
}

__device__ __noinline__ double plain_quotient(double x, double y) { return x / y; }

// The inverse of an 8x8 matrix (:1504-1576) by 16 lanes: lane l < 8 brings
// column l of the matrix in a, lane 8 + l the unit matrix's and ends with
// column l of the inverse.  The reference's Gauss-Jordan steps with row pivots
// treat columns alike, so each lane keeps one, and lane k shows its own (pivot
// row, pivot, factors) to the others at step k.
__device__ __forceinline__ void invert8(double *a, unsigned group, int lane0) {
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    double col[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) col[j] = __shfl_sync(group, a[j], lane0 + k);
    int mx = k;
    double big = fabs(col[k]);
#pragma unroll
    for (int j = k + 1; j < 8; ++j)
      if (fabs(col[j]) > big) { mx = j; big = fabs(col[j]); }
#pragma unroll
    for (int j = k + 1; j < 8; ++j)
      if (mx == j) {  // swap rows k and mx
        double t = a[j]; a[j] = a[k]; a[k] = t;
        t = col[j]; col[j] = col[k]; col[k] = t;
      }
    const double t = col[k];
    a[k] = plain_quotient(a[k], t);
    const double one = t == t && t != 0 && fabs(t) < INFINITY ? 1.0 : plain_quotient(t, t);
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (j != k) a[j] = a[j] - a[k] * (one == 1.0 ? col[j] : plain_quotient(col[j], one));
  }
}

// Per ghost cell: status (0 dropped, 1 turned fluid, 2 minus entry, 3 plus
// entry, these two if k_ibm_weights agrees), the image point's base cell, its
// offsets s1..s3 in it and the cell's edges (weight[0..5]).
constexpr int kPlaceThreads = 32;
__global__ void __launch_bounds__(kPlaceThreads)
    k_ibm_place(int ng, int n, const int *__restrict__ gidx, const double *__restrict__ cen,
                const double *__restrict__ srch, const double *__restrict__ dotp_eff,
                const double *__restrict__ cube_size, int ncube, const double *__restrict__ ctr,
                int *__restrict__ status, int *__restrict__ base, double *__restrict__ weight) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= ng) return;
  const int c = gidx[4 * g];
  const double o[3] = {cen[3 * g], cen[3 * g + 1], cen[3 * g + 2]};
  const double *r = srch + 8 * (size_t)g;
  const int hits = (int)r[0];
  const double tmin = r[1], d0 = r[2], d1 = r[3], d2 = r[4];
  const double dotp = dotp_eff[g];
  double BI[3], IP[3];
  if (dotp == 0) {
    for (int q = 0; q < 3; ++q) BI[q] = IP[q] = o[q];
  } else if (dotp > 0) {
    if (hits > 0) {
      BI[0] = o[0] - tmin * d0; BI[1] = o[1] - tmin * d1; BI[2] = o[2] - tmin * d2;
      IP[0] = o[0] + tmin * d0; IP[1] = o[1] + tmin * d1; IP[2] = o[2] + tmin * d2;
    } else {
      BI[0] = d0; BI[1] = d1; BI[2] = d2;
      for (int q = 0; q < 3; ++q) IP[q] = 2 * o[q] - BI[q];
    }
  } else {
    if (hits > 0) {
      BI[0] = o[0] + tmin * d0; BI[1] = o[1] + tmin * d1; BI[2] = o[2] + tmin * d2;
      IP[0] = o[0] - tmin * d0; IP[1] = o[1] - tmin * d1; IP[2] = o[2] - tmin * d2;
    } else {
      BI[0] = d0; BI[1] = d1; BI[2] = d2;
      for (int q = 0; q < 3; ++q) IP[q] = 2 * o[q] - BI[q];
    }
  }
  const double dx = cube_size[c] / n;
  const double dis = sqrt((BI[0] - o[0]) * (BI[0] - o[0]) + (BI[1] - o[1]) * (BI[1] - o[1]) +
                          (BI[2] - o[2]) * (BI[2] - o[2]));
  if (dis > sqrt(2.0) * dx) {
    status[g] = 1;
    return;
  }
  // cell centres of the cube along x, y, z (Xcnt, Ycnt, Zcnt)
  const int S = n + 4, nxx = n + 2;
  const double *cx = ctr + (size_t)c * S, *cy = ctr + ((size_t)ncube + c) * S,
               *cz = ctr + (2 * (size_t)ncube + c) * S;
  int ii, jj, kk, found = 0;
  for (ii = 0; ii <= nxx; ++ii)
    if (IP[0] >= cx[ii] && IP[0] <= cx[ii] + dx) { ++found; break; }
  for (jj = 0; jj <= nxx; ++jj)
    if (IP[1] >= cy[jj] && IP[1] <= cy[jj] + dx) { ++found; break; }
  for (kk = 0; kk <= nxx; ++kk)
    if (IP[2] >= cz[kk] && IP[2] <= cz[kk] + dx) { ++found; break; }
  if (found < 3) {
    status[g] = 0;
    return;
  }
  const double s1 = IP[0] - cx[ii], s2 = IP[1] - cy[jj], s3 = IP[2] - cz[kk];
  const double hx = cx[ii + 1] - cx[ii];
  const double hy = cy[jj + 1] - cy[jj];
  const double hz = cz[kk + 1] - cz[kk];
  status[g] = dotp >= 0 ? 2 : 3;
  base[3 * g] = ii;
  base[3 * g + 1] = jj;
  base[3 * g + 2] = kk;
  const double mid[6] = {s1, s2, s3, hx, hy, hz};
  for (int q = 0; q < 6; ++q) weight[8 * (size_t)g + q] = mid[q];
}

// The eight trilinear weights of the cells k_ibm_place kept, 16 lanes a cell;
// status 0 where one lies outside [0, 1].  A thread per cell with both
// matrices in local memory took 214 us for 5,984 cells (47 CTAs); this, with
// k_ibm_place, 62.
constexpr int kWeightThreads = 128;
__global__ void __launch_bounds__(kWeightThreads)
    k_ibm_weights(int ng, int *__restrict__ status, double *__restrict__ weight) {
  const int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 4;
  if (g >= ng || status[g] < 2) return;  // all 16 lanes
  const int l = threadIdx.x & 15, lane0 = threadIdx.x & 16;
  const unsigned group = 0xffffu << lane0;
  double *const w = weight + 8 * (size_t)g;
  const double s1 = w[0], s2 = w[1], s3 = w[2], hx = w[3], hy = w[4], hz = w[5];
  double a[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {  // corners 000, 100, 010, 001, 110, 101, 011, 111
    const double sx = q == 1 || q == 4 || q == 5 || q == 7 ? hx : 0,
                 sy = q == 2 || q == 4 || q == 6 || q == 7 ? hy : 0,
                 sz = q == 3 || q == 5 || q == 6 || q == 7 ? hz : 0;
    a[q] = l == 7 ? 1.0 : l == 6 ? sz : l == 5 ? sy : l == 4 ? sx : l == 3 ? sy * sz
         : l == 2 ? sx * sz : l == 1 ? sx * sy : l == 0 ? sx * sy * sz : (l - 8 == q ? 1.0 : 0.0);
  }
  invert8(a, group, lane0);
  const double x = a[0] * s1 * s2 * s3 + a[1] * s1 * s2 + a[2] * s1 * s3 + a[3] * s2 * s3 +
                   a[4] * s1 + a[5] * s2 + a[6] * s3 + a[7];
  const bool in = x >= (-kMinimum) && x <= (1 + kMinimum);
  const unsigned all = __ballot_sync(group, l < 8 || in);
  if ((all & group) != group) {
    if (l == 0) status[g] = 0;
  } else if (l >= 8) {
    w[l - 8] = x;
  }
}

// Device memory of one call: a single allocation, handed out in pieces.
struct DevArena {
  char *p = nullptr;
  size_t cap = 0, used = 0;
  ~DevArena() { if (p) cudaFree(p); }
  cudaError_t reserve(size_t bytes) {
    cap = bytes;
    return cudaMalloc((void **)&p, bytes);
  }
  static size_t padded(size_t bytes) { return (bytes + 255) / 256 * 256; }
};
template <typename T>
struct DevBuf {
  T *p = nullptr;
  cudaError_t alloc(DevArena &a, size_t count) {
    const size_t bytes = DevArena::padded(sizeof(T) * count);
    if (a.used + bytes > a.cap) return cudaErrorMemoryAllocation;
    p = reinterpret_cast<T *>(a.p + a.used);
    a.used += bytes;
    return cudaSuccess;
  }
};

}  // namespace
}  // namespace bcmg

using namespace bcmg;

namespace {

int fail(const std::string &m, int code) {
  bcmg_internal_set_error(m.c_str());
  return code;
}

#define CKI(expr)                                                                   \
  do {                                                                              \
    cudaError_t e__ = (expr);                                                       \
    if (e__ != cudaSuccess)                                                         \
      return fail(std::string(#expr) + ": " + cudaGetErrorString(e__), BCMG_ERR_CUDA); \
  } while (0)

}  // namespace

namespace {

// The preprocessing over a cell-centre table ctr[3][ncube][n+4] (x, y, z
// centres of every cube, BCM_Grid.cpp:124-148).
int ibm_run(int n, int ncube, const double *cube_size, const int *csl, const double *Xcube,
            const double *Ycube, const double *Zcube, const double *ctr, int *FWS, int ntri,
            const double *tri, int cap, int *nminus, int *gc_minus, int *ip_minus,
            double *w_minus, int *nplus, int *gc_plus, int *ip_plus, double *w_plus) {
  const int S = n + 4, nx = n + 1;
  // Ghost cells of the finest cubes, in (cube, i, j, k) order, and centres.
  std::vector<int> gidx;
  std::vector<double> cen;
  for (int c = 1; c < ncube; ++c) {
    if (csl[c] != 0) continue;
    if (!(cube_size[c] > 0)) return fail("cube_size must be positive", BCMG_ERR_ARG);
    for (int i = 2; i <= nx; ++i)
      for (int j = 2; j <= nx; ++j) {
        const int *row = FWS + cell_index(S, c, i, j, 0);
        int zeros = 0;
        for (int k = 2; k <= nx; ++k) zeros += row[k] == 0;
        if (zeros == 0) continue;
        for (int k = 2; k <= nx; ++k)
          if (row[k] == 0) {
            gidx.insert(gidx.end(), {c, i, j, k});
            cen.insert(cen.end(), {ctr[(size_t)c * S + i], ctr[((size_t)ncube + c) * S + j],
                                   ctr[(2 * (size_t)ncube + c) * S + k]});
          }
      }
  }
  const int ng = (int)(gidx.size() / 4);
  if (ng == 0 || ntri == 0) return BCMG_OK;  // nothing to do
  DevBuf<double> dtri, dsize, dX, dY, dZ, dctr, dcen, drec, dsrch, ddot, dw;
  DevBuf<int> dkeep, dg, dstat, dbase;
  DevBuf<float4> dfilter;
  DevArena mem;
  {
    // everything allocated below; a search's split results are at most
    // (8 SMs + blocks) blocks of cells
    const size_t blocks = (ng + kGhostBlock - 1) / kGhostBlock;
    const size_t parts = (ibm_splits((int)blocks, ntri) * blocks + 1) * kGhostBlock;
    const size_t parts_m = std::max(parts, (8 * (size_t)sm_count() + blocks + 1) * kGhostBlock);
    CKI(mem.reserve(64 * 256 + (size_t)ntri * (9 * 8 + 4 + kRec * 8 + 3 * 16) +
                    (size_t)ncube * (4 * 8 + 6 * 8 + 3 * 8 * (size_t)S) +
                    (size_t)ng * (3 * 8 + 4 * 4 + 8 * 8 + 8 + 4 + 3 * 4 + 8 * 8 + 8) +
                    (parts + parts_m) * 16));
  }
  CKI(dtri.alloc(mem, (size_t)ntri * 9));
  CKI(dsize.alloc(mem, ncube));
  CKI(dX.alloc(mem, ncube));
  CKI(dY.alloc(mem, ncube));
  CKI(dZ.alloc(mem, ncube));
  CKI(dkeep.alloc(mem, ntri));
  CKI(cudaMemcpy(dtri.p, tri, sizeof(double) * 9 * (size_t)ntri, cudaMemcpyHostToDevice));
  CKI(cudaMemcpy(dsize.p, cube_size, sizeof(double) * ncube, cudaMemcpyHostToDevice));
  CKI(cudaMemcpy(dX.p, Xcube, sizeof(double) * ncube, cudaMemcpyHostToDevice));
  CKI(cudaMemcpy(dY.p, Ycube, sizeof(double) * ncube, cudaMemcpyHostToDevice));
  CKI(cudaMemcpy(dZ.p, Zcube, sizeof(double) * ncube, cudaMemcpyHostToDevice));
  {
    DevBuf<double> dbox;
    CKI(dbox.alloc(mem, (size_t)6 * ncube));
    k_ibm_cube_box<<<(ncube + 127) / 128, 128>>>(ncube, n, dsize.p, dX.p, dY.p, dZ.p, dbox.p);
    CKI(cudaGetLastError());
    k_ibm_keep<<<(ntri + kKeepThreads - 1) / kKeepThreads, kKeepThreads>>>(ntri, dtri.p, ncube, dbox.p, dkeep.p);
    CKI(cudaGetLastError());
  }
  std::vector<int> keep(ntri);
  CKI(cudaMemcpy(keep.data(), dkeep.p, sizeof(int) * ntri, cudaMemcpyDeviceToHost));
  std::vector<double> kept;
  for (int t = 0; t < ntri; ++t)
    if (keep[t]) kept.insert(kept.end(), tri + 9 * (size_t)t, tri + 9 * (size_t)t + 9);
  const int nk = (int)(kept.size() / 9);
  if (nk == 0) return BCMG_OK;  // no triangle near any cube
  CKI(cudaMemcpy(dtri.p, kept.data(), sizeof(double) * kept.size(), cudaMemcpyHostToDevice));
  CKI(drec.alloc(mem, (size_t)nk * kRec));
  CKI(dfilter.alloc(mem, (size_t)nk * 3));
  GhostBox box;
  for (int q = 0; q < 3; ++q) {
    double lo = cen[q], hi = cen[q];
    for (int g = 1; g < ng; ++g) {
      lo = std::min(lo, cen[3 * (size_t)g + q]);
      hi = std::max(hi, cen[3 * (size_t)g + q]);
    }
    box.org[q] = 0.5 * (lo + hi);
    box.ext[q] = 0.5 * (hi - lo) * (1 + 1e-9) + 1e-300;
  }
  k_ibm_tri_prep<<<(nk + 127) / 128, 128>>>(nk, dtri.p, box, drec.p, dfilter.p);
  CKI(cudaGetLastError());
  CKI(dcen.alloc(mem, cen.size()));
  CKI(dg.alloc(mem, gidx.size()));
  CKI(dsrch.alloc(mem, (size_t)ng * 8));
  CKI(cudaMemcpy(dcen.p, cen.data(), sizeof(double) * cen.size(), cudaMemcpyHostToDevice));
  CKI(cudaMemcpy(dg.p, gidx.data(), sizeof(int) * gidx.size(), cudaMemcpyHostToDevice));
  {
    const int gb = (ng + kGhostBlock - 1) / kGhostBlock;
    const int ns = ibm_splits(gb, nk), per = (nk + ns - 1) / ns;
    DevBuf<int> hp, bp;
    DevBuf<double> np_;
    CKI(hp.alloc(mem, (size_t)ns * ng));
    CKI(bp.alloc(mem, (size_t)ns * ng));
    CKI(np_.alloc(mem, (size_t)ns * ng));
    k_ibm_ray_part<<<dim3(gb, ns), kGhostBlock>>>(ng, dcen.p, box, nk, per, drec.p, dfilter.p,
                                                  hp.p, bp.p, np_.p);
    CKI(cudaGetLastError());
    k_ibm_ray_combine<<<(ng + 3) / 4, 128>>>(ng, ns, dcen.p, drec.p, hp.p, bp.p, np_.p,
                                                 dsrch.p);
    CKI(cudaGetLastError());
  }
  // The side test's dotp carries over cells without a hit (in order).
  std::vector<double> srch((size_t)ng * 8), deff(ng);
  CKI(cudaMemcpy(srch.data(), dsrch.p, sizeof(double) * srch.size(), cudaMemcpyDeviceToHost));
  double carry = 0.0;
  std::vector<int> nohit;
  for (int g = 0; g < ng; ++g) {
    if (srch[8 * (size_t)g] > 0)
      carry = srch[8 * (size_t)g + 5];
    else
      nohit.push_back(g);
    deff[g] = carry;
  }
  // Closest points of the cells without a hit.
  if (!nohit.empty()) {
    const int m = (int)nohit.size();
    const int gb = (m + kGhostBlock - 1) / kGhostBlock;
    const int ns = ibm_splits(gb, nk), per = (nk + ns - 1) / ns;
    DevBuf<int> dl, bp;
    DevBuf<unsigned> db;
    DevBuf<double> np_;
    CKI(dl.alloc(mem, m));
    CKI(db.alloc(mem, m));
    CKI(cudaMemsetAsync(db.p, 0x7f, sizeof(unsigned) * m, nullptr));
    CKI(bp.alloc(mem, (size_t)ns * m));
    CKI(np_.alloc(mem, (size_t)ns * m));
    CKI(cudaMemcpy(dl.p, nohit.data(), sizeof(int) * m, cudaMemcpyHostToDevice));
    k_ibm_closest_part<<<dim3(gb, ns), kGhostBlock>>>(m, dl.p, dcen.p, box, nk, per, dtri.p,
                                                      dfilter.p, db.p, bp.p, np_.p);
    CKI(cudaGetLastError());
    k_ibm_closest_combine<<<(m + 3) / 4, 128>>>(m, ns, dl.p, dcen.p, dtri.p, bp.p, np_.p,
                                                    dsrch.p);
    CKI(cudaGetLastError());
  }
  CKI(dctr.alloc(mem, (size_t)3 * ncube * S));
  CKI(ddot.alloc(mem, ng));
  CKI(dstat.alloc(mem, ng));
  CKI(dbase.alloc(mem, (size_t)ng * 3));
  CKI(dw.alloc(mem, (size_t)ng * 8));
  CKI(cudaMemcpy(dctr.p, ctr, sizeof(double) * 3 * (size_t)ncube * S, cudaMemcpyHostToDevice));
  CKI(cudaMemcpy(ddot.p, deff.data(), sizeof(double) * ng, cudaMemcpyHostToDevice));
  k_ibm_place<<<(ng + kPlaceThreads - 1) / kPlaceThreads, kPlaceThreads>>>(
      ng, n, dg.p, dcen.p, dsrch.p, ddot.p, dsize.p, ncube, dctr.p, dstat.p, dbase.p, dw.p);
  CKI(cudaGetLastError());
  k_ibm_weights<<<(16 * (long long)ng + kWeightThreads - 1) / kWeightThreads, kWeightThreads>>>(
      ng, dstat.p, dw.p);
  CKI(cudaGetLastError());
  std::vector<int> stat(ng), base((size_t)ng * 3);
  std::vector<double> w((size_t)ng * 8);
  CKI(cudaMemcpy(stat.data(), dstat.p, sizeof(int) * ng, cudaMemcpyDeviceToHost));
  CKI(cudaMemcpy(base.data(), dbase.p, sizeof(int) * base.size(), cudaMemcpyDeviceToHost));
  CKI(cudaMemcpy(w.data(), dw.p, sizeof(double) * w.size(), cudaMemcpyDeviceToHost));
  int cm = 0, cp = 0;
  for (int g = 0; g < ng; ++g) {
    cm += stat[g] == 2;
    cp += stat[g] == 3;
  }
  if (cm > cap || cp > cap) return fail("IBM table capacity exceeded", BCMG_ERR_ARG);
  if ((cm && (!gc_minus || !ip_minus || !w_minus)) || (cp && (!gc_plus || !ip_plus || !w_plus)))
    return fail("output table pointer missing", BCMG_ERR_ARG);
  for (int g = 0; g < ng; ++g) {
    const int *G = &gidx[4 * (size_t)g];
    if (stat[g] == 1) {
      FWS[cell_index(S, G[0], G[1], G[2], G[3])] = 1;  // boundary point too far: fluid
      continue;
    }
    if (stat[g] < 2) continue;
    const bool minus = stat[g] == 2;
    const int m = minus ? (*nminus)++ : (*nplus)++;
    int *GC = minus ? gc_minus : gc_plus, *IP = minus ? ip_minus : ip_plus;
    double *W = minus ? w_minus : w_plus;
    for (int q = 0; q < 4; ++q) GC[4 * m + q] = G[q];
    IP[4 * m] = G[0];
    for (int q = 0; q < 3; ++q) IP[4 * m + 1 + q] = base[3 * (size_t)g + q];
    for (int q = 0; q < 8; ++q) W[8 * m + q] = w[8 * (size_t)g + q];
  }
  return BCMG_OK;
}

}  // namespace

extern "C" int bcmg_ibm_preprocess(int n, int ncube, const double *cube_size, const int *csl,
                                   const double *Xcube, const double *Ycube, const double *Zcube,
                                   int *FWS, int ntri, const double *tri, int cap, int *nminus,
                                   int *gc_minus, int *ip_minus, double *w_minus, int *nplus,
                                   int *gc_plus, int *ip_plus, double *w_plus) {
  bcmg::TraceRange trace("bcmg_ibm_preprocess");
  bcmg_internal_set_error(nullptr);
  if (!nminus || !nplus) return fail("bad arguments", BCMG_ERR_ARG);
  *nminus = 0;
  *nplus = 0;
  if (n < 1 || ncube < 1 || !cube_size || !csl || !Xcube || !Ycube || !Zcube || !FWS ||
      ntri < 0 || (ntri > 0 && !tri) || cap < 0)
    return fail("bad arguments", BCMG_ERR_ARG);
  const int S = n + 4;
  // Cell centres as BCM_Grid.cpp:124-148 forms them.
  std::vector<double> ctr((size_t)3 * ncube * S, 0.0);
  const double *corner[3] = {Xcube, Ycube, Zcube};
  for (int a = 0; a < 3; ++a)
    for (int c = 1; c < ncube; ++c) {
      const double dx = cube_size[c] / n;
      for (int i = 0; i < S; ++i) ctr[((size_t)a * ncube + c) * S + i] = corner[a][c] + (i - 1.5) * dx;
    }
  return ibm_run(n, ncube, cube_size, csl, Xcube, Ycube, Zcube, ctr.data(), FWS, ntri, tri, cap,
                 nminus, gc_minus, ip_minus, w_minus, nplus, gc_plus, ip_plus, w_plus);
}

// ---------------------------------------------------------------------------
// Drop-in twin of BCM_Immersed_boundary (main.h:113-147, called at
// main.cpp:811): reads BCM_STL_fine.stl from the working directory with the
// reference's parsing (:197-270), runs the GPU preprocessing with the
// reference configuration's NcubeX, updates FWS and writes
// IBM_minus<myid>.dat / IBM_plus<myid>.dat exactly as :989-1047 does.  Cell
// centres come from Xcnt/Ycnt/Zcnt ([ncube][NcubeX+4] each, as the
// reference reads them); null arrays: formed from the cube corners like
// BCM_Grid.cpp:124-148.  Errors: bcmg_last_error() (the reference has no
// error path; a missing STL file is an error here).
// ---------------------------------------------------------------------------
extern "C" void BCM_Immersed_boundary(int myid, int ncube, int n_wallcube, int *NBC, double Xmin,
                                      double Xmax, double Ymin, double Ymax, double Zmin,
                                      double Zmax, double *cube_size, int *csl, double *Xcube,
                                      double *Ycube, double *Zcube, double *Xcnt, double *Ycnt,
                                      double *Zcnt, int *FWS, int *wallcube) {
  bcmg::TraceRange trace("BCM_Immersed_boundary");
  (void)n_wallcube; (void)NBC; (void)Xmin; (void)Xmax; (void)Ymin; (void)Ymax; (void)Zmin;
  (void)Zmax; (void)wallcube;
  bcmg_internal_set_error(nullptr);
  bcmg_reference_config cfg;
  bcmg_get_reference_config(&cfg);
  FILE *f = std::fopen("BCM_STL_fine.stl", "r");
  if (!f) { fail("cannot open BCM_STL_fine.stl", BCMG_ERR_ARG); return; }
  // Facets: after each token "normal", the normal, "outer loop vertex",
  // three coordinates, "vertex", three, "vertex", three.
  std::vector<double> tri;
  char tok[1024];
  while (std::fscanf(f, "%1023s", tok) == 1) {
    if (std::strstr("normal", tok) == nullptr) continue;
    double nv[3], v[9];
    char s1[1024], s2[1024], s3[1024], s4[1024], s5[1024];
    if (std::fscanf(f, "%lf%lf%lf%1023s%1023s%1023s%lf%lf%lf%1023s%lf%lf%lf%1023s%lf%lf%lf",
                    &nv[0], &nv[1], &nv[2], s1, s2, s3, &v[0], &v[1], &v[2], s4, &v[3], &v[4],
                    &v[5], s5, &v[6], &v[7], &v[8]) != 17)
      break;
    tri.insert(tri.end(), v, v + 9);
  }
  std::fclose(f);
  const int ntri = (int)(tri.size() / 9);
  const int n = cfg.ncube_x, S = n + 4;
  if (n < 1 || ncube < 1 || !cube_size || !csl || !Xcube || !Ycube || !Zcube || !FWS) {
    fail("bad arguments", BCMG_ERR_ARG);
    return;
  }
  std::vector<double> ctr((size_t)3 * ncube * S, 0.0);
  const double *cnt[3] = {Xcnt, Ycnt, Zcnt}, *corner[3] = {Xcube, Ycube, Zcube};
  for (int a = 0; a < 3; ++a)
    for (int c = 1; c < ncube; ++c) {
      const double dx = cube_size[c] / n;
      for (int i = 0; i < S; ++i)
        ctr[((size_t)a * ncube + c) * S + i] =
            cnt[a] ? cnt[a][(size_t)c * S + i] : corner[a][c] + (i - 1.5) * dx;
    }
  int cap = 1;
  for (size_t e = 0; e < (size_t)ncube * S * S * S; ++e) cap += FWS[e] == 0;
  std::vector<int> gm(4 * (size_t)cap), im(4 * (size_t)cap), gp(4 * (size_t)cap),
      ipp(4 * (size_t)cap);
  std::vector<double> wm(8 * (size_t)cap), wp(8 * (size_t)cap);
  int nm = 0, np = 0;
  if (ibm_run(n, ncube, cube_size, csl, Xcube, Ycube, Zcube, ctr.data(), FWS, ntri, tri.data(),
              cap, &nm, gm.data(), im.data(), wm.data(), &np, gp.data(), ipp.data(),
              wp.data()) != BCMG_OK)
    return;
  for (int side = 0; side < 2; ++side) {
    char name[64];
    std::snprintf(name, sizeof name, side == 0 ? "IBM_plus%05d.dat" : "IBM_minus%05d.dat", myid);
    FILE *o = std::fopen(name, "w");
    if (!o) { fail(std::string("cannot write ") + name, BCMG_ERR_ARG); return; }
    const int m = side == 0 ? np : nm;
    const int *G = side == 0 ? gp.data() : gm.data(), *I = side == 0 ? ipp.data() : im.data();
    const double *W = side == 0 ? wp.data() : wm.data();
    for (int e = 0; e < m; ++e) {
      std::fprintf(o, "%d\t%d\t%d\t%d\n", G[4 * e], G[4 * e + 1], G[4 * e + 2], G[4 * e + 3]);
      std::fprintf(o, "%d\t%d\t%d\t%d\n", I[4 * e], I[4 * e + 1], I[4 * e + 2], I[4 * e + 3]);
      std::fprintf(o, "%f\t%f\t%f\t%f\t%f\t%f\t%f\t%f\n", W[8 * e], W[8 * e + 1], W[8 * e + 2],
                   W[8 * e + 3], W[8 * e + 4], W[8 * e + 5], W[8 * e + 6], W[8 * e + 7]);
    }
    std::fprintf(o, "Number of Boundary Cells\n");
    std::fprintf(o, "%d", m);
    std::fclose(o);
  }
}
