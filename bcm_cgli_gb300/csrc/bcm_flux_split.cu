// Split-precision residual, preconditioned increment and stage update, fused.
//
// Same operator as BCM_Flux_XYZ_Viscous_Runge_kutta (BCM_Flux_XYZ_Viscous_
// Runge_kutta.cpp:326-2652) with the arithmetic split by where precision is
// needed:
//  * FP64: the conservative state Q (HBM), the time-level differences
//    Q - Q^n and Q^n - Q^(n-1) of the BDF2 source (the cancellation in
//    3Q - 4Q^n + Q^(n-1)), the state update Q += w * dQ, and the sums of the
//    residual/force norms;
//  * FP32: reconstruction, the preconditioned Roe flux, viscous gradients and
//    stresses, the residual sum and the pointwise 5x5 preconditioner.
// FP32 works on deltas from a per-case reference state (rho0, 0, 0, 0,
// P0/(K-1)) formed in FP64 (k_mirror), so pressure jumps are p' = p - P0
// differences and temperatures T' = T - T0 are O(1) numbers instead of
// 1e5 Pa / 300 K values whose FP32 rounding would swamp the low-Mach jumps.
// The constant P0 cancels exactly in every face-flux difference, so the
// momentum and force terms use p'.  The preconditioner's
// temp3 = H - H*K - VV + K*(T+VV) is formed as its exact identity
// 0.5*(K-1)*VV (C = K*T), avoiding a 1e5-scale cancellation in FP32.
#include <cuda_runtime.h>

#include "bcm_common.cuh"
#include "bcm_kernels.h"
#include "bcm_split_cell.cuh"

namespace bcmg {

// ---------------------------------------------------------------------------
// FP64 -> FP32 deltas of the state, all cells of all cubes (ghosts included),
// into one or both mirror buffers: once per dual-time step, and whenever the
// state was set from outside.  16-byte loads and 8-byte stores (a cube holds
// S^3 cells, S even, so cells pair up within a cube); 32-bit indices within a
// cube.  The conversions are the integer-pipe IEEE roundings of bcm_mirror.cuh,
// which every other mirror writer uses too.
// ---------------------------------------------------------------------------
// One block row per cube (blockIdx.y); lanes take consecutive 16-byte pairs of
// doubles (two cells are five pairs), kMirrorPairs of them per thread in flight.
// A thread of two whole cells reads with a stride of 80 bytes:
// 11.2 M cells (80 bytes each) 234 us, now 137.
constexpr int kMirrorPairs = 4;
__global__ void __launch_bounds__(256) k_mirror(const double2 *__restrict__ U,
                                                float2 *__restrict__ M, float2 *__restrict__ M1,
                                                double rho0_, double E0_, Batch bt, int cube_pairs,
                                                int ncubes) {
  for (int cube = 1 + blockIdx.y; cube <= ncubes; cube += gridDim.y) {
    double rho0 = rho0_, E0 = E0_;
    if (bt.cube_case) {  // the reference state of the cube's case
      const CaseConst *cq = bt.cases + bt.cube_case[cube];
      rho0 = cq->rho0;
      E0 = cq->E0;
    }
    const size_t base = (size_t)cube * cube_pairs;
    const int p0 = blockIdx.x * (256 * kMirrorPairs) + threadIdx.x;
    double2 u[kMirrorPairs];
#pragma unroll
    for (int r = 0; r < kMirrorPairs; ++r)
      if (p0 + 256 * r < cube_pairs) u[r] = U[base + p0 + 256 * r];
#pragma unroll
    for (int r = 0; r < kMirrorPairs; ++r) {
      const int p = p0 + 256 * r;
      if (p >= cube_pairs) break;
      // pairs 0..4: rho mx, my mz, E rho, mx my, mz E
      const int k = p % 5;
      const double x0 = k == 0 ? rho0 : (k == 2 ? E0 : 0.0), y0 = k == 2 ? rho0 : (k == 4 ? E0 : 0.0);
      const float2 m = make_float2(to_float_int(u[r].x - x0), to_float_int(u[r].y - y0));
      M[base + p] = m;
      if (M1) M1[base + p] = m;
    }
  }
}

cudaError_t launch_mirror(const double *U, float *M0, float *M1, int n, int ncube, double rho0,
                          double P0, const Batch &bt, cudaStream_t s) {
  if (ncube <= 1) return cudaSuccess;  // cube slot 0 is unused
  const int S = n + 4, pairs = 5 * S * S * S / 2;  // S is even
  const dim3 grid((pairs + 256 * kMirrorPairs - 1) / (256 * kMirrorPairs),
                  ncube - 1 < 65535 ? ncube - 1 : 65535);
  k_mirror<<<grid, 256, 0, s>>>(reinterpret_cast<const double2 *>(U),
                               reinterpret_cast<float2 *>(M0), reinterpret_cast<float2 *>(M1),
                               rho0, P0 / (BCMG_K - 1), bt, pairs, ncube - 1);
  return cudaGetLastError();
}

__global__ void k_mirror_flip(int *parity) { *parity ^= 1; }

cudaError_t launch_mirror_flip(int *parity, cudaStream_t s) {
  k_mirror_flip<<<1, 1, 0, s>>>(parity);
  return cudaGetLastError();
}

// Q^n - Q^(n-1) of the interior cells, formed in FP64 and stored in FP32, when
// the levels were set from outside; within a run the time shift forms it.
__global__ void k_level_diff(const double *__restrict__ U1, const double *__restrict__ U1q,
                             float *__restrict__ D2, int n, long long total) {
  const int S = n + 4;
  const long long n3 = (long long)n * n * n;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int c = 1 + (int)(t / n3);
    const int r = (int)(t % n3);
    const size_t o = 5 * cell_index(S, c, 2 + r / (n * n), 2 + (r / n) % n, 2 + r % n);
#pragma unroll
    for (int v = 0; v < 5; ++v) D2[o + v] = (float)(U1[o + v] - U1q[o + v]);
  }
}

cudaError_t launch_level_diff(const double *U1, const double *U1q, float *D2, int n, int ncube,
                              cudaStream_t s) {
  const long long total = (long long)(ncube - 1) * n * n * n;
  if (total <= 0) return cudaSuccess;
  int blocks = (int)((total + 255) / 256);
  if (blocks > 152 * 8) blocks = 152 * 8;
  k_level_diff<<<blocks, 256, 0, s>>>(U1, U1q, D2, n, total);
  return cudaGetLastError();
}

template <int T>
struct SplitSmem {
  static constexpr int B = T + 2;      // primitive box edge (tile + 1 halo)
  static constexpr int X = T + 6;      // stencil box edge (tile + 3 halo)
  static constexpr int nPrim = B * B * B;
  static constexpr int nCell = T * T * T;
  static constexpr int nBox = X * X * X;
  // Box pitches in floats: a row of X cells along k (5 floats each), a plane
  // of X rows.  For 8^3 tiles the pitches are padded (72 = 8 mod 32, 1011
  // odd) so that the stencil reads of a warp hit 32 distinct banks for x- and
  // z-faces (2 ways for y-faces) instead of 2 and 4 ways.
  static constexpr int RP = T == 8 ? 72 : 5 * X;
  static constexpr int PP = T == 8 ? 1011 : X * RP;
  static constexpr int nBoxF = X * PP;
  static constexpr int nFace = (T + 1) * T * T;  // faces of one axis
  static constexpr int nBits = (3 * nFace + 31) / 32;
  static constexpr size_t bytes = sizeof(float) * nBoxF /*state deltas*/ +
                                  sizeof(PrimF) * nPrim +
                                  sizeof(float) * 15 * nFace /*face fluxes, 3 axes*/ +
                                  sizeof(float) * 2 * nFace /*x, z face pressure halves*/ +
                                  sizeof(unsigned) * ((nBits + 3) / 4) * 4 /*second views*/ +
                                  ((nBox + 15) / 16) * 16 /*flags*/;
  static_assert(RP >= 5 * X && PP >= X * RP, "box pitches hold the rows");
  static_assert(T != 8 || bytes + 1024 <= 233472 / 2, "two CTAs per SM");
};

// Index of face fa (0..T along axis ax) at in-plane position (p, q) in the
// value-major face arrays.  The in-plane coordinates are (j, k) for x-faces,
// (i, k) for y-faces and (j, i) for z-faces.  For 8^3 tiles the plane index
// is rotated per face (by 8 fa for y-faces, by fa for z-faces) so that the
// 32 faces a warp stores (4 x 8 of one plane) and the faces 32 consecutive
// cells read (i, j, k order) land in distinct banks for every axis.
template <int T>
__device__ __forceinline__ int face_idx(int ax, int fa, int p, int q) {
  if (T == 8) {
    const int in = 8 * p + q;
    return fa * 64 + (ax == 0 ? in : ((in + (ax == 1 ? 8 * fa : fa)) & 63));
  }
  return (fa * T + p) * T + q;
}

// Threads per CTA: for 8^3 tiles, half the 576 faces of an axis (two faces
// and up to two cells per thread) so that two CTAs (~110 KB shared memory
// each) share an SM and one CTA's staging, barriers and FP64 tail overlap
// the other's FP32 work; for 4^3 tiles one face per thread.  Whole warps
// (the staging loop gives every warp whole rows).
template <int T>
__host__ __device__ constexpr int split_threads() {
  return T == 8 ? 288 : (((T + 1) * T * T) + 31) / 32 * 32;
}
template <int T>
__host__ __device__ constexpr int split_ctas_per_sm() { return T == 8 ? 2 : 1; }

// PACK (8^3 tiles only): each thread evaluates its two faces of an axis
// together in packed FP32 pairs; otherwise one after the other.
template <int T, bool VISCOUS, bool PACK>
__global__ void __launch_bounds__(split_threads<T>(), split_ctas_per_sm<T>())
    k_flux_split(FluxSplitArgs a) {
  static_assert(!PACK || (T == 8 && 2 * split_threads<T>() == (T + 1) * T * T),
                "packed face pairs: two faces of an axis per thread");
  using SM = SplitSmem<T>;
  constexpr int B = SM::B;
  constexpr int X = SM::X;
  constexpr int NT = split_threads<T>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float *box = reinterpret_cast<float *>(smem_raw);  // [X][X][X][5] deltas, pitches RP, PP
  PrimF *prim = reinterpret_cast<PrimF *>(box + SM::nBoxF);
  // Face fluxes stored once per face: [3 axes][5][nFace], the x- and z-face
  // pressure halves [2][nFace], and one bit per face whose minus-side cell
  // takes a different reconstruction order (that cell recomputes its view).
  constexpr int NF = SM::nFace;
  float *FF = reinterpret_cast<float *>(prim + SM::nPrim);
  float *FdP = FF + 15 * NF;
  unsigned *dbits = reinterpret_cast<unsigned *>(FdP + 2 * NF);
  signed char *fbox =
      reinterpret_cast<signed char *>(dbits + ((SM::nBits + 3) / 4) * 4);  // [X][X][X] flags
  float *Fb = FF;  // staging area of the int flags (before the face pass)

  const int n = a.ph.n, S = n + 4, nx = n + 1;
  const int nt = n / T;
  const int tid = threadIdx.x;
  const int tiles = nt * nt * nt;
  const int cube = a.cube0 + blockIdx.x / tiles;
  if (!case_active(a.bt, cube)) return;  // converged case (uniform per CTA)
  const int tl = blockIdx.x % tiles;
  const int bi = 2 + (tl / (nt * nt)) * T, bj = 2 + ((tl / nt) % nt) * T, bk = 2 + (tl % nt) * T;
  // Mirror buffers: read the current one; stages 1..3 write the deltas of
  // the tile's cells into the other one.
  const int par = mirror_index(a.mir);
  const float *__restrict__ M = a.mir.buf[par];
  float *const Mw = a.RK >= 1 ? a.mir.buf[par ^ 1] : nullptr;
  const int *__restrict__ F = a.FWS;
  const size_t cb = cell_index(S, cube, 0, 0, 0);
  const SplitConst z = split_const(a, cube);
  const float rho0 = z.rho0, P0 = z.P0, ef = z.ef;

  // The FP64 state, the previous level and the level difference of the
  // tile's own cells are read at the end of the stage: start moving their
  // rows (8 cells: 320 B, 320 B, 160 B) into L2 now.
  for (int r = tid; r < T * T * 4; r += NT) {
    const int row = r >> 2, part = r & 3;
    const size_t go = cb + ((size_t)(bi + row / T) * S + (bj + row % T)) * S + bk;
    const int od = part == 3 ? 5 * T - 1 : 16 * part;  // doubles
    const int of = part == 3 ? 5 * T - 1 : (part == 2 ? 32 : 0);  // floats
    prefetch_l2(a.U1_ + 5 * go + od);
    prefetch_l2(a.U1 + 5 * go + od);
    prefetch_l2(a.D2 + 5 * go + of);
  }

  // Phase 0: stage the stencil box (tile +- 3 cells, clipped to the padded
  // cube) of FP32 deltas and flags into shared memory with asynchronous
  // 4-byte copies (the rows of the AoS layout start at any 4-byte boundary),
  // all in flight at once and waited for once.  Each box row along k is a
  // contiguous run of 5*X floats, so the copies are coalesced.  The flags go
  // as ints into the face buffers (unused until the face passes) and are
  // narrowed to bytes below.  Box cells outside the padded cube are never
  // read by the stencil (the reconstruction order falls back before reaching
  // them) and are left unset.
  int *ftmp = reinterpret_cast<int *>(Fb);
  static_assert(SM::nBox <= 17 * SM::nFace, "int flags fit the face buffers");
  for (int w = tid; w < SM::nBits; w += NT) dbits[w] = 0u;
  {
    const int k0 = bk - 3;
    const int klo = k0 < 0 ? -k0 : 0;                 // first valid column
    const int khi = (k0 + X > S) ? S - k0 : X;        // one past the last
    const int ncol = khi - klo;
    const int warp = tid >> 5, lane = tid & 31;
    constexpr int NW = (NT + 31) / 32;
    for (int row = warp; row < X * X; row += NW) {
      const int bi_ = row / X, bj_ = row - (row / X) * X;
      const int gi = bi - 3 + bi_, gj = bj - 3 + bj_;
      if (gi < 0 || gi >= S || gj < 0 || gj >= S) continue;
      const size_t g = cb + ((size_t)gi * S + gj) * S + (k0 + klo);
      const float *src = M + 5 * g;
      float *dst = box + bi_ * SM::PP + bj_ * SM::RP + klo * 5;
      for (int e = lane; e < 5 * ncol; e += 32) cp_async4(dst + e, src + e);
      const int *fsrc = F + g;
      int *fdst = ftmp + row * X + klo;
      for (int e = lane; e < ncol; e += 32) cp_async4(fdst + e, fsrc + e);
    }
    cp_async_wait_all();
  }
  __syncthreads();
  for (int p = tid; p < SM::nBox; p += NT) fbox[p] = (signed char)ftmp[p];
  auto BX = [&](int li, int lj, int lk) -> const float * {  // li.. relative to tile origin
    return box + (li + 3) * SM::PP + (lj + 3) * SM::RP + (lk + 3) * 5;
  };
  auto FL = [&](int li, int lj, int lk) -> int {
    return fbox[((li + 3) * X + (lj + 3)) * X + (lk + 3)];
  };

  // Phase 1: primitives (u, v, w, T - T0) over the tile plus one halo cell.
  for (int p = tid; p < SM::nPrim; p += NT) {
    int li = p / (B * B), lj = (p / B) % B, lk = p % B;
    const float *q = BX(li - 1, lj - 1, lk - 1);
    prim[p] = prim_split(z, q);
  }
  __syncthreads();  // byte flags complete; the face buffers are free again

  const float inv = a.inv_dx[cube];

  // The three axes are unrolled: every axis-dependent index, stride and
  // flux variant is then a compile-time choice (6% of the launch on the
  // 7 M-cell TGV case, measured).
  // One face f of axis ax: reconstruction order of the stored view, the
  // left/right states, the second-view bit; returns the face's slot.
  auto face_prep = [&](int ax, int f, float *ML, float *MR) -> int {
    const int fa = f / (T * T), p = (f / T) % T, q = f % T;
    int li, lj, lk;  // a warp covers 4 x 8 faces of a plane (8 x 4 for z-faces)
    if (ax == 0) { li = fa; lj = p; lk = q; }
    else if (ax == 1) { li = p; lj = fa; lk = q; }
    else { li = q; lj = p; lk = fa; }
    const int g = (ax == 0 ? bi + li : (ax == 1 ? bj + lj : bk + lk));
    const int di = ax == 0, dj = ax == 1, dk = ax == 2;
    const int fm2 = FL(li - 2 * di, lj - 2 * dj, lk - 2 * dk),
              fm1 = FL(li - di, lj - dj, lk - dk), f0 = FL(li, lj, lk),
              fp1 = FL(li + di, lj + dj, lk + dk);
    const bool needB = fa < T, needF = fa > 0;
    const int ob = order_backward(g, fm2, fm1, fp1);
    const int of = order_forward(g, nx, fm2, f0, fp1);
    const float *base = BX(li, lj, lk);
    const int sstride = ax == 0 ? SM::PP : (ax == 1 ? SM::RP : 5);
    auto ld = [&](int d, int v) -> float { return base[sstride * d + v]; };
    // The stored view is the plus-side cell's (the minus-side cell's for
    // the last face, which has no plus cell in the tile); where the
    // minus-side cell's order differs it recomputes its own view.
    recon_split(needB ? ob : of, ld, ML, MR);
    const int fi = face_idx<T>(ax, fa, p, q);
    if (needB && needF && ob != of) {
      const int bit = ax * NF + fi;
      atomicOr(dbits + (bit >> 5), 1u << (bit & 31));
    }
    return fi;
  };

  // The three axes are unrolled: every axis-dependent index, stride and
  // flux variant is then a compile-time choice (6% of the launch on the
  // 7 M-cell TGV case, measured).
#pragma unroll
  for (int ax = 0; ax < 3; ++ax) {
    if (PACK) {
      // 8^3 tiles: the axis's 576 faces are two per thread (f and f + 288),
      // evaluated together in packed pairs.
      float MLa[5], MRa[5], MLb[5], MRb[5];
      const int fa_ = face_prep(ax, tid, MLa, MRa);
      const int fb_ = face_prep(ax, tid + NT, MLb, MRb);
      float2 ML2[5], MR2[5], F2v[5], dP2;
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        ML2[v] = make_float2(MLa[v], MLb[v]);
        MR2[v] = make_float2(MRa[v], MRb[v]);
      }
      if (ax == 0) face_flux_delta2<0>(ML2, MR2, ef, rho0, P0, F2v, dP2);
      else if (ax == 1) face_flux_delta2<1>(ML2, MR2, ef, rho0, P0, F2v, dP2);
      else face_flux_delta2<2>(ML2, MR2, ef, rho0, P0, F2v, dP2);
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        FF[(5 * ax + v) * NF + fa_] = F2v[v].x;
        FF[(5 * ax + v) * NF + fb_] = F2v[v].y;
      }
      if (ax != 1) {
        FdP[(ax == 2) * NF + fa_] = dP2.x;
        FdP[(ax == 2) * NF + fb_] = dP2.y;
      }
    } else {
      for (int f = tid; f < (T + 1) * T * T; f += NT) {
        float ML[5], MR[5], Fx[5], dP;
        const int fi = face_prep(ax, f, ML, MR);
        if (ax == 0) face_flux_delta<0>(ML, MR, ef, rho0, P0, Fx, dP);
        else if (ax == 1) face_flux_delta<1>(ML, MR, ef, rho0, P0, Fx, dP);
        else face_flux_delta<2>(ML, MR, ef, rho0, P0, Fx, dP);
#pragma unroll
        for (int v = 0; v < 5; ++v) FF[(5 * ax + v) * NF + fi] = Fx[v];
        if (ax != 1) FdP[(ax == 2) * NF + fi] = dP;
      }
    }
  }
  __syncthreads();
  // Norm / force partial sums of this CTA (stage 3), reduced below by all
  // threads.
  double s5[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  __shared__ double red8[T == 8 ? 16 * 7 : 1];  // n = 8: each warp turn's sums
  // Not unrolled: with the packed face pass, two cells' tails interleaved
  // measured 2.5% slower per launch (n = 16; 1.9% at n = 24, same bits).
#pragma unroll 1
  for (int cl = tid; cl < SM::nCell; cl += NT) {
  const int mi = cl / (T * T), mj = (cl / T) % T, mk = cl % T;
  // Flux balance of the cell from its six faces, axis by axis.
  float acc[5], dPdx = 0.f, dPdz = 0.f;
#pragma unroll
  for (int ax = 0; ax < 3; ++ax) {
    const int m = ax == 0 ? mi : (ax == 1 ? mj : mk);
    const int p = ax == 2 ? mj : (ax == 0 ? mj : mi), q = ax == 2 ? mi : mk;
    const int fb = face_idx<T>(ax, m, p, q), ff = face_idx<T>(ax, m + 1, p, q);
    float Fbv[5], Ffv[5], dPbv = 0.f, dPfv = 0.f;
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      Fbv[v] = FF[(5 * ax + v) * NF + fb];
      Ffv[v] = FF[(5 * ax + v) * NF + ff];
    }
    if (ax != 1) {
      dPbv = FdP[(ax == 2) * NF + fb];
      dPfv = FdP[(ax == 2) * NF + ff];
    }
    const int bit = ax * NF + ff;
    if (m + 1 < T && ((dbits[bit >> 5] >> (bit & 31)) & 1u)) {
      // the forward face's stored view is the next cell's: form this cell's
      const int li = mi + (ax == 0), lj = mj + (ax == 1), lk = mk + (ax == 2);
      const int g = (ax == 0 ? bi + li : (ax == 1 ? bj + lj : bk + lk));
      const int di = ax == 0, dj = ax == 1, dk = ax == 2;
      const int of = order_forward(g, nx, FL(li - 2 * di, lj - 2 * dj, lk - 2 * dk),
                                   FL(li, lj, lk), FL(li + di, lj + dj, lk + dk));
      const float *base = BX(li, lj, lk);
      const int sstride = ax == 0 ? SM::PP : (ax == 1 ? SM::RP : 5);
      auto ld = [&](int d, int v) -> float { return base[sstride * d + v]; };
      float ML[5], MR[5];
      recon_split(of, ld, ML, MR);
      if (ax == 0) face_flux_delta<0>(ML, MR, ef, rho0, P0, Ffv, dPfv);
      else if (ax == 1) face_flux_delta<1>(ML, MR, ef, rho0, P0, Ffv, dPfv);
      else face_flux_delta<2>(ML, MR, ef, rho0, P0, Ffv, dPfv);
    }
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      const float t = (Ffv[v] - Fbv[v]) * inv;
      acc[v] = ax == 0 ? t : acc[v] + t;
    }
    if (ax == 0) dPdx = dPfv - dPbv;
    if (ax == 2) dPdz = dPfv - dPbv;
  }
  auto P = [&](int di, int dj, int dk) -> const PrimF & {
    return prim[((mi + 1 + di) * B + (mj + 1 + dj)) * B + (mk + 1 + dk)];
  };
  const size_t go = cb + ((size_t)(bi + mi) * S + (bj + mj)) * S + (bk + mk);
  SplitLevels lv;
  float src[5];
  split_load(a, go, lv);
  constexpr int CVT = 2;
  split_source<CVT>(lv, src);
  split_cell<VISCOUS, true, CVT>(a, z, cube, inv, P, BX(mi, mj, mk), acc, lv.x, src, dPdx, dPdz, go,
                      FL(mi, mj, mk) == kFluid, Mw, s5, [&](auto *U, const auto *un) {
                        if (a.push) push_same_level(U, a.push, n, cube, bi + mi, bj + mj, bk + mk, un);
                      });
  if (T == 8 && nt == 1 && a.RK == 3) {  // (whole warps: 288 and 224 cells)
    const int m = norm_exchange(s5, tid & 31);
    if ((tid & 31) < 8 && m < 7) red8[(cl >> 5) * 7 + m] = s5[0];
#pragma unroll
    for (int v = 0; v < 8; ++v) s5[v] = 0;
  }
  }  // cells of this thread
  if (a.RK != 3) return;
  if (T == 8 && nt == 1) {
    // n = 8: the march's partial sums (two planes each: a plane is two warp
    // turns), so that either kernel gives a case the same norms
    __syncthreads();
    if (tid < 28) {
      const int c = tid / 7, m = tid - 7 * c;
      const double *r = red8 + 28 * c + m;
      a.partials[(size_t)blockIdx.x * 28 + tid] = 0 + (r[0] + r[14]) + (r[7] + r[21]);
    }
    return;
  }
  __syncthreads();  // the face buffers are reused for the block reduction
  double *red = reinterpret_cast<double *>(Fb);  // [NW][7]
  constexpr int NWR = NT / 32;
#pragma unroll
  for (int m = 0; m < 7; ++m) {
    double v = s5[m];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    if ((tid & 31) == 0) red[(tid >> 5) * 7 + m] = v;
  }
  __syncthreads();
  if (tid < 7) {
    double v = 0;
    for (int wv = 0; wv < NWR; ++wv) v += red[wv * 7 + tid];
    a.partials[(size_t)blockIdx.x * 7 + tid] = v;
  }
}

template <int T, bool VISCOUS, bool PACK>
static cudaError_t launch_split_k(const FluxSplitArgs &a, unsigned grid, cudaStream_t s) {
  const size_t smem = SplitSmem<T>::bytes;
  cudaError_t e = cudaFuncSetAttribute(k_flux_split<T, VISCOUS, PACK>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k_flux_split<T, VISCOUS, PACK><<<grid, split_threads<T>(), smem, s>>>(a);
  return cudaGetLastError();
}

template <int T>
static cudaError_t launch_split_t(const FluxSplitArgs &a, int ncubes, cudaStream_t s) {
  const int nt = a.ph.n / T;
  const unsigned grid = (unsigned)(ncubes * nt * nt * nt);
  if (grid == 0) return cudaSuccess;
  const bool visc = a.ph.mu_L != 0.0;
  if (T == 8 && a.form == 1)
    return visc ? launch_split_k<T, true, T == 8>(a, grid, s)
                : launch_split_k<T, false, T == 8>(a, grid, s);
  return visc ? launch_split_k<T, true, false>(a, grid, s) : launch_split_k<T, false, false>(a, grid, s);
}

int flux_tile(int n, int tile) {
  if (tile == 8 && n % 8 == 0) return 8;
  if (tile == 4 && n % 4 == 0) return 4;
  return n % 8 == 0 ? 8 : 4;
}

// Which kernel serves a cube edge.  The march holds seven planes of its rows in
// shared memory, so the larger the edge, the fewer its rows (4 at 48, 2 at 52 to
// 64, 1 at 68 to 80) and the more often values are loaded and formed, while 8^3
// tiles cost the same per cell at every edge they divide: 8^3 tiles and march, us a
// launch, 40 (64 cubes) 643 592, 48 (27) 475 390, 56 (27) 746 927, 64 (27) 1097
// 1163, 72 (8) 477 825, 80 (27) 2129 3389.  Edges that 8 does not divide would take
// 4^3 tiles, which the march beats wherever it fits: 52 (27) 1533 923, 60 (27) 2355
// 1179, 68 (8) 1023 784, 76 (8) 1428 922.
// For n = 8 a whole cube is one tile: the march wins while its two-plane
// units spread few cubes over the SMs (8 cubes 26 -> 20 us, 216 cubes 34 ->
// 28 us); the tile kernel's 18 warps per SM against 12 win from about 700
// cubes on (1000 cubes: 101 against 109 us).  Both leave the same bits,
// norms included.
constexpr int kMarchEdge8 = 48;  // the largest edge divisible by 8 that marches
static bool use_march(int n, int tile) {
  return tile != 4 && flux_march_fits(n) && (n % 8 != 0 || n <= kMarchEdge8);
}
constexpr int kMarchCubes8 = 700;

int flux_split_blocks(int n, int ncubes, int tile) {
  if (use_march(n, tile)) return flux_march_blocks(n, ncubes);
  const int T = flux_tile(n, tile);
  const int nt = n / T;
  return ncubes * nt * nt * nt;
}

cudaError_t launch_flux_split(const FluxSplitArgs &a, int ncubes, cudaStream_t s) {
  if (a.ph.n % 4 != 0) return cudaErrorInvalidValue;
  if (use_march(a.ph.n, a.tile) && !(a.ph.n == 8 && ncubes >= kMarchCubes8))
    return launch_flux_march(a, ncubes, s);
  if (flux_tile(a.ph.n, a.tile) == 8) return launch_split_t<8>(a, ncubes, s);
  return launch_split_t<4>(a, ncubes, s);
}

}  // namespace bcmg
