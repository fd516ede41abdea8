// The split-precision stage as a march along i.
//
// Same operator and arithmetic as k_flux_split (bcm_flux_split.cu); another
// walk.  A CTA owns TJ rows (j) of whole k extent of a cube and marches along
// i, two planes a step; each thread owns one (j, k) column.  Against 8^3
// tiles:
//  * the delta planes arrive once per CTA through a ring of seven (a 16^3 cube
//    loads 1.6 cells per cell instead of 5.4), by 16-byte asynchronous copies
//    issued a step ahead, so their latency hides behind the cells' work;
//  * a thread's offsets, pushes and column are set up once and then step by a
//    plane: index arithmetic was a third of the tile kernel's instructions;
//  * the i-faces of a column stay in registers, their stencils overlap (35
//    loads for two faces instead of 60), and primitives are formed 1.27 times
//    per cell instead of 1.95;
//  * reconstruction orders come from a two-byte code per cell formed once per
//    case (flags do not change while it steps) instead of staged flags.
// The two planes of a step go through the face arithmetic as packed FP32
// pairs (PACK), like the tile kernel's two faces per thread.
//
// One RK-stage launch, tile kernel -> march (ms): 2,744 cubes of 16^3 1.726 ->
// 1.278, 512 of 16^3 0.336 -> 0.259, 512 of 24^3 1.094 -> 0.871, 216 of 32^3
// 1.096 -> 0.750; edges that 8 does not divide took 4^3 tiles: 512 cubes of
// 12^3 0.361 -> 0.148, 216 of 20^3 0.696 -> 0.257, 125 of 28^3 1.104 -> 0.412.
// 44% fewer instructions than the tiles at n = 16.  What bounds it now (ncu, n =
// 16): instruction latency with four warps per scheduler (issue slots 43%
// active, no pipe above 26%; 128 registers and 108 KB a CTA allow no more
// warps).  Tried and left out, against 1.37 ms at 2,744 cubes then: nine warps
// of 96 registers with a warp for the far faces (spills: 1.69), loading the
// next cell's FP64 levels ahead into registers (spills: 1.63), whole cubes per
// CTA instead of equal shares (1.34 there, but 0.294 at 512 cubes), one CTA of
// 576 threads for n = 24 (1.11 against 0.93).
#include <algorithm>
#include <type_traits>

#include "bcm_split_cell.cuh"

namespace bcmg {

// ---------------------------------------------------------------------------
// Cell codes.  bit 0: fluid; bits 1-2, 3-4, 5-6: the order (0: 1, 1: 3, 2: 5)
// of the cell's low x, y, z faces as the cell sees them (backward); bits 7-8,
// 9-10, 11-12: as the cell before sees them (forward); bits 13-15: the two
// views of the cell's high x, y, z face differ.
// ---------------------------------------------------------------------------
__global__ void k_cell_codes(const int *__restrict__ F, uint16_t *__restrict__ codes, int n,
                             long long total) {
  const int S = n + 4, nx = n + 1;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int k = (int)(t % S), j = (int)(t / S % S), i = (int)(t / ((long long)S * S) % S);
    const int x[3] = {i, j, k};
    const long long st[3] = {(long long)S * S, S, 1};
    unsigned c = F[t] == kFluid ? 1u : 0u;
    const int inside = (i >= 2 && i <= nx) + (j >= 2 && j <= nx) + (k >= 2 && k <= nx);
    for (int ax = 0; ax < 3; ++ax) {
      const int g = x[ax];
      const bool others = inside - (g >= 2 && g <= nx) == 2;
      if (!others || g < 2 || g > n + 2) continue;
      auto f = [&](int d) { return F[t + d * st[ax]]; };
      auto code = [](int ord) { return ord == 1 ? 0u : (ord == 3 ? 1u : 2u); };
      const int ob = order_backward(g, f(-2), f(-1), f(1));
      const int of = order_forward(g, nx, f(-2), f(0), f(1));
      c |= code(ob) << (1 + 2 * ax) | code(of) << (7 + 2 * ax);
      if (g <= nx && order_backward(g + 1, f(-1), f(0), f(2)) !=
                         order_forward(g + 1, nx, f(-1), f(1), f(2)))
        c |= 1u << (13 + ax);
    }
    codes[t] = (uint16_t)c;
  }
}

cudaError_t launch_cell_codes(const int *FWS, uint16_t *codes, int n, int ncube, cudaStream_t s) {
  const int S = n + 4;
  const long long total = (long long)ncube * S * S * S;
  if (total <= 0) return cudaSuccess;
  const int blocks = (int)std::min<long long>((total + 255) / 256, 152 * 32);
  k_cell_codes<<<blocks, 256, 0, s>>>(FWS, codes, n, total);
  return cudaGetLastError();
}

namespace {

__device__ __forceinline__ int code_back(unsigned c, int ax) { return 1 + 2 * ((c >> (1 + 2 * ax)) & 3); }
__device__ __forceinline__ int code_fwd(unsigned c, int ax) { return 1 + 2 * ((c >> (7 + 2 * ax)) & 3); }

__device__ __forceinline__ void cp_async16(float *smem_dst, const float *gmem_src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gmem_src) : "memory");
}

constexpr int kRing = 7;    // delta planes i-2 .. i+4 of a step (i, i+1)
constexpr int kPrimRing = 4;  // primitive planes i-1 .. i+2
constexpr int kChunk = 2;   // planes per unit of work and norm partial sum

// Shared-memory layout (floats) for cubes of edge n in tiles of tj rows.  The
// row pitch is 5 n (mod 32), so the columns of consecutive threads fall into
// consecutive multiples of five banks across rows: no conflicts.
struct MarchLayout {
  int pitch, rows, plane, prim_row, prim_plane, fy, fz, flux;
  __host__ __device__ MarchLayout(int n, int tj) {
    pitch = 5 * n + 32;
    rows = tj == n ? n + 4 : tj + 6;
    plane = rows * pitch;
    prim_row = n + 2;
    prim_plane = (tj + 2) * (n + 2);
    fy = (tj + 1) * n;
    fz = tj * (n + 1);
    flux = 5 * fy + 6 * fz;
  }
  __host__ __device__ size_t bytes() const {
    return sizeof(float) * ((size_t)kRing * plane + 4 * kPrimRing * prim_plane + 2 * flux);
  }
};

}  // namespace

// Work is counted in chunks of kChunk planes of a tile, tiles in order; CTA b
// takes chunks [b * each, (b + 1) * each), a march segment per tile it
// touches, so that every CTA of one wave does the same work whatever the
// number of cubes.
template <int NN>
__host__ __device__ constexpr int march_rows() {
  return NN == 20 ? 10 : (NN == 24 ? 8 : (NN == 28 ? 7 : (NN == 32 ? 16 : NN)));
}
struct MarchShape {
  int tj, each, total;  // rows of a tile, chunks per CTA, chunks in all
};

template <int NN, bool VISCOUS, bool PACK, bool NORMS>
__global__ void __launch_bounds__(NN == 32 ? 512 : 256, NN == 32 ? 1 : 2)
    k_flux_march(FluxSplitArgs a, MarchShape sh) {
  constexpr int CVT = NN == 32 ? 3 : (NN >= 16 ? 1 : 2);  // measured there
  extern __shared__ __align__(16) float smem[];
  const int n = NN ? NN : a.ph.n, S = n + 4;
  const int tj = NN ? march_rows<NN>() : sh.tj;
  const MarchLayout L(n, tj);
  float *const ring = smem;
  PrimF *const prims = reinterpret_cast<PrimF *>(ring + kRing * L.plane);
  float *const flux = reinterpret_cast<float *>(prims + kPrimRing * L.prim_plane);

  const int tid = threadIdx.x, NT = blockDim.x;
  const int tiles = n / tj, per_tile = n / kChunk;
  const int u1 = min(sh.total, ((int)blockIdx.x + 1) * sh.each);
#pragma unroll 1
  for (int u = (int)blockIdx.x * sh.each, len; u < u1; u += len) {
  const int tile = u / per_tile, chunk = u - tile * per_tile;
  len = min(per_tile - chunk, u1 - u);
  const int cube = a.cube0 + tile / tiles;
  if (!case_active(a.bt, cube)) continue;  // converged case (uniform per CTA)
  const int j0 = 2 + (tile % tiles) * tj, i0 = 2 + chunk * kChunk, i1 = i0 + len * kChunk;
  const SplitConst z = split_const(a, cube);
  const float inv = a.inv_dx[cube];
  // Mirror buffers: read the current one; stages 1..3 write the other one.
  const int par = mirror_index(a.mir);
  const float *__restrict__ M = a.mir.buf[par];
  float *const Mw = a.RK >= 1 ? a.mir.buf[par ^ 1] : nullptr;
  const size_t cb = cell_index(S, cube, 0, 0, 0);
  const int SS = S * S;
  const int jlo = j0 - 3 < 0 ? 0 : j0 - 3, jhi = j0 + tj + 3 > S ? S : j0 + tj + 3;

  // Column of this thread (idle threads stay on a valid cell).
  const int ncol = tj * n;
  const bool is_cell = tid < ncol;
  const int jl = is_cell ? tid / n : 0, kl = is_cell ? tid - (tid / n) * n : 0;
  const int col = (j0 + jl - jlo) * L.pitch + 5 * (kl + 2);  // in a ring plane
  const int prow = (jl + 1) * L.prim_row + kl + 1;           // in a primitive plane
  const size_t go0 = cb + (size_t)(j0 + jl) * S + (kl + 2);  // cell offset of plane 0
  // pushes of the cell along j and k: offsets (in values) into the neighbour
  // cubes' ghost layers, the same for every plane; 0: none
  ptrdiff_t pushJ = 0, pushK = 0;
  int pI0 = 0, pI1 = 0;
  if (a.push && is_cell) {
    const int j = j0 + jl, k = kl + 2;
    const size_t SSS = (size_t)SS * S;
    auto to = [&](int d, int delta) -> ptrdiff_t {
      return 5 * ((ptrdiff_t)((ptrdiff_t)d - cube) * (ptrdiff_t)SSS + delta);
    };
    const int *pp = a.push + 6 * cube;
    pI0 = pp[0];
    pI1 = pp[1];
    const int dj = j <= 3 ? pp[2] : (j >= n ? pp[3] : 0), dk = k <= 3 ? pp[4] : (k >= n ? pp[5] : 0);
    if (dj > 0) pushJ = to(dj, (j <= 3 ? n : -n) * S);
    if (dk > 0) pushK = to(dk, k <= 3 ? n : -n);
  }

  auto load_plane = [&](int p) {
    if (p < 0 || p >= S) return;
    float *dst = ring + (p % kRing) * L.plane;
    const float *src = M + 5 * (cb + (size_t)p * SS + (size_t)jlo * S);
    const int q = 5 * S / 4, total = (jhi - jlo) * q;  // 16-byte pieces of a row
    for (int w = tid; w < total; w += NT) {
      const int r = w / q, e = w - r * q;
      cp_async16(dst + r * L.pitch + 4 * e, src + 4 * w);
    }
  };
  auto make_prims = [&](int p) {
    PrimF *dst = prims + (p & (kPrimRing - 1)) * L.prim_plane;
    const float *src = ring + (p % kRing) * L.plane + (j0 - 1 - jlo) * L.pitch + 5;
    for (int w = tid; w < L.prim_plane; w += NT) {
      const int r = w / L.prim_row, e = w - r * L.prim_row;
      dst[w] = prim_split(z, src + r * L.pitch + 5 * e);
    }
  };
  auto code_at = [&](int p) -> unsigned { return __ldg(a.codes + go0 + (size_t)p * SS); };

  // One face of axis ax: order, left and right states.
  auto states = [&](int ord, const float *base, int stride, float *ML, float *MR) {
    auto ld = [&](int d, int v) -> float { return base[stride * d + v]; };
    recon_split(ord, ld, ML, MR);
  };

  // The first planes, and the segment's first i-face (seen from its plus
  // side); a segment inside the cube needs one plane more below it.
  const bool inner = i0 > 2;
  for (int p = inner ? i0 - 3 : i0 - 2; p <= i0 + (inner ? 3 : 4); ++p) load_plane(p);
  cp_async_wait_all();
  __syncthreads();
  float Fx[6];  // i-face below the current cell: five fluxes, pressure
  if (is_cell) {
    float ML[5], MR[5];
    const int ord = code_back(code_at(i0), 0);
    const float *c = ring + col;
    auto ld = [&](int d, int v) -> float { return c[((i0 + d + 2 * kRing) % kRing) * L.plane + v]; };
    recon_split(ord, ld, ML, MR);
    if (PACK) {
      float2 ML2[5], MR2[5], F2[5], dP2;
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        ML2[v] = f2(ML[v]);
        MR2[v] = f2(MR[v]);
      }
      face_flux_delta2<0>(ML2, MR2, z.ef, z.rho0, z.P0, F2, dP2);
#pragma unroll
      for (int v = 0; v < 5; ++v) Fx[v] = F2[v].x;
      Fx[5] = dP2.x;
    } else {
      face_flux_delta<0>(ML, MR, z.ef, z.rho0, z.P0, Fx, Fx[5]);
    }
  }
  make_prims(i0 - 1);
  make_prims(i0);
  if (inner) {
    __syncthreads();
    load_plane(i0 + 4);
    cp_async_wait_all();
    __syncthreads();
  }

  double s5[8] = {0, 0, 0, 0, 0, 0, 0, 0}, s8 = 0;
  unsigned c0 = code_at(i0), c1 = code_at(i0 + 1), c2 = code_at(i0 + 2);
#pragma unroll 1
  for (int i = i0; i < i1; i += 2) {
    // Ring offsets of planes i-2 .. i+4.
    int off[kRing];
#pragma unroll
    for (int d = 0; d < kRing; ++d) off[d] = ((i - 2 + d) % kRing) * L.plane;
    // Start moving the next step's FP64 rows into L2 (a line holds three
    // cells of doubles, six of floats).
    if (is_cell && i + 2 < i1) {
#pragma unroll
      for (int q = 2; q < 4; ++q) {
        const size_t go = go0 + (size_t)(i + q) * SS;
        if (kl % 3 == 0) {
          prefetch_l2(a.U1_ + 5 * go);
          prefetch_l2(a.U1 + 5 * go);
        }
        if (kl % 6 == 0) prefetch_l2(a.D2 + 5 * go);
      }
    }
    make_prims(i + 1);
    make_prims(i + 2);
    // Faces of the two planes (lanes .x and .y): low y and z faces of planes
    // i, i + 1 into shared memory, i-faces above planes i, i + 1 in registers.
    auto pair = [&](auto ax_, const float *b0, const float *b1, int stride, int o0, int o1,
                    float *d0, float *d1, int nf) {
      constexpr int AX = decltype(ax_)::value;
      float MLa[5], MRa[5], MLb[5], MRb[5];
      states(o0, b0, stride, MLa, MRa);
      states(o1, b1, stride, MLb, MRb);
      if (PACK) {
        float2 ML2[5], MR2[5], F2[5], dP2;
#pragma unroll
        for (int v = 0; v < 5; ++v) {
          ML2[v] = make_float2(MLa[v], MLb[v]);
          MR2[v] = make_float2(MRa[v], MRb[v]);
        }
        face_flux_delta2<AX>(ML2, MR2, z.ef, z.rho0, z.P0, F2, dP2);
#pragma unroll
        for (int v = 0; v < 5; ++v) {
          d0[v * nf] = F2[v].x;
          d1[v * nf] = F2[v].y;
        }
        if (AX != 1) {
          d0[5 * nf] = dP2.x;
          d1[5 * nf] = dP2.y;
        }
      } else {
        float F[5], dP;
        face_flux_delta<AX>(MLa, MRa, z.ef, z.rho0, z.P0, F, dP);
#pragma unroll
        for (int v = 0; v < 5; ++v) d0[v * nf] = F[v];
        if (AX != 1) d0[5 * nf] = dP;
        face_flux_delta<AX>(MLb, MRb, z.ef, z.rho0, z.P0, F, dP);
#pragma unroll
        for (int v = 0; v < 5; ++v) d1[v * nf] = F[v];
        if (AX != 1) d1[5 * nf] = dP;
      }
    };
    const float *const p0 = ring + off[2] + col, *const p1 = ring + off[3] + col;
    float *const g0 = flux, *const g1 = flux + L.flux;
    // The column's own faces; then the tile's far faces (y beyond the last
    // row, z beyond the last k), whose turn goes round the warps.
    const int ex = tid - 32 * ((i >> 1) % (NT / 32)) ;
    const int far = ex >= 0 ? ex : ex + NT;
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
      int j = jl, k = kl;
      if (pass == 1) {
        if (far >= n + tj) break;
        j = far < n ? tj : far - n;
        k = far < n ? far : n;
      }
      const int dj = (j - jl), dk = (k - kl);
      const float *const b0 = p0 + dj * L.pitch + 5 * dk, *const b1 = p1 + dj * L.pitch + 5 * dk;
      unsigned e0 = c0, e1 = c1;
      if (pass == 1) {
        const ptrdiff_t o = (ptrdiff_t)(go0 + (size_t)i * SS) + dj * S + dk;
        e0 = __ldg(a.codes + o);
        e1 = __ldg(a.codes + o + SS);
      }
      if (pass == 0 ? is_cell : far < n) {
        const int f = j * n + k;
        const bool end = pass == 1 && j0 + tj == n + 2;  // the cube's last y face
        pair(std::integral_constant<int, 1>(), b0, b1, L.pitch,
             end ? code_fwd(e0, 1) : code_back(e0, 1), end ? code_fwd(e1, 1) : code_back(e1, 1),
             g0 + f, g1 + f, L.fy);
      }
      if (pass == 0 ? is_cell : far >= n) {
        const int f = 5 * L.fy + j * (n + 1) + k;
        pair(std::integral_constant<int, 2>(), b0, b1, 5,
             pass ? code_fwd(e0, 2) : code_back(e0, 2), pass ? code_fwd(e1, 2) : code_back(e1, 2),
             g0 + f, g1 + f, L.fz);
      }
    }
    float Fa[6], Fb[6];     // i-faces above planes i and i + 1
    float own[2][6];        // the minus-side cell's view where it differs (rare)
    unsigned second = 0;
    if (is_cell) {
      const bool last = i + 2 == n + 2;  // the cube's last face: seen from its minus side
      const float *const c = ring + col;
      float MLa[5], MRa[5], MLb[5], MRb[5];
      auto lda = [&](int d, int v) -> float { return c[off[3 + d] + v]; };
      auto ldb = [&](int d, int v) -> float { return c[off[4 + d] + v]; };
      recon_split(code_back(c1, 0), lda, MLa, MRa);
      recon_split(last ? code_fwd(c2, 0) : code_back(c2, 0), ldb, MLb, MRb);
      if (PACK) {
        float2 ML2[5], MR2[5], F2[5], dP2;
#pragma unroll
        for (int v = 0; v < 5; ++v) {
          ML2[v] = make_float2(MLa[v], MLb[v]);
          MR2[v] = make_float2(MRa[v], MRb[v]);
        }
        face_flux_delta2<0>(ML2, MR2, z.ef, z.rho0, z.P0, F2, dP2);
#pragma unroll
        for (int v = 0; v < 5; ++v) {
          Fa[v] = F2[v].x;
          Fb[v] = F2[v].y;
        }
        Fa[5] = dP2.x;
        Fb[5] = dP2.y;
      } else {
        face_flux_delta<0>(MLa, MRa, z.ef, z.rho0, z.P0, Fa, Fa[5]);
        face_flux_delta<0>(MLb, MRb, z.ef, z.rho0, z.P0, Fb, Fb[5]);
      }
      if (c0 & (1u << 13)) {
        recon_split(code_fwd(c1, 0), lda, MLa, MRa);
        face_flux_delta<0>(MLa, MRa, z.ef, z.rho0, z.P0, own[0], own[0][5]);
        second |= 1u;
      }
      if (!last && (c1 & (1u << 13))) {
        recon_split(code_fwd(c2, 0), ldb, MLb, MRb);
        face_flux_delta<0>(MLb, MRb, z.ef, z.rho0, z.P0, own[1], own[1][5]);
        second |= 2u;
      }
    }
    __syncthreads();  // fluxes and primitives complete; planes i-2, i-1 are free
    if (i + 2 < i1) {
      load_plane(i + 5);
      load_plane(i + 6);
    }
    unsigned c3 = 0, c4 = 0;  // the next step's codes
    if (i + 2 < i1) {
      c3 = code_at(i + 3);
      c4 = code_at(i + 4);
    }
    if (is_cell) {
#pragma unroll 1
      for (int q = 0; q < 2; ++q) {
        SplitLevels lv;
        float src[5];
        split_load(a, go0 + (size_t)(i + q) * SS, lv);
        split_source<CVT>(lv, src);

        const int p = i + q;
        const unsigned cc = q == 0 ? c0 : c1;
        const float *const g = q == 0 ? g0 : g1;
        const float *const qm = q == 0 ? p0 : p1;
        float acc[5], dPdx, dPdz;
        {
          float Ff[6];
#pragma unroll
          for (int v = 0; v < 6; ++v) Ff[v] = Fa[v];
          if (second & (1u << q)) {
#pragma unroll
            for (int v = 0; v < 6; ++v) Ff[v] = own[q][v];
          }
#pragma unroll
          for (int v = 0; v < 5; ++v) acc[v] = __fmul_rn(Ff[v] - Fx[v], inv);
          dPdx = Ff[5] - Fx[5];
        }
        {
          const float *const lo = g + jl * n + kl, *const hi = lo + n;
          float Fbv[5], Ffv[5], dummy;
#pragma unroll
          for (int v = 0; v < 5; ++v) {
            Fbv[v] = lo[v * L.fy];
            Ffv[v] = hi[v * L.fy];
          }
          if ((cc & (1u << 14)) && j0 + jl <= n) {
            float ML[5], MR[5];
            states(code_fwd(__ldg(a.codes + go0 + (size_t)p * SS + S), 1), qm + L.pitch, L.pitch,
                   ML, MR);
            face_flux_delta<1>(ML, MR, z.ef, z.rho0, z.P0, Ffv, dummy);
          }
#pragma unroll
          for (int v = 0; v < 5; ++v) acc[v] = __fmaf_rn(Ffv[v] - Fbv[v], inv, acc[v]);
        }
        {
          const float *const lo = g + 5 * L.fy + jl * (n + 1) + kl, *const hi = lo + 1;
          float Fbv[6], Ffv[6];
#pragma unroll
          for (int v = 0; v < 6; ++v) {
            Fbv[v] = lo[v * L.fz];
            Ffv[v] = hi[v * L.fz];
          }
          if ((cc & (1u << 15)) && kl + 1 < n) {
            float ML[5], MR[5];
            states(code_fwd(__ldg(a.codes + go0 + (size_t)p * SS + 1), 2), qm + 5, 5, ML, MR);
            face_flux_delta<2>(ML, MR, z.ef, z.rho0, z.P0, Ffv, Ffv[5]);
          }
#pragma unroll
          for (int v = 0; v < 5; ++v) acc[v] = __fmaf_rn(Ffv[v] - Fbv[v], inv, acc[v]);
          dPdz = Ffv[5] - Fbv[5];
        }
        const PrimF *const q0 = prims + ((p - 1) & (kPrimRing - 1)) * L.prim_plane + prow;
        const PrimF *const q1 = prims + (p & (kPrimRing - 1)) * L.prim_plane + prow;
        const PrimF *const q2 = prims + ((p + 1) & (kPrimRing - 1)) * L.prim_plane + prow;
        auto P = [&](int di, int dj, int dk) -> const PrimF & {
          return (di < 0 ? q0 : (di == 0 ? q1 : q2))[dj * L.prim_row + dk];
        };
        const size_t go = go0 + (size_t)p * SS;
        // i-pushes: planes 2, 3 and n, n + 1
        ptrdiff_t pushI = 0;
        {
          const int d = p <= 3 ? pI0 : (p >= n ? pI1 : 0);
          if (d > 0)
            pushI = 5 * ((ptrdiff_t)(d - cube) * ((ptrdiff_t)SS * S) +
                         (ptrdiff_t)(p <= 3 ? n : -n) * SS);
        }
        split_cell<VISCOUS, NORMS, CVT>(a, z, cube, inv, P, qm, acc, lv.x, src, dPdx, dPdz, go, (cc & 1u) != 0, Mw, s5,
                            [&](auto *U, const auto *un) {
                              auto *u = U + 5 * go;
                              if (pushI) {
#pragma unroll
                                for (int r = 0; r < 5; ++r) u[pushI + r] = un[r];
                              }
                              if (pushJ) {
#pragma unroll
                                for (int r = 0; r < 5; ++r) u[pushJ + r] = un[r];
                              }
                              if (pushK) {
#pragma unroll
                                for (int r = 0; r < 5; ++r) u[pushK + r] = un[r];
                              }
                            });
        if (NORMS && NN == 8 && q == 0) {
          norm_exchange(s5, tid & 31);
          s8 = s5[0];
#pragma unroll
          for (int v = 0; v < 8; ++v) s5[v] = 0;
        }
#pragma unroll
        for (int v = 0; v < 6; ++v) {
          Fx[v] = Fa[v];
          Fa[v] = Fb[v];
        }
      }
    }
    // Norm and force partial sums of the step's planes (stage 3), through the
    // flux area: each warp's sums, then the warps' in order.  For n = 8 each
    // warp adds the two planes' sums, as the tile kernel's warps do.
    if (NORMS) {
      __syncthreads();  // the cells have read the fluxes
      double *red = reinterpret_cast<double *>(flux);
      const int m = norm_exchange(s5, tid & 31);
      if ((tid & 31) < 8 && m < 7) red[(tid >> 5) * 7 + m] = NN == 8 ? s8 + s5[0] : s5[0];
      __syncthreads();
      if (tid < 7) {
        double v = 0;
        for (int w = 0; w < NT / 32; ++w) v += red[w * 7 + tid];
        a.partials[(size_t)(tile * per_tile + (i - 2) / kChunk) * 7 + tid] = v;
      }
#pragma unroll
      for (int v = 0; v < 8; ++v) s5[v] = 0;
    }
    c0 = c2;
    c1 = c3;
    c2 = c4;
    cp_async_wait_all();
    __syncthreads();  // planes i+5, i+6 have arrived; fluxes may be written again
  }
  }  // march segments of this CTA
}

// Rows of a tile: the whole cross-section where two CTAs fit an SM, else the
// widest divisor of n that leaves room for two (one of 16 rows for n = 32,
// whose eight rows are a little too wide for two); 0: none fits.
static int march_threads(int n, int tj) { return (tj * n + 31) & ~31; }

static int march_tj(int n) {
  if (n < 8) return 0;
  if (n == 32) return 16;

  for (int tj = n; tj >= 1; --tj) {
    if (n % tj) continue;
    if (march_threads(n, tj) <= 256 && march_threads(n, tj) >= n + tj && MarchLayout(n, tj).bytes() <= 112 * 1024) return tj;
  }
  return 0;
}

bool flux_march_fits(int n) { return march_tj(n) > 0; }

int flux_march_blocks(int n, int ncubes) { return ncubes * (n / march_tj(n)) * (n / kChunk); }

template <int NN, bool VISCOUS, bool PACK, bool NORMS>
static cudaError_t launch_march_k(const FluxSplitArgs &a, const MarchShape &sh, unsigned grid,
                                  unsigned threads, size_t smem, cudaStream_t s) {
  const cudaError_t e = cudaFuncSetAttribute(  // (a compile-time edge has one need)
      k_flux_march<NN, VISCOUS, PACK, NORMS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
      NN ? (int)smem : kMaxSmem);
  if (e != cudaSuccess) return e;
  k_flux_march<NN, VISCOUS, PACK, NORMS><<<grid, threads, smem, s>>>(a, sh);
  return cudaGetLastError();
}

template <int NN, bool PACK>
static cudaError_t launch_march_n(const FluxSplitArgs &a, const MarchShape &sh, unsigned grid,
                                  unsigned threads, size_t smem, cudaStream_t s) {
  if (a.ph.mu_L != 0.0)
    return a.RK == 3 ? launch_march_k<NN, true, PACK, true>(a, sh, grid, threads, smem, s)
                     : launch_march_k<NN, true, PACK, false>(a, sh, grid, threads, smem, s);
  return a.RK == 3 ? launch_march_k<NN, false, PACK, true>(a, sh, grid, threads, smem, s)
                   : launch_march_k<NN, false, PACK, false>(a, sh, grid, threads, smem, s);
}

cudaError_t launch_flux_march(const FluxSplitArgs &a, int ncubes, cudaStream_t s) {
  const int n = a.ph.n, tj = march_tj(n);
  if (tj == 0) return cudaErrorInvalidValue;
  if (ncubes <= 0) return cudaSuccess;
  const MarchLayout L(n, tj);
  const unsigned threads = march_threads(n, tj);
  const int per_sm = std::max<int>(
      1, std::min<int>(512 / threads, (int)(kMaxSmem / (L.bytes() + 1024))));
  const long long total = (long long)ncubes * (n / tj) * (n / kChunk), slots = 152LL * per_sm;
  if (total > INT32_MAX - slots) return cudaErrorInvalidValue;
  const int each = (int)((total + slots - 1) / slots);
  const MarchShape sh{tj, each, (int)total};
  const unsigned grid = (unsigned)((total + each - 1) / each);
  // Faces in packed pairs where 8 divides n, one at a time elsewhere (where
  // the 4^3 tiles evaluated them so) or on request.
  if (a.form == 1 && n % 8 == 0) {
    if (n == 8) return launch_march_n<8, true>(a, sh, grid, threads, L.bytes(), s);
    if (n == 16) return launch_march_n<16, true>(a, sh, grid, threads, L.bytes(), s);
    if (n == 24) return launch_march_n<24, true>(a, sh, grid, threads, L.bytes(), s);
    if (n == 32) return launch_march_n<32, true>(a, sh, grid, threads, L.bytes(), s);
    return launch_march_n<0, true>(a, sh, grid, threads, L.bytes(), s);
  }
  if (n == 8) return launch_march_n<8, false>(a, sh, grid, threads, L.bytes(), s);
  if (n == 12) return launch_march_n<12, false>(a, sh, grid, threads, L.bytes(), s);
  if (n == 20) return launch_march_n<20, false>(a, sh, grid, threads, L.bytes(), s);
  if (n == 28) return launch_march_n<28, false>(a, sh, grid, threads, L.bytes(), s);
  if (n == 32) return launch_march_n<32, false>(a, sh, grid, threads, L.bytes(), s);
  return launch_march_n<0, false>(a, sh, grid, threads, L.bytes(), s);
}

}  // namespace bcmg
