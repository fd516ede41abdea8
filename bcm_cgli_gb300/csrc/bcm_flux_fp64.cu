// FP64 residual + pointwise-preconditioned increment for one RK stage.
//
// Replaces the cube loop of BCM_Flux_XYZ_Viscous_Runge_kutta
// (BCM_Flux_XYZ_Viscous_Runge_kutta.cpp:326-2411): for every interior cell
// it forms the BDF2 source, the upwind-biased inviscid flux balance, the
// viscous flux balance and Rku1 = dTau * D * Rk (0 on non-fluid cells), and
// the force integrands in Residual1 on non-fluid cells.  The RK combination
// itself runs in bcm_rk.cu once all increments exist (the reference also
// runs it after its cube loop, :2417-2599: cells read each other's old
// state).
//
// GB300 design: FP64 runs at 1/64 of the FP32 rate on this part, so the
// kernel does less FP64 work than the reference without changing a single
// rounding:
//  * one CTA per T^3 tile of a cube; the primitive variables (u,v,w,T) of
//    the tile plus a one-cell halo are formed once into shared memory
//    instead of 18 times per cell (the reference converts each neighbour
//    inside every cell's body, :1729-1895);
//  * each inviscid face flux is evaluated once and used by both cells that
//    share the face whenever both cells pick the same reconstruction order
//    (then their left/right states are identical bit for bit); only faces
//    next to non-fluid flags or cube edges get two evaluations;
//  * divisions and square roots, which were over 40% of the FP64 pipe's
//    work, and about two thirds of the multiplications run on the integer
//    pipes (bcm_fp64_int.cuh: the same correctly rounded results, several
//    quotients sharing one reciprocal);
//  * factors that are powers of two are exact, so c*x + y with such a c is
//    one fused multiply-add with the reference's bits, and common factors
//    are applied once at the end of a sum;
//  * one CTA of 16 warps per SM, all in the same phase, and loops instead of
//    unrolled components: the integer sequences are long, and more resident
//    CTAs or unrolled copies miss the instruction cache (4^3 boxes: 4.1 ms
//    for seven CTAs of two warps in an SM, 2.1 ms for one CTA of seven boxes;
//    8^3: 1.95 ms unrolled, 1.84 ms in loops; 0.88 M cells, viscous);
//  * where an operand is out of the integer routines' range the face, cell
//    or primitive is redone by the reference's own expressions;
//  * everything else keeps the reference's expression order, and this
//    translation unit is compiled with --fmad=false, so every value equals
//    the reference's (checked against the C oracle in tests/).
// One launch over 0.88 M viscous cells in 16^3 cubes: 4.95 -> 1.84 ms (5.6 ->
// 2.1 ns per cell).  What bounds it now: the FP64 pipe is 71% busy, nearly
// all additions and fused multiply-adds, with four warps per scheduler to
// hide its latency; moving the remaining products too was slower (their
// chains are serial).
#include <cuda_runtime.h>

#include <algorithm>

#include "bcm_common.cuh"
#include "bcm_fp64_int.cuh"
#include "bcm_kernels.h"

namespace bcmg {

struct Prim {
  double U, V, W, T;  // T = P/(rho*R): the neighbour form (:1734)
};

// The tiles of a CTA: `groups` boxes of ti x tj x tk cells, each inside one
// cube.  Cubes whose edge is a multiple of 8 take one 8^3 box (compile-time
// sizes); others the best box of divisors of n (flux_shape).
constexpr int kFluxThreads = 512;
struct Shape888 {
  static constexpr int ti = 8, tj = 8, tk = 8, groups = 1;
};
struct ShapeAny {
  int ti, tj, tk, groups;
};
// Sizes that follow from a shape, and the shared memory of a CTA:
//  * the faces' values, value-major per axis: five fluxes and the pressure in
//    the plus-side cell's view (the minus-side cell's for the box's last
//    face);
//  * kSecond slots for the minus-side cell's view of faces where its
//    reconstruction order differs, and each face's slot;
//  * the primitives and centre temperatures;
//  * work columns of the face phase (one double per thread and row).
constexpr int kSecond = 256, kCols = 22;
template <typename Sh>
__host__ __device__ inline int box_cells(const Sh &s) { return s.ti * s.tj * s.tk; }
template <typename Sh>
__host__ __device__ inline int box_prims(const Sh &s) {
  return (s.ti + 2) * (s.tj + 2) * (s.tk + 2);
}
template <typename Sh>
__host__ __device__ inline int box_faces(const Sh &s, int ax) {
  return box_cells(s) + (ax == 0 ? s.tj * s.tk : (ax == 1 ? s.ti * s.tk : s.ti * s.tj));
}
template <typename Sh>
__host__ __device__ inline int box_faces(const Sh &s) {
  return box_faces(s, 0) + box_faces(s, 1) + box_faces(s, 2);
}
template <typename Sh>
__host__ __device__ inline size_t flux_smem(const Sh &s) {
  const size_t faces = (size_t)s.groups * box_faces(s);
  const size_t prims = s.groups * (sizeof(Prim) * box_prims(s) + sizeof(double) * box_cells(s));
  const size_t cols = sizeof(double) * kCols * kFluxThreads;
  return 6 * sizeof(double) * (faces + kSecond) + prims + cols + sizeof(uint16_t) * faces + 16;
}

// Division by a constant.
#define BCMG_BY(value) \
  RecipConst<__builtin_bit_cast(uint64_t, (double)(value))>::get()

__device__ __forceinline__ Prim prim_of(double q0, double q1, double q2, double q3,
                                        double q4) {
  Prim p;
  double rho = q0;
  p.U = q1 / rho;
  p.V = q2 / rho;
  p.W = q3 / rho;
  double P = (q4 - 0.5 * rho * (p.U * p.U + p.V * p.V + p.W * p.W)) * (BCMG_K - 1);
  p.T = P / (rho * BCMG_R);
  return p;
}

// Viscous face (BCM_Flux...cpp:1906-2265).  c/o are the centre and normal
// neighbour primitives, Tc the centre temperature in its P/rho/R form,
// a0..a3 / b0..b3 the terms of the two transverse central differences in the
// reference's (a + b - c - d) order (transverse axes in x<y<z order).
template <int AX, bool FWD>
__device__ __forceinline__ void visc_face(double mu_L, double T0, double Tc, const Prim &c,
                                          const Prim &o, double inv, const Prim &a0,
                                          const Prim &a1, const Prim &a2, const Prim &a3,
                                          const Prim &b0, const Prim &b1, const Prim &b2,
                                          const Prim &b3, double *L) {
  double Tm = 0.5 * (Tc + o.T);
  double temp = Tm / T0;
  double mu_E = mu_L * temp * sqrt(temp) * (T0 + 110.) / (Tm + 110.);
  double gn[4];
  if (FWD) {
    gn[0] = (o.U - c.U) * inv; gn[1] = (o.V - c.V) * inv;
    gn[2] = (o.W - c.W) * inv; gn[3] = (o.T - Tc) * inv;
  } else {
    gn[0] = (c.U - o.U) * inv; gn[1] = (c.V - o.V) * inv;
    gn[2] = (c.W - o.W) * inv; gn[3] = (Tc - o.T) * inv;
  }
  double ga[3], gb[3];
  ga[0] = (a0.U + a1.U - a2.U - a3.U) / 4 * inv;
  ga[1] = (a0.V + a1.V - a2.V - a3.V) / 4 * inv;
  ga[2] = (a0.W + a1.W - a2.W - a3.W) / 4 * inv;
  gb[0] = (b0.U + b1.U - b2.U - b3.U) / 4 * inv;
  gb[1] = (b0.V + b1.V - b2.V - b3.V) / 4 * inv;
  gb[2] = (b0.W + b1.W - b2.W - b3.W) / 4 * inv;
  double d[3][3];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    d[AX][m] = gn[m];
    d[AX == 0 ? 1 : 0][m] = ga[m];
    d[AX == 2 ? 1 : 2][m] = gb[m];
  }
  const double du_dx = d[0][0], dv_dx = d[0][1], dw_dx = d[0][2];
  const double du_dy = d[1][0], dv_dy = d[1][1], dw_dy = d[1][2];
  const double du_dz = d[2][0], dv_dz = d[2][1], dw_dz = d[2][2];
  double Um = 0.5 * (c.U + o.U), Vm = 0.5 * (c.V + o.V), Wm = 0.5 * (c.W + o.W);
  double div = du_dx + dv_dy + dw_dz;
  double s1, s2, s3;
  if (AX == 0) {
    s1 = mu_E * (2 * du_dx - 2.0 / 3.0 * div);
    s2 = mu_E * (du_dy + dv_dx);
    s3 = mu_E * (du_dz + dw_dx);
  } else if (AX == 1) {
    s1 = mu_E * (du_dy + dv_dx);
    s2 = mu_E * (2 * dv_dy - 2.0 / 3.0 * div);
    s3 = mu_E * (dv_dz + dw_dy);
  } else {
    s1 = mu_E * (du_dz + dw_dx);
    s2 = mu_E * (dv_dz + dw_dy);
    s3 = mu_E * (2 * dw_dz - 2.0 / 3.0 * div);
  }
  L[0] = s1;
  L[1] = s2;
  L[2] = s3;
  L[3] = Um * s1 + Vm * s2 + Wm * s3 + mu_E * BCMG_CV * BCMG_K * gn[3] / (BCMG_PR);
}


// Primitives of one cell with the divisions on the integer pipes; Tc is the
// centre temperature as the viscous block forms it, P/rho/R (:1841).
__device__ __forceinline__ Prim prim_int(double q0, double q1, double q2, double q3, double q4,
                                         double &Tc) {
  IntFp o;
  Prim p;
  const Recip k = o.recip(q0);
  p.U = o.div(q1, k);
  p.V = o.div(q2, k);
  p.W = o.div(q3, k);
  const double VV = p.U * p.U + p.V * p.V + p.W * p.W;
  const double P = fma64(-0.5, q0 * VV, q4) * (BCMG_K - 1);
  p.T = o.div(P, o.recip(q0 * BCMG_R));
  Tc = o.div(o.div(P, k), BCMG_BY(BCMG_R));
  if (!o.ok) {
    p = prim_of(q0, q1, q2, q3, q4);
    const double VVr = p.U * p.U + p.V * p.V + p.W * p.W;
    Tc = (q4 - 0.5 * q0 * VVr) * (BCMG_K - 1) / q0 / BCMG_R;
  }
  return p;
}

// One view of a face by the reference's own expressions (recon, face_flux),
// for operands out of the integer routines' range; it loads the stencil
// again (values kept for it would spill the common path).
__device__ __noinline__ void face_ref(int ax, int ord, const double *base, ptrdiff_t stride,
                                      double e, double *dst, int nf) {
  double ML[5], MR[5], F[5], dP;
  auto ld = [&](int d, int v) -> double { return __ldg(base + 5 * stride * d + v); };
  recon<double>(ord, ld, ML, MR);
  if (ax == 0) face_flux<0, double>(ML, MR, e, F, dP);
  else if (ax == 1) face_flux<1, double>(ML, MR, e, F, dP);
  else face_flux<2, double>(ML, MR, e, F, dP);
#pragma unroll
  for (int v = 0; v < 5; ++v) dst[v * nf] = F[v];
  dst[5 * nf] = dP;
}

// A constant factor of a product.
#define BCMG_TIMES(value) const_factor<__builtin_bit_cast(uint64_t, (double)(value))>()

// recon() (bcm_common.cuh) with the fifth-order products on the integer
// pipes: the raw values' small-integer multiples and the final 1/60.
template <typename Ld>
__device__ __forceinline__ void recon_int(IntFp &o, int ord, Ld ld, double *col) {
  if (ord != 5) {
    double ML[5], MR[5];
    recon<double>(ord, ld, ML, MR);
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      col[2 * v * kFluxThreads] = ML[v];
      col[(2 * v + 1) * kFluxThreads] = MR[v];
    }
    return;
  }
#pragma unroll 1
  for (int v = 0; v < 5; ++v) {
    const Factor b = o.plain(ld(-2, v)), c = o.plain(ld(-1, v)), d = o.plain(ld(0, v)),
                 f = o.plain(ld(1, v));
    const double l = fma64(2.0, ld(-3, v), -o.times<13>(b)) + o.times<47>(c) + o.times<27>(d) -
                     o.times<3>(f);
    const double r = fma64(2.0, ld(2, v), -o.times<3>(b) + o.times<27>(c) + o.times<47>(d) -
                                              o.times<13>(f));
    col[2 * v * kFluxThreads] = o.mul(BCMG_TIMES(1. / 60), l);
    col[(2 * v + 1) * kFluxThreads] = o.mul(BCMG_TIMES(1. / 60), r);
  }
}

// face_flux (bcm_common.cuh) with the divisions, roots and most products on
// the integer pipes and exact power-of-two factors folded.  The axis is a
// run-time value and the sides and components are loops over the thread's
// work column (rows: 0..9 left and right values in turn; 10..13 and 14..17
// velocity and enthalpy of the sides; 18..21 their averages): the code has to
// stay in the instruction cache (unrolled, it was 5% slower and used 200
// bytes of spills).
__device__ __forceinline__ void face_int(IntFp &o, int ax, double *col, double e, double *F,
                                         double &dP) {
  const double K = BCMG_K;
  auto at = [&](int row) -> double & { return col[row * kFluxThreads]; };
  double PL = 0, PR = 0, EL = 0, ER = 0, sL = 0, sR = 0;
#pragma unroll 1
  for (int s = 0; s < 2; ++s) {
    const double r = at(s);
    const Recip k = o.recip(r);
    double VV = 0;
#pragma unroll 1
    for (int m = 0; m < 3; ++m) {
      const double v = o.div(at(2 + 2 * m + s), k);
      at(10 + 4 * s + m) = v;
      const double vv = o.mul(v, v);
      VV = m == 0 ? vv : VV + vv;
    }
    const double rV = o.mul(r, VV);  // twice 0.5 rho VV
    const double P = o.mul(BCMG_TIMES(BCMG_K - 1), fma64(-0.5, rV, at(8 + s)));
    at(13 + 4 * s) = fma64(0.5, VV, o.div(o.div(K * P, k), BCMG_BY(BCMG_K - 1)));
    PL = PR; PR = P;
    EL = ER; ER = fma64(0.5, rV, 3.5 * P);
    sL = sR; sR = o.root(r);
  }
  const Recip kS = o.recip(sL + sR);
  const double rho = o.root(o.mul(at(0), at(1)));
  double VV = 0;
#pragma unroll 1
  for (int m = 0; m < 4; ++m) {
    const double v = o.div(o.mul(sL, at(10 + m)) + o.mul(sR, at(14 + m)), kS);
    at(18 + m) = v;
    if (m < 3) {
      const double vv = o.mul(v, v);
      VV = m == 0 ? vv : VV + vv;
    }
  }
  const double H = at(21);
  const double C = o.mul(BCMG_TIMES(BCMG_K - 1), fma64(-0.5, VV, H));
  const Recip kC = o.recip(C);
  const double beta = o.floor_at(o.div(VV, kC), e);
  const double un = at(18 + ax), unL = at(10 + ax), unR = at(14 + ax);
  const double omb = 1 - beta;
  const double t2 = (1 + beta) * un;  // twice temp
  const double S2 = o.root(fma64(4.0, beta * C, un * un * omb * omb));  // twice Sp
  const Recip kSp = o.recip(S2);
  const double dp = PR - PL, du = unR - unL;
  const double temp1 = o.div(o.div(o.div(dp, o.recip(rho)), o.recip(beta)), kC);
  const double tS = o.div(t2, kSp);
  const double x3 = o.div(omb * un * t2, kSp);  // twice temp3
  const double an = fabs(un);
  const double deltaU = (fma64(0.5, S2 - x3, -(beta * an))) * temp1 + tS * du;
  const double deltaP = tS * dp + fma64(0.5, x3, fma64(0.5, S2, -an)) * rho * du;
  const double dr = deltaU * rho;
  F[0] = o.half((o.mul(at(0), unL) + o.mul(at(1), unR)) - (o.mul(an, at(1) - at(0)) + dr));
#pragma unroll 1
  for (int m = 0; m < 3; ++m) {
    double s = o.mul(unL, o.mul(at(0), at(10 + m)));
    double d = o.mul(an, at(3 + 2 * m) - at(2 + 2 * m)) + o.mul(dr, at(18 + m));
    const double r = o.mul(unR, o.mul(at(1), at(14 + m)));
    if (ax == m) {
      s = s + PL + r + PR;
      d = d + deltaP;
    } else {
      s = s + r;
    }
    at(18 + m) = o.half(s - d);
  }
  const double F5 = o.mul(an, at(9) - at(8)) + o.mul(dr, H) + deltaP * un;
  F[4] = o.half(o.mul(unL, EL) + o.mul(unR, ER) - F5);
  dP = o.half(PL + PR);
#pragma unroll
  for (int m = 0; m < 3; ++m) F[1 + m] = at(18 + m);
}

// The tile's primitives as [cell][u, v, w, T].
struct ViscIn {
  const double *c;  // the cell
  double mu_L, T0p, inv, invq, Tc;
  Recip by2T0;
};

// visc_face with the divisions, root and products on the integer pipes, for
// the face towards the neighbour at offset sn (doubles, signed: side) of
// axis ax.  One copy of the code for the six faces of a cell: the axis and
// side are run-time values (six unrolled copies miss the instruction
// cache).  sa and sb are the strides of the other axes, lower axis first.
__device__ __forceinline__ void visc_int(IntFp &o, const ViscIn &z, int ax, bool fwd, int sn,
                                         int sa, int sb, double *L) {
  const int ia = ax == 0 ? 1 : 0, ib = ax == 2 ? 1 : 2;
  const double *c = z.c, *p = c + sn;
  const double Ts = z.Tc + p[3];
  const double temp = o.div(Ts, z.by2T0);
  const Factor fmu = o.factor(
      o.div(o.mul(o.mul(o.factor(z.mu_L), temp), o.root(temp)) * z.T0p,
            o.recip(fma64(0.5, Ts, 110.))));
  const Factor finv = o.factor(z.inv), finvq = o.factor(z.invq);
  // normal differences, plus side less minus side
  const double sg = fwd ? 1.0 : -1.0;
  auto dn = [&](double x, double y) {  // (x - y) forward, (y - x) backward
    const double d = x - y;
    return d_make(d_hi(d) ^ (d_hi(sg) & 0x80000000u), d_lo(d));
  };
  const double cn = c[ax], ca = c[ia], cb = c[ib], pn = p[ax], pa = p[ia], pb = p[ib];
  const double gn = o.mul(finv, dn(pn, cn)), ga = o.mul(finv, dn(pa, ca)),
               gb = o.mul(finv, dn(pb, cb)), gT = o.mul(finv, dn(p[3], z.Tc));
  // transverse differences of the velocity along ax and of the transverse one
  auto tr = [&](int st, int comp) {
    return o.mul(finvq, c[st + comp] + p[st + comp] - c[comp - st] - p[comp - st]);
  };
  const double an = tr(sa, ax), aa = tr(sa, ia), bn = tr(sb, ax), bb = tr(sb, ib);
  // the divergence in x, y, z order
  const double div = ax == 2 ? aa + bb + gn : gn + aa + bb;
  const double tn = o.mul(fmu, fma64(2.0, gn, -(2.0 / 3.0 * div)));
  const double ta = o.mul(fmu, an + ga), tb = o.mul(fmu, bn + gb);
  const double wn = o.mul(cn + pn, tn), wa = o.mul(ca + pa, ta), wb = o.mul(cb + pb, tb);
  const double w0 = ax == 0 ? wn : wa, w1 = ax == 0 ? wa : (ax == 1 ? wn : wb),
               w2 = ax == 2 ? wn : wb;
  L[0] = ax == 0 ? tn : ta;
  L[1] = ax == 0 ? ta : (ax == 1 ? tn : tb);
  L[2] = ax == 2 ? tn : tb;
  const double heat =
      o.mul(BCMG_TIMES(BCMG_K), o.mul(fmu, BCMG_CV)) * gT;
  L[3] = fma64(0.5, w0 + w1 + w2, o.div(heat, BCMG_BY(BCMG_PR)));
}

// What the cell phase reads of its box and cell.
struct CellIn {
  const double *c;              // primitives of the cell
  int si, sj;                   // strides of the box's i and j (doubles; k: 4)
  // per axis: the values of the backward and forward faces in the cell's view
  // and the distances between them
  const double *Fb[3], *Ff[3];
  int nf[3], nff[3];
  size_t go;                    // cell offset in the state
  int flag;
  double Tc, dx, e, dT, dTau, mu_L, rho0, P0;

  __device__ __forceinline__ const Prim &P(int di, int dj, int dk) const {
    return *reinterpret_cast<const Prim *>(c + di * si + dj * sj + dk * 4);
  }
};

// The cell phase by the reference's own expressions (BDF2 source, viscous
// balance, preconditioner), for operands out of the integer routines' range.
template <bool VISCOUS>
__device__ __noinline__ void cell_ref(const FluxArgs &a, const CellIn &z) {
  const double dx = z.dx, inv = 1. / dx, e = z.e, dT = z.dT, dTau = z.dTau, mu_L = z.mu_L;
  const size_t go = z.go;
  double acc[5], dPdx = 0, dPdz = 0;
  for (int ax = 0; ax < 3; ++ax) {
    for (int v = 0; v < 5; ++v) {
      const double t = (z.Ff[ax][v * z.nff[ax]] - z.Fb[ax][v * z.nf[ax]]) / dx;
      acc[v] = ax == 0 ? t : acc[v] + t;
    }
    if (ax == 0) dPdx = z.Ff[0][5 * z.nff[0]] - z.Fb[0][5 * z.nf[0]];
    if (ax == 2) dPdz = z.Ff[2][5 * z.nff[2]] - z.Fb[2][5 * z.nf[2]];
  }
  const Prim &c = z.P(0, 0, 0);
  double vF[5] = {0, 0, 0, 0, 0};
  if (VISCOUS) {
    const double T0 = z.P0 / z.rho0 / BCMG_R;
    const double Tc = z.Tc;
    double Lb[4], Lf[4], Mb[4], Mf[4], Nb[4], Nf[4];
    visc_face<0, false>(mu_L, T0, Tc, c, z.P(-1, 0, 0), inv, z.P(0, 1, 0), z.P(-1, 1, 0), z.P(0, -1, 0),
                        z.P(-1, -1, 0), z.P(0, 0, 1), z.P(-1, 0, 1), z.P(0, 0, -1), z.P(-1, 0, -1), Lb);
    visc_face<0, true>(mu_L, T0, Tc, c, z.P(1, 0, 0), inv, z.P(0, 1, 0), z.P(1, 1, 0), z.P(0, -1, 0),
                       z.P(1, -1, 0), z.P(0, 0, 1), z.P(1, 0, 1), z.P(0, 0, -1), z.P(1, 0, -1), Lf);
    visc_face<1, false>(mu_L, T0, Tc, c, z.P(0, -1, 0), inv, z.P(1, 0, 0), z.P(1, -1, 0), z.P(-1, 0, 0),
                        z.P(-1, -1, 0), z.P(0, 0, 1), z.P(0, -1, 1), z.P(0, 0, -1), z.P(0, -1, -1), Mb);
    visc_face<1, true>(mu_L, T0, Tc, c, z.P(0, 1, 0), inv, z.P(1, 0, 0), z.P(1, 1, 0), z.P(-1, 0, 0),
                       z.P(-1, 1, 0), z.P(0, 0, 1), z.P(0, 1, 1), z.P(0, 0, -1), z.P(0, 1, -1), Mf);
    visc_face<2, false>(mu_L, T0, Tc, c, z.P(0, 0, -1), inv, z.P(1, 0, 0), z.P(1, 0, -1), z.P(-1, 0, 0),
                        z.P(-1, 0, -1), z.P(0, 1, 0), z.P(0, 1, -1), z.P(0, -1, 0), z.P(0, -1, -1), Nb);
    visc_face<2, true>(mu_L, T0, Tc, c, z.P(0, 0, 1), inv, z.P(1, 0, 0), z.P(1, 0, 1), z.P(-1, 0, 0),
                       z.P(-1, 0, 1), z.P(0, 1, 0), z.P(0, 1, 1), z.P(0, -1, 0), z.P(0, -1, 1), Nf);
#pragma unroll
    for (int v = 1; v < 5; ++v)
      vF[v] = (Lf[v - 1] - Lb[v - 1]) * inv + (Mf[v - 1] - Mb[v - 1]) * inv +
              (Nf[v - 1] - Nb[v - 1]) * inv;
  }

  const double *u = a.U1_ + 5 * go;
  const double *uu = a.U1 + 5 * go;
  const double *uq = a.U1q + 5 * go;
  const int IF = z.flag;
  double Rk[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    double Rp = -(3 * __ldg(u + v) - 4 * __ldg(uu + v) + __ldg(uq + v)) / (2 * dT);
    double Rf = -acc[v];
    Rk[v] = v == 0 ? Rp + Rf : Rp + Rf + vF[v];
  }
  double *rk = a.Rku1 + 5 * go;
  if (IF == kFluid && a.raw) {
#pragma unroll
    for (int r = 0; r < 5; ++r) rk[r] = Rk[r];
  } else if (IF == kFluid) {
    const double K = BCMG_K;
    const double rho = __ldg(u);
    const double Uc = c.U, Vc = c.V, Wc = c.W;
    const double VV = Uc * Uc + Vc * Vc + Wc * Wc;
    const double Pc = (__ldg(u + 4) - 0.5 * rho * VV) * (BCMG_K - 1);
    const double C = K * Pc / rho;
    const double Tt = Pc / rho;
    const double H = 0.5 * VV + C / (BCMG_K - 1);
    const double qv = VV / C;
    const double beta = qv > e ? qv : e;
    const double temp = K * Tt * (2 * dT + 3 * dTau) * (2 * dT + 3 * beta * dTau);
    const double temp2 = (BCMG_K - 1) * (beta - 1) * dT * dT;
    const double temp3 = H - H * K - VV + K * (Tt + VV);
    double d[5][5];
    d[0][0] = (2 * dT * (-2 * (-(BCMG_K - 1) * (H - VV) - temp3 * beta) * dT + 3 * K * Tt * beta * dTau)) / temp;
    d[0][1] = (-4 * Uc * temp2) / temp;
    d[0][2] = (-4 * Vc * temp2) / temp;
    d[0][3] = (-4 * Wc * temp2) / temp;
    d[0][4] = (4 * temp2) / temp;
    d[1][0] = (4 * Uc * temp3 * (beta - 1) * dT * dT) / temp;
    d[1][1] = (2 * dT * (2 * K * (Tt - Uc * Uc * (beta - 1)) * dT + 2 * Uc * Uc * (beta - 1) * dT + 3 * K * Tt * beta * dTau)) / temp;
    d[1][2] = (-4 * Uc * Vc * temp2) / temp;
    d[1][3] = (-4 * Uc * Wc * temp2) / temp;
    d[1][4] = (4 * Uc * temp2) / temp;
    d[2][0] = (4 * Vc * temp3 * (beta - 1) * dT * dT) / temp;
    d[2][1] = (-4 * Uc * Vc * temp2) / temp;
    d[2][2] = (2 * dT * (2 * K * (Tt - Vc * Vc * (beta - 1)) * dT + 2 * Vc * Vc * (beta - 1) * dT + 3 * K * Tt * beta * dTau)) / temp;
    d[2][3] = (-4 * Vc * Wc * temp2) / temp;
    d[2][4] = (4 * Vc * temp2) / temp;
    d[3][0] = (4 * Wc * temp3 * (beta - 1) * dT * dT) / temp;
    d[3][1] = (-4 * Uc * Wc * temp2) / temp;
    d[3][2] = (-4 * Vc * Wc * temp2) / temp;
    d[3][3] = (2 * dT * (2 * K * (Tt - Wc * Wc * (beta - 1)) * dT + 2 * Wc * Wc * (beta - 1) * dT + 3 * K * Tt * beta * dTau)) / temp;
    d[3][4] = (4 * Wc * temp2) / temp;
    d[4][0] = (4 * H * temp3 * (beta - 1) * dT * dT) / temp;
    d[4][1] = (-4 * H * Uc * temp2) / temp;
    d[4][2] = (-4 * H * Vc * temp2) / temp;
    d[4][3] = (-4 * H * Wc * temp2) / temp;
    d[4][4] = (2 * dT * (2 * H * (BCMG_K - 1) * (beta - 1) * dT + K * Tt * (2 * dT + 3 * beta * dTau))) / temp;
#pragma unroll
    for (int r = 0; r < 5; ++r)
      rk[r] = dTau * (d[r][0] * Rk[0] + d[r][1] * Rk[1] + d[r][2] * Rk[2] + d[r][3] * Rk[3] +
                      d[r][4] * Rk[4]);
  } else {
#pragma unroll
    for (int r = 0; r < 5; ++r) rk[r] = 0;
    // Force integrands on non-fluid cells (:2395-2398).
    const double dV = dx;  // dx = dy = dz
    a.Residual1[5 * go + 0] = -(-(dPdx) / dx + vF[1]) * dx * dV * dV;
    a.Residual1[5 * go + 1] = -(-(dPdz) / dV + vF[3]) * dx * dV * dV;
  }
}


// The cell phase with the divisions on the integer pipes and the exact
// factors 2 and 4 of the preconditioner's rows applied to whole rows.
// Returns false (and writes nothing) where an operand is out of range.
template <bool VISCOUS>
__device__ __forceinline__ bool cell_int(const FluxArgs &a, const CellIn &z) {
  IntFp o;
  const double dx = z.dx, e = z.e, dT = z.dT, dTau = z.dTau;
  const size_t go = z.go;
  const Recip kdx = o.recip(dx);
  const double inv = o.div(1.0, kdx);
  double acc[5], dPdx = 0, dPdz = 0;
#pragma unroll
  for (int ax = 0; ax < 3; ++ax) {
    const int nf = z.nf[ax], nff = z.nff[ax];
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      const double t = o.div(z.Ff[ax][v * nff] - z.Fb[ax][v * nf], kdx);
      acc[v] = ax == 0 ? t : acc[v] + t;
    }
    if (z.flag != kFluid) {
      if (ax == 0) dPdx = z.Ff[0][5 * nff] - z.Fb[0][5 * nf];
      if (ax == 2) dPdz = z.Ff[2][5 * nff] - z.Fb[2][5 * nf];
    }
  }
  const Prim &c = z.P(0, 0, 0);
  double vF[5] = {0, 0, 0, 0, 0};
  if (VISCOUS) {
    static_assert(sizeof(Prim) == 4 * sizeof(double), "u, v, w, T");
    const double T0 = o.div(o.div(z.P0, o.recip(z.rho0)), BCMG_BY(BCMG_R));
    ViscIn q;
    q.c = &c.U;
    q.mu_L = z.mu_L;
    q.T0p = T0 + 110.;
    q.inv = inv;
    q.invq = 0.25 * inv;
    q.Tc = z.Tc;
    q.by2T0 = o.recip(2 * T0);
#pragma unroll 1
    for (int ax = 0; ax < 3; ++ax) {
      const int sn = ax == 0 ? z.si : (ax == 1 ? z.sj : 4);
      const int sa = ax == 0 ? z.sj : z.si, sb = ax == 2 ? z.sj : 4;
      double Lb[4], L[4] = {0, 0, 0, 0};
#pragma unroll 1
      for (int side = 0; side < 2; ++side) {
#pragma unroll
        for (int v = 0; v < 4; ++v) Lb[v] = L[v];
        visc_int(o, q, ax, side == 1, side == 1 ? sn : -sn, sa, sb, L);
      }
#pragma unroll
      for (int v = 1; v < 5; ++v) {
        const double x = (L[v - 1] - Lb[v - 1]) * inv;
        vF[v] = ax == 0 ? x : vF[v] + x;
      }
    }
  }
  double *rk = a.Rku1 + 5 * go;
  if (z.flag != kFluid) {
    if (!o.ok) return false;
#pragma unroll
    for (int r = 0; r < 5; ++r) rk[r] = 0;
    // Force integrands on non-fluid cells (:2395-2398).
    const double dV = dx;  // dx = dy = dz
    a.Residual1[5 * go + 0] = -(-(dPdx) / dx + vF[1]) * dx * dV * dV;
    a.Residual1[5 * go + 1] = -(-(dPdz) / dV + vF[3]) * dx * dV * dV;
    return true;
  }
  const double *u = a.U1_ + 5 * go;
  const double *uu = a.U1 + 5 * go;
  const double *uq = a.U1q + 5 * go;
  const Recip k2dT = o.recip(2 * dT);
  double R[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    const double Rp = -o.div(fma64(-4.0, __ldg(uu + v), 3 * __ldg(u + v)) + __ldg(uq + v), k2dT);
    R[v] = v == 0 ? Rp - acc[v] : Rp - acc[v] + vF[v];
  }
  if (a.raw) {
    if (!o.ok) return false;
#pragma unroll
    for (int r = 0; r < 5; ++r) rk[r] = R[r];
    return true;
  }
  const double K = BCMG_K, Km1 = BCMG_K - 1;
  const double rho = __ldg(u), Uc = c.U, Vc = c.V, Wc = c.W;
  const double VV = Uc * Uc + Vc * Vc + Wc * Wc;
  const double Pc = fma64(-0.5, rho * VV, __ldg(u + 4)) * Km1;
  const Recip kr = o.recip(rho);
  const double C = o.div(K * Pc, kr), Tt = o.div(Pc, kr);
  const double H = fma64(0.5, VV, o.div(C, BCMG_BY(BCMG_K - 1)));
  const double beta = o.floor_at(o.div(VV, o.recip(C)), e);
  const double bm1 = beta - 1, b3 = 3 * beta * dTau;
  const double A2 = fma64(2.0, dT, b3);
  const Recip kt = o.recip(K * Tt * (2 * dT + 3 * dTau) * A2);
  const double t2 = Km1 * bm1 * dT * dT;
  const double t3 = H - H * K - VV + K * (Tt + VV);
  const double Z = 3 * K * Tt * beta * dTau;
  const double dTau2 = 2 * dTau;
  // Row r is 2 (sum of +-1 or +-2 times the products below).
  {
    const double eu = o.div(Uc * t2, kt), ev = o.div(Vc * t2, kt), ew = o.div(Wc * t2, kt),
                 e1 = o.div(t2, kt);
    const double Y = -Km1 * (H - VV) - t3 * beta;
    const double d00 = o.div(dT * fma64(-2.0, Y * dT, Z), kt);
    double s = fma64(-2.0, eu * R[1], d00 * R[0]);
    s = fma64(-2.0, ev * R[2], s);
    s = fma64(-2.0, ew * R[3], s);
    s = fma64(2.0, e1 * R[4], s);
    const double x0 = dTau2 * s;
    const double d10 = o.div(Uc * t3 * bm1 * dT * dT, kt);
    const double d20 = o.div(Vc * t3 * bm1 * dT * dT, kt);
    const double d30 = o.div(Wc * t3 * bm1 * dT * dT, kt);
    const double euv = o.div(Uc * Vc * t2, kt), euw = o.div(Uc * Wc * t2, kt),
                 evw = o.div(Vc * Wc * t2, kt);
    auto diag = [&](double w) {
      const double ww = w * w * bm1;
      return o.div(dT * fma64(2.0, K * (Tt - ww) * dT + ww * dT, Z), kt);
    };
    s = fma64(2.0, d10 * R[0], diag(Uc) * R[1]);
    s = fma64(-2.0, euv * R[2], s);
    s = fma64(-2.0, euw * R[3], s);
    s = fma64(2.0, eu * R[4], s);
    const double x1 = dTau2 * s;
    s = fma64(2.0, d20 * R[0] - euv * R[1], diag(Vc) * R[2]);
    s = fma64(-2.0, evw * R[3], s);
    s = fma64(2.0, ev * R[4], s);
    const double x2 = dTau2 * s;
    s = fma64(2.0, d30 * R[0] - euw * R[1] - evw * R[2], diag(Wc) * R[3]);
    s = fma64(2.0, ew * R[4], s);
    const double x3 = dTau2 * s;
    const double d40 = o.div(H * t3 * bm1 * dT * dT, kt);
    const double hu = o.div(H * Uc * t2, kt), hv = o.div(H * Vc * t2, kt),
                 hw = o.div(H * Wc * t2, kt);
    const double d44 = o.div(dT * fma64(2.0, H * Km1 * bm1 * dT, K * Tt * A2), kt);
    s = fma64(2.0, d40 * R[0] - hu * R[1] - hv * R[2] - hw * R[3], d44 * R[4]);
    const double x4 = dTau2 * s;
    if (!o.ok) return false;
    rk[0] = x0; rk[1] = x1; rk[2] = x2; rk[3] = x3; rk[4] = x4;
  }
  return true;
}

template <bool VISCOUS, typename Sh>
__global__ void __launch_bounds__(kFluxThreads, 1) k_flux_fp64(FluxArgs a, Sh sh, int nboxes) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nprim = box_prims(sh), ncell = box_cells(sh), nface = box_faces(sh);
  const int f0 = box_faces(sh, 0), f1 = box_faces(sh, 1);  // x, y faces; the rest z
  double *const F0 = reinterpret_cast<double *>(smem_raw), *const F1 = F0 + 6 * sh.groups * nface;
  Prim *const prim = reinterpret_cast<Prim *>(F1 + 6 * kSecond);
  double *const Tcs = reinterpret_cast<double *>(prim + sh.groups * nprim);
  double *const cols = Tcs + sh.groups * ncell;
  int *const nsecond = reinterpret_cast<int *>(cols + kCols * kFluxThreads);
  uint16_t *const second = reinterpret_cast<uint16_t *>(nsecond + 1);  // 0: none, else slot + 1

  const int n = a.ph.n, S = n + 4, nx = n + 1;
  const int nti = n / sh.ti, ntj = n / sh.tj, ntk = n / sh.tk, boxes = nti * ntj * ntk;
  const int tid = threadIdx.x;
  const double *__restrict__ U = a.U1_;
  const int *__restrict__ F = a.FWS;
  // Box g of this CTA: its cube (0: past the last box, or a converged case)
  // and the first cell of the box.
  struct Box { int cube, bi, bj, bk; };
  auto box = [&](int g) -> Box {
    const int b = blockIdx.x * sh.groups + g;
    if (b >= nboxes) return {0, 0, 0, 0};
    const int cube = a.cube0 + b / boxes, tl = b % boxes;
    if (!case_active(a.bt, cube)) return {0, 0, 0, 0};
    return {cube, 2 + (tl / (ntj * ntk)) * sh.ti, 2 + ((tl / ntk) % ntj) * sh.tj,
            2 + (tl % ntk) * sh.tk};
  };
  const Box only = box(0);
  if (sh.groups == 1 && only.cube == 0) return;
  if (tid == 0) *nsecond = 0;
  __syncthreads();
  // The constants of a cube's case (kernel arguments for a single case).
  const CaseConst *cases = a.bt.cube_case ? a.bt.cases : nullptr;
  auto case_at = [&](int cube) { return cases + __ldg(a.bt.cube_case + cube); };

  // Face fa (0..extent) of axis ax at in-plane position (p, q), seen from the
  // cell on its minus or plus side: where its stencil starts and the order.
  struct Stencil { const double *base; ptrdiff_t stride; int ob, of; };
  auto stencil = [&](const Box &b, int ax, int fa, int p, int q) -> Stencil {
    int li, lj, lk;  // local index of the + cell of this face
    if (ax == 0) { li = fa; lj = p; lk = q; }
    else if (ax == 1) { li = p; lj = fa; lk = q; }
    else { li = p; lj = q; lk = fa; }
    const int gx = (ax == 0 ? b.bi + li : (ax == 1 ? b.bj + lj : b.bk + lk));
    const ptrdiff_t stride = ax == 0 ? (ptrdiff_t)S * S : (ax == 1 ? (ptrdiff_t)S : 1);
    const size_t c0 = cell_index(S, b.cube, b.bi + li, b.bj + lj, b.bk + lk);
    const int fm2 = __ldg(F + c0 - 2 * stride), fm1 = __ldg(F + c0 - stride), fc = __ldg(F + c0),
              fp1 = __ldg(F + c0 + stride);
    return {U + 5 * c0, stride, order_backward(gx, fm2, fm1, fp1),
            order_forward(gx, nx, fm2, fc, fp1)};
  };

  // Phase 1: inviscid face fluxes of all three axes, one face per thread and
  // turn (no barrier between axes: the 54 warp turns of an 8^3 box spread
  // over 16 warps).
#pragma unroll 1
  for (int w = tid; w < sh.groups * nface; w += kFluxThreads) {
    const int g = sh.groups == 1 ? 0 : w / nface, fw = w - g * nface;
    const Box b = sh.groups == 1 ? only : box(g);
    if (b.cube == 0) continue;
    const int ax = fw < f0 ? 0 : (fw < f0 + f1 ? 1 : 2);
    const int f = fw - (ax == 0 ? 0 : (ax == 1 ? f0 : f0 + f1));
    const int nf = ax == 0 ? f0 : (ax == 1 ? f1 : nface - f0 - f1);
    const int dp = ax == 0 ? sh.tj : sh.ti, dq = ax == 2 ? sh.tj : sh.tk;  // in-plane extents
    const int fa = f / (dp * dq);
    const Stencil st = stencil(b, ax, fa, (f / dq) % dp, f % dq);
    const bool needB = fa < (ax == 0 ? sh.ti : (ax == 1 ? sh.tj : sh.tk)), needF = fa > 0;
    const int views = needB && needF && st.ob != st.of ? 2 : 1;
    if (views == 1) second[w] = 0;
    const double e = cases ? case_at(b.cube)->e : a.e;
    auto ld = [&](int d, int v) -> double { return __ldg(st.base + 5 * st.stride * d + v); };
#pragma unroll 1
    for (int view = 0; view < views; ++view) {
      double *dst = F0 + 6 * (w - f) + f;
      int stv = nf;  // distance between a face's values
      if (view == 1) {
        const int slot = atomicAdd(nsecond, 1);
        second[w] = slot < kSecond ? (uint16_t)(slot + 1) : (uint16_t)0xffff;
        if (slot >= kSecond) break;  // the cell forms its view itself
        dst = F1 + 6 * slot;
        stv = 1;
      }
      double Fx[5], dP;
      double *const col = cols + tid;
      IntFp o;
      const int ord = view == 0 && needB ? st.ob : st.of;
      recon_int(o, ord, ld, col);
      face_int(o, ax, col, e, Fx, dP);
      if (o.ok) {
#pragma unroll
        for (int v = 0; v < 5; ++v) dst[v * stv] = Fx[v];
        dst[5 * stv] = dP;
      } else {
        face_ref(ax, ord, st.base, st.stride, e, dst, stv);
      }
    }
  }
  // and the primitives over the boxes plus a one-cell halo (edges included),
  // by the threads that have no face left
  const int bj2 = sh.tj + 2, bk2 = sh.tk + 2;
  const int turns = (sh.groups * nface + kFluxThreads - 1) / kFluxThreads;
  const int done = sh.groups * nface - (turns - 1) * kFluxThreads;  // threads with a last face
  for (int w = tid >= done ? tid - done : tid + kFluxThreads - done; w < sh.groups * nprim;
       w += kFluxThreads) {
    const int g = sh.groups == 1 ? 0 : w / nprim, p = w - g * nprim;
    const Box b = sh.groups == 1 ? only : box(g);
    if (b.cube == 0) continue;
    const int li = p / (bj2 * bk2), lj = (p / bk2) % bj2, lk = p % bk2;
    const double *q =
        U + 5 * cell_index(S, b.cube, b.bi - 1 + li, b.bj - 1 + lj, b.bk - 1 + lk);
    double Tc;
    prim[w] = prim_int(__ldg(q), __ldg(q + 1), __ldg(q + 2), __ldg(q + 3), __ldg(q + 4), Tc);
    if (li >= 1 && li <= sh.ti && lj >= 1 && lj <= sh.tj && lk >= 1 && lk <= sh.tk)
      Tcs[g * ncell + ((li - 1) * sh.tj + (lj - 1)) * sh.tk + (lk - 1)] = Tc;
  }
  __syncthreads();

  // Phase 2: the cell's balance, viscous fluxes, source, preconditioner,
  // increment, force integrands.
  if (tid >= sh.groups * ncell) return;
  const int g = sh.groups == 1 ? 0 : tid / ncell, cell = tid - g * ncell;
  const Box b = sh.groups == 1 ? only : box(g);
  if (b.cube == 0) return;
  const int mi = cell / (sh.tj * sh.tk), mj = (cell / sh.tk) % sh.tj, mk = cell % sh.tk;
  CellIn z;
  z.si = 4 * bj2 * bk2;
  z.sj = 4 * bk2;
  z.c = &prim[g * nprim].U + (mi + 1) * z.si + (mj + 1) * z.sj + (mk + 1) * 4;
  z.e = a.e; z.dT = a.dT; z.dTau = a.dTau;
  z.mu_L = a.ph.mu_L; z.rho0 = a.ph.rho0; z.P0 = a.ph.P0;
  if (cases) {
    const CaseConst *q = case_at(b.cube);
    z.e = q->e; z.dT = q->dT; z.dTau = q->dTau;
    z.mu_L = q->mu_L; z.rho0 = q->rho0; z.P0 = q->P0;
  }
  double own[3][6];  // the cell's view of a forward face that has no slot
#pragma unroll
  for (int ax = 0; ax < 3; ++ax) {
    const int first = g * nface + (ax == 0 ? 0 : (ax == 1 ? f0 : f0 + f1));  // of the axis
    const int plane = ax == 0 ? sh.tj * sh.tk : (ax == 1 ? sh.ti * sh.tk : sh.ti * sh.tj);
    const int p = ax == 0 ? mj : mi, q = ax == 2 ? mj : mk, m = ax == 0 ? mi : (ax == 1 ? mj : mk);
    const int fb = m * plane + p * (ax == 2 ? sh.tj : sh.tk) + q, ff = fb + plane;
    z.nf[ax] = ax == 0 ? f0 : (ax == 1 ? f1 : nface - f0 - f1);
    z.Fb[ax] = F0 + 6 * first + fb;
    z.Ff[ax] = F0 + 6 * first + ff;
    z.nff[ax] = z.nf[ax];
    const int slot = second[first + ff];
    if (slot != 0) {
      z.nff[ax] = 1;
      if (slot != 0xffff) {
        z.Ff[ax] = F1 + 6 * (slot - 1);
      } else {
        const Stencil st = stencil(b, ax, m + 1, p, q);
        face_ref(ax, st.of, st.base, st.stride, z.e, own[ax], 1);
        z.Ff[ax] = own[ax];
      }
    }
  }
  z.go = cell_index(S, b.cube, b.bi + mi, b.bj + mj, b.bk + mk);
  z.flag = __ldg(F + z.go);
  z.Tc = Tcs[g * ncell + cell];
  z.dx = a.cube_size[b.cube] / n;
  if (!cell_int<VISCOUS>(a, z)) {
    const CellIn zr = z;  // (the copy lives in local memory, z in registers)
    cell_ref<VISCOUS>(a, zr);
  }
}

// The boxes of a cube edge that is not a multiple of 8: divisors of n, at most
// 512 cells in all groups together, with the least waves of CTAs (one to an SM)
// times the time of a CTA: 28 us, 11 per turn of the 512 threads over its faces,
// 0.047 per face and 0.006 per primitive (fitted to 186 launches of one wave at
// edges 4 to 36, within 13%).  Of the groups with the least waves the fewest: where
// few boxes fill one wave, large CTAs would leave SMs idle (one cube of 20^3 in 16
// CTAs of 500 cells 160 us, in 125 of 64 cells 51, with solids 318 and 66; eight
// of 4^3 in two CTAs 139, in 128 of four cells 49).  Many cubes take the largest
// boxes (512 of 12^3 1.88 ms in boxes of 432 cells).
static ShapeAny flux_shape(int n, int tile, int ncubes) {
  constexpr int kSms = 152;
  ShapeAny best{4, 4, 4, 1};
  double least = 1e300;
  auto consider = [&](int i, int j, int k) {
    ShapeAny s{i, j, k, 1};
    const int cells = box_cells(s), faces = box_faces(s);
    if (cells > kFluxThreads || flux_smem(s) > kMaxSmem) return;
    s.groups = 2;  // shared memory grows by as much with every box
    const size_t two = flux_smem(s);
    s.groups = 1;
    const size_t one = flux_smem(s);
    const int most = (int)std::min<size_t>(kFluxThreads / cells,
                                           1 + (kMaxSmem - one) / (two - one));
    const long long boxes = (long long)ncubes * (n / i) * (n / j) * (n / k);
    const long long waves = (boxes + (long long)kSms * most - 1) / ((long long)kSms * most);
    s.groups = (int)((boxes + kSms * waves - 1) / (kSms * waves));
    const int turns = (s.groups * faces + kFluxThreads - 1) / kFluxThreads;
    const double t =
        waves * (28 + 11 * turns + s.groups * (0.047 * faces + 0.006 * box_prims(s)));
    if (t < least * 0.9999) {
      least = t;
      best = s;
    }
  };
  if (tile == 4) {
    consider(4, 4, 4);
    return best;
  }
  int d[64], nd = 0;  // divisors of n (at most 256)
  for (int i = 1; i <= n; ++i)
    if (n % i == 0) d[nd++] = i;
  // (of a box's turns the one that is longest along k, whose rows are contiguous)
  for (int i = 0; i < nd; ++i)
    for (int j = 0; j < nd; ++j)
      for (int k = 0; k < nd; ++k) consider(d[i], d[j], d[k]);
  return best;
}

template <bool VISCOUS, typename Sh>
static cudaError_t launch_shape(const FluxArgs &a, const Sh &sh, int ncubes, cudaStream_t s) {
  const size_t smem = flux_smem(sh);
  const int n = a.ph.n;
  const int nboxes = ncubes * (n / sh.ti) * (n / sh.tj) * (n / sh.tk);
  if (nboxes == 0) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(
      k_flux_fp64<VISCOUS, Sh>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
  if (e != cudaSuccess) return e;
  const unsigned grid = (unsigned)((nboxes + sh.groups - 1) / sh.groups);
  k_flux_fp64<VISCOUS, Sh><<<grid, kFluxThreads, smem, s>>>(a, sh, nboxes);
  return cudaGetLastError();
}

// Cubes [a.cube0, a.cube0 + ncubes) of the flat list.
cudaError_t launch_flux_fp64(const FluxArgs &a, int ncubes, cudaStream_t s) {
  if (a.ph.n % 4 != 0) return cudaErrorInvalidValue;
  const bool visc = a.ph.mu_L != 0.0;
  if (flux_tile(a.ph.n, a.tile) == 8) {
    const Shape888 sh;
    return visc ? launch_shape<true>(a, sh, ncubes, s) : launch_shape<false>(a, sh, ncubes, s);
  }
  if (ncubes <= 0) return cudaSuccess;
  // (a search of a few us: a caller's launches in a row are of one size)
  thread_local struct { int n = 0, tile, ncubes; ShapeAny sh; } last;
  if (last.n != a.ph.n || last.tile != a.tile || last.ncubes != ncubes)
    last = {a.ph.n, a.tile, ncubes, flux_shape(a.ph.n, a.tile, ncubes)};
  const ShapeAny sh = last.sh;
  return visc ? launch_shape<true>(a, sh, ncubes, s) : launch_shape<false>(a, sh, ncubes, s);
}

}  // namespace bcmg
