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
//    work, run on the integer pipes (bcm_fp64_int.cuh: the same correctly
//    rounded results, several quotients sharing one reciprocal);
//  * factors that are powers of two are exact, so c*x + y with such a c is
//    one fused multiply-add with the reference's bits, and common factors
//    are applied once at the end of a sum;
//  * where an operand is out of the integer routines' range the face, cell
//    or primitive is redone by the reference's own expressions;
//  * everything else keeps the reference's expression order, and this
//    translation unit is compiled with --fmad=false, so every value equals
//    the reference's (checked against the C oracle in tests/).
#include <cuda_runtime.h>

#include "bcm_common.cuh"
#include "bcm_fp64_int.cuh"
#include "bcm_kernels.h"

namespace bcmg {

struct Prim {
  double U, V, W, T;  // T = P/(rho*R): the neighbour form (:1734)
};

template <int T>
struct FluxSmem {
  static constexpr int B = T + 2;  // primitive box edge
  static constexpr int nPrim = B * B * B;
  static constexpr int nCell = T * T * T;
  static constexpr int nFace = (T + 1) * T * T;  // faces of one axis
  // Two views of a face: the plus-side cell's (the minus-side cell's for the
  // tile's last face), and the minus-side cell's where its reconstruction
  // order differs; five fluxes for each axis and the pressure of x and z
  // faces, value-major.
  static constexpr int nView = 17 * nFace;
  static constexpr size_t bytes = sizeof(Prim) * nPrim + sizeof(double) * nCell /*Tc*/ +
                                  2 * sizeof(double) * nView +
                                  ((3 * nFace + 15) / 16) * 16 /*second view present*/;
};
// Threads per CTA: 8^3 tiles one per cell.  For 4^3 tiles two warps.
template <int T>
__host__ __device__ constexpr int flux_ctas_per_sm() { return T == 8 ? 1 : 7; }

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

// The reference's face flux (face_flux), for operands out of range.
__device__ __noinline__ void face_ref(int ax, const double *ML, const double *MR, double e,
                                      double *F, double *dP) {
  if (ax == 0) face_flux<0, double>(ML, MR, e, F, *dP);
  else if (ax == 1) face_flux<1, double>(ML, MR, e, F, *dP);
  else face_flux<2, double>(ML, MR, e, F, *dP);
}

// face_flux (bcm_common.cuh) with the divisions and roots on the integer
// pipes and exact power-of-two factors folded; the axis is a run-time value
// (one copy of the code: three unrolled copies miss the instruction cache).
__device__ __forceinline__ bool face_int(int ax, const double *ML, const double *MR, double e,
                                         double *F, double &dP) {
  const double K = BCMG_K, Km1 = BCMG_K - 1;
  IntFp o;
  const Recip kL = o.recip(ML[0]), kR = o.recip(MR[0]);
  double vL[3], vR[3], v[3];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    vL[m] = o.div(ML[1 + m], kL);
    vR[m] = o.div(MR[1 + m], kR);
  }
  const double VVL = vL[0] * vL[0] + vL[1] * vL[1] + vL[2] * vL[2];
  const double VVR = vR[0] * vR[0] + vR[1] * vR[1] + vR[2] * vR[2];
  const double rVL = ML[0] * VVL, rVR = MR[0] * VVR;  // twice 0.5 rho VV
  const double PL = fma64(-0.5, rVL, ML[4]) * Km1, PR = fma64(-0.5, rVR, MR[4]) * Km1;
  const double HL = fma64(0.5, VVL, o.div(o.div(K * PL, kL), BCMG_BY(BCMG_K - 1)));
  const double HR = fma64(0.5, VVR, o.div(o.div(K * PR, kR), BCMG_BY(BCMG_K - 1)));
  const double sL = o.root(ML[0]), sR = o.root(MR[0]);
  const Recip kS = o.recip(sL + sR);
  const double rho = o.root(ML[0] * MR[0]);
#pragma unroll
  for (int m = 0; m < 3; ++m) v[m] = o.div(sL * vL[m] + sR * vR[m], kS);
  const double VV = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
  const double H = o.div(sL * HL + sR * HR, kS);
  const double C = fma64(-0.5, VV, H) * Km1;
  const Recip kC = o.recip(C);
  const double beta = o.floor_at(o.div(VV, kC), e);
  const double un = ax == 0 ? v[0] : (ax == 1 ? v[1] : v[2]);
  const double unL = ax == 0 ? vL[0] : (ax == 1 ? vL[1] : vL[2]);
  const double unR = ax == 0 ? vR[0] : (ax == 1 ? vR[1] : vR[2]);
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
  double rvL[3], rvR[3];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    rvL[m] = ML[0] * vL[m];
    rvR[m] = MR[0] * vR[m];
  }
  const double mL = ax == 0 ? rvL[0] : (ax == 1 ? rvL[1] : rvL[2]);
  const double mR = ax == 0 ? rvR[0] : (ax == 1 ? rvR[1] : rvR[2]);
  F[0] = o.half((mL + mR) - (an * (MR[0] - ML[0]) + dr));
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    double s = rvL[m] * unL, d = an * (MR[1 + m] - ML[1 + m]) + dr * v[m];
    const double r = rvR[m] * unR;
    if (ax == m) {
      s = s + PL + r + PR;
      d = d + deltaP;
    } else {
      s = s + r;
    }
    F[1 + m] = o.half(s - d);
  }
  const double F5 = an * (MR[4] - ML[4]) + dr * H + deltaP * un;
  F[4] = o.half(unL * fma64(0.5, rVL, 3.5 * PL) + unR * fma64(0.5, rVR, 3.5 * PR) - F5);
  dP = o.half(PL + PR);
  return o.ok;
}

// visc_face with the divisions and root on the integer pipes.  by2T0 divides
// by 2 T0, T0p is T0 + 110, invq inv / 4.
template <int AX, bool FWD>
__device__ __forceinline__ void visc_int(IntFp &o, double mu_L, const Recip &by2T0, double T0p,
                                         double Tc, const Prim &c, const Prim &p, double inv,
                                         double invq, const Prim &a0, const Prim &a1,
                                         const Prim &a2, const Prim &a3, const Prim &b0,
                                         const Prim &b1, const Prim &b2, const Prim &b3,
                                         double *L) {
  const double Ts = Tc + p.T;
  const double temp = o.div(Ts, by2T0);
  const double mu_E = o.div(mu_L * temp * o.root(temp) * T0p, o.recip(fma64(0.5, Ts, 110.)));
  double gn[4];
  if (FWD) {
    gn[0] = (p.U - c.U) * inv; gn[1] = (p.V - c.V) * inv;
    gn[2] = (p.W - c.W) * inv; gn[3] = (p.T - Tc) * inv;
  } else {
    gn[0] = (c.U - p.U) * inv; gn[1] = (c.V - p.V) * inv;
    gn[2] = (c.W - p.W) * inv; gn[3] = (Tc - p.T) * inv;
  }
  double d[3][3];
  constexpr int TA = AX == 0 ? 1 : 0, TB = AX == 2 ? 1 : 2;
#pragma unroll
  for (int m = 0; m < 3; ++m) d[AX][m] = gn[m];
  d[TA][0] = (a0.U + a1.U - a2.U - a3.U) * invq;
  d[TA][1] = (a0.V + a1.V - a2.V - a3.V) * invq;
  d[TA][2] = (a0.W + a1.W - a2.W - a3.W) * invq;
  d[TB][0] = (b0.U + b1.U - b2.U - b3.U) * invq;
  d[TB][1] = (b0.V + b1.V - b2.V - b3.V) * invq;
  d[TB][2] = (b0.W + b1.W - b2.W - b3.W) * invq;
  const double div = d[0][0] + d[1][1] + d[2][2];
  double s[3];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    s[m] = m == AX ? mu_E * fma64(2.0, d[AX][AX], -(2.0 / 3.0 * div))
                   : mu_E * (d[m][AX] + d[AX][m]);
    L[m] = s[m];
  }
  const double work = (c.U + p.U) * s[0] + (c.V + p.V) * s[1] + (c.W + p.W) * s[2];  // twice
  L[3] = fma64(0.5, work, o.div(mu_E * BCMG_CV * BCMG_K * gn[3], BCMG_BY(BCMG_PR)));
}

// What the cell phase reads and writes of its CTA and cell.
template <int T>
struct CellIn {
  const Prim *prim;
  const double *F0, *F1;       // face views
  const unsigned char *two;
  int mi, mj, mk;
  size_t go;                    // cell offset in the state
  int flag;
  double Tc, dx, e, dT, dTau, mu_L, rho0, P0;

  __device__ __forceinline__ const Prim &P(int di, int dj, int dk) const {
    constexpr int B = T + 2;
    return prim[((mi + 1 + di) * B + (mj + 1 + dj)) * B + (mk + 1 + dk)];
  }
  // the cell's backward and forward faces of an axis
  __device__ __forceinline__ int face(int ax, int step) const {
    const int fa = (ax == 0 ? mi : (ax == 1 ? mj : mk)) + step;
    const int p = ax == 0 ? mj : mi, q = ax == 2 ? mj : mk;
    return (fa * T + p) * T + q;
  }
  __device__ __forceinline__ const double *fwd(int ax, int ff) const {
    return two[ax * (T + 1) * T * T + ff] ? F1 : F0;
  }
};

// The cell phase by the reference's own expressions (BDF2 source, viscous
// balance, preconditioner), for operands out of the integer routines' range.
template <int T, bool VISCOUS>
__device__ __noinline__ void cell_ref(const FluxArgs &a, const CellIn<T> &z) {
  constexpr int NF = (T + 1) * T * T;
  const double dx = z.dx, inv = 1. / dx, e = z.e, dT = z.dT, dTau = z.dTau, mu_L = z.mu_L;
  const size_t go = z.go;
  double acc[5], dPdx = 0, dPdz = 0;
  for (int ax = 0; ax < 3; ++ax) {
    const int fb = z.face(ax, 0), ff = z.face(ax, 1);
    const double *Fw = z.fwd(ax, ff);
    for (int v = 0; v < 5; ++v) {
      const double t = (Fw[(5 * ax + v) * NF + ff] - z.F0[(5 * ax + v) * NF + fb]) / dx;
      acc[v] = ax == 0 ? t : acc[v] + t;
    }
    if (ax == 0) dPdx = Fw[15 * NF + ff] - z.F0[15 * NF + fb];
    if (ax == 2) dPdz = Fw[16 * NF + ff] - z.F0[16 * NF + fb];
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
template <int T, bool VISCOUS>
__device__ __forceinline__ bool cell_int(const FluxArgs &a, const CellIn<T> &z) {
  constexpr int NF = (T + 1) * T * T;
  IntFp o;
  const double dx = z.dx, e = z.e, dT = z.dT, dTau = z.dTau;
  const size_t go = z.go;
  const Recip kdx = o.recip(dx);
  const double inv = o.div(1.0, kdx);
  double acc[5], dPdx = 0, dPdz = 0;
#pragma unroll
  for (int ax = 0; ax < 3; ++ax) {
    const int fb = z.face(ax, 0), ff = z.face(ax, 1);
    const double *Fw = z.fwd(ax, ff);
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      const double t = o.div(Fw[(5 * ax + v) * NF + ff] - z.F0[(5 * ax + v) * NF + fb], kdx);
      acc[v] = ax == 0 ? t : acc[v] + t;
    }
    if (z.flag != kFluid) {
      if (ax == 0) dPdx = Fw[15 * NF + ff] - z.F0[15 * NF + fb];
      if (ax == 2) dPdz = Fw[16 * NF + ff] - z.F0[16 * NF + fb];
    }
  }
  const Prim &c = z.P(0, 0, 0);
  double vF[5] = {0, 0, 0, 0, 0};
  if (VISCOUS) {
    auto P = [&](int di, int dj, int dk) -> const Prim & { return z.P(di, dj, dk); };
    const double T0 = o.div(o.div(z.P0, o.recip(z.rho0)), BCMG_BY(BCMG_R)), T0p = T0 + 110.;
    const Recip by2T0 = o.recip(2 * T0);
    const double invq = 0.25 * inv, Tc = z.Tc, mu_L = z.mu_L;
    double Lb[4], Lf[4];
    visc_int<0, false>(o, mu_L, by2T0, T0p, Tc, c, P(-1, 0, 0), inv, invq, P(0, 1, 0),
                       P(-1, 1, 0), P(0, -1, 0), P(-1, -1, 0), P(0, 0, 1), P(-1, 0, 1),
                       P(0, 0, -1), P(-1, 0, -1), Lb);
    visc_int<0, true>(o, mu_L, by2T0, T0p, Tc, c, P(1, 0, 0), inv, invq, P(0, 1, 0), P(1, 1, 0),
                      P(0, -1, 0), P(1, -1, 0), P(0, 0, 1), P(1, 0, 1), P(0, 0, -1),
                      P(1, 0, -1), Lf);
#pragma unroll
    for (int v = 1; v < 5; ++v) vF[v] = (Lf[v - 1] - Lb[v - 1]) * inv;
    visc_int<1, false>(o, mu_L, by2T0, T0p, Tc, c, P(0, -1, 0), inv, invq, P(1, 0, 0),
                       P(1, -1, 0), P(-1, 0, 0), P(-1, -1, 0), P(0, 0, 1), P(0, -1, 1),
                       P(0, 0, -1), P(0, -1, -1), Lb);
    visc_int<1, true>(o, mu_L, by2T0, T0p, Tc, c, P(0, 1, 0), inv, invq, P(1, 0, 0), P(1, 1, 0),
                      P(-1, 0, 0), P(-1, 1, 0), P(0, 0, 1), P(0, 1, 1), P(0, 0, -1),
                      P(0, 1, -1), Lf);
#pragma unroll
    for (int v = 1; v < 5; ++v) vF[v] = vF[v] + (Lf[v - 1] - Lb[v - 1]) * inv;
    visc_int<2, false>(o, mu_L, by2T0, T0p, Tc, c, P(0, 0, -1), inv, invq, P(1, 0, 0),
                       P(1, 0, -1), P(-1, 0, 0), P(-1, 0, -1), P(0, 1, 0), P(0, 1, -1),
                       P(0, -1, 0), P(0, -1, -1), Lb);
    visc_int<2, true>(o, mu_L, by2T0, T0p, Tc, c, P(0, 0, 1), inv, invq, P(1, 0, 0), P(1, 0, 1),
                      P(-1, 0, 0), P(-1, 0, 1), P(0, 1, 0), P(0, 1, 1), P(0, -1, 0),
                      P(0, -1, 1), Lf);
#pragma unroll
    for (int v = 1; v < 5; ++v) vF[v] = vF[v] + (Lf[v - 1] - Lb[v - 1]) * inv;
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

template <int T, bool VISCOUS>
__global__ void __launch_bounds__(T *T *T, flux_ctas_per_sm<T>()) k_flux_fp64(FluxArgs a) {
  using SM = FluxSmem<T>;
  constexpr int B = SM::B, NF = SM::nFace;
  constexpr int NT = T * T * T;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Prim *prim = reinterpret_cast<Prim *>(smem_raw);
  double *Tcs = reinterpret_cast<double *>(prim + SM::nPrim);
  double *F0 = Tcs + SM::nCell, *F1 = F0 + SM::nView;
  unsigned char *two = reinterpret_cast<unsigned char *>(F1 + SM::nView);

  const int n = a.ph.n, S = n + 4, nx = n + 1;
  const int nt = n / T;
  const int tid = threadIdx.x;
  const int tiles = nt * nt * nt;
  const int cube = a.cube0 + blockIdx.x / tiles;
  if (!case_active(a.bt, cube)) return;  // converged case (uniform per CTA)
  const int tl = blockIdx.x % tiles;
  const int bi = 2 + (tl / (nt * nt)) * T, bj = 2 + ((tl / nt) % nt) * T, bk = 2 + (tl % nt) * T;
  const double *__restrict__ U = a.U1_;
  const int *__restrict__ F = a.FWS;
  const size_t cb = cell_index(S, cube, 0, 0, 0);
  // Constants of the cube's case (kernel arguments for a single case).
  double e = a.e, dT = a.dT, dTau = a.dTau, mu_L = a.ph.mu_L, rho0 = a.ph.rho0, P0 = a.ph.P0;
  if (a.bt.cube_case) {
    const CaseConst *q = a.bt.cases + __ldg(a.bt.cube_case + cube);
    e = q->e; dT = q->dT; dTau = q->dTau; mu_L = q->mu_L; rho0 = q->rho0; P0 = q->P0;
  }

  // Phase 1: primitives over the tile plus a one-cell halo (edges included).
  for (int p = tid; p < SM::nPrim; p += NT) {
    int li = p / (B * B), lj = (p / B) % B, lk = p % B;
    const double *q =
        U + 5 * (cb + ((size_t)(bi - 1 + li) * S + (bj - 1 + lj)) * S + (bk - 1 + lk));
    double Tc;
    prim[p] = prim_int(__ldg(q), __ldg(q + 1), __ldg(q + 2), __ldg(q + 3), __ldg(q + 4), Tc);
    if (li >= 1 && li <= T && lj >= 1 && lj <= T && lk >= 1 && lk <= T)
      Tcs[((li - 1) * T + (lj - 1)) * T + (lk - 1)] = Tc;
  }

  // Phase 2: inviscid face fluxes of all three axes, one face per thread and
  // turn (no barrier between axes: 54 warp turns of an 8^3 tile spread over
  // 16 warps).
#pragma unroll 1
  for (int w = tid; w < 3 * NF; w += NT) {
    const int ax = w / NF, f = w - ax * NF;
    const int fa = f / (T * T), p = (f / T) % T, q = f % T;
    int li, lj, lk;  // local index of the + cell of this face (fa may be T)
    if (ax == 0) { li = fa; lj = p; lk = q; }
    else if (ax == 1) { li = p; lj = fa; lk = q; }
    else { li = p; lj = q; lk = fa; }
    const int g = (ax == 0 ? bi + li : (ax == 1 ? bj + lj : bk + lk));
    const ptrdiff_t stride = ax == 0 ? (ptrdiff_t)S * S : (ax == 1 ? (ptrdiff_t)S : 1);
    const size_t c0 = cb + ((size_t)(bi + li) * S + (bj + lj)) * S + (bk + lk);
    const int fm2 = __ldg(F + c0 - 2 * stride), fm1 = __ldg(F + c0 - stride), f0 = __ldg(F + c0),
              fp1 = __ldg(F + c0 + stride);
    const bool needB = fa < T, needF = fa > 0;
    const int ob = order_backward(g, fm2, fm1, fp1);
    const int of = order_forward(g, nx, fm2, f0, fp1);
    const bool second = needB && needF && ob != of;
    two[w] = second ? 1 : 0;
    const double *base = U + 5 * c0;
    auto ld = [&](int d, int v) -> double { return __ldg(base + 5 * stride * d + v); };
#pragma unroll 1
    for (int view = 0; view < (second ? 2 : 1); ++view) {
      double ML[5], MR[5], Fx[5], dP;
      recon<double>(view == 0 && needB ? ob : of, ld, ML, MR);
      if (!face_int(ax, ML, MR, e, Fx, dP)) {
        double a5[5], b5[5], F5[5], d5;
        for (int v = 0; v < 5; ++v) { a5[v] = ML[v]; b5[v] = MR[v]; }
        face_ref(ax, a5, b5, e, F5, &d5);
        for (int v = 0; v < 5; ++v) Fx[v] = F5[v];
        dP = d5;
      }
      double *dst = view == 0 ? F0 : F1;
#pragma unroll
      for (int v = 0; v < 5; ++v) dst[(5 * ax + v) * NF + f] = Fx[v];
      if (ax != 1) dst[(ax == 0 ? 15 : 16) * NF + f] = dP;
    }
  }
  __syncthreads();

  // Phase 3: the cell's balance, viscous fluxes, source, preconditioner,
  // increment, force integrands.
  CellIn<T> z;
  z.prim = prim;
  z.F0 = F0;
  z.F1 = F1;
  z.two = two;
  z.mi = tid / (T * T);
  z.mj = (tid / T) % T;
  z.mk = tid % T;
  z.go = cb + ((size_t)(bi + z.mi) * S + (bj + z.mj)) * S + (bk + z.mk);
  z.flag = __ldg(F + z.go);
  z.Tc = Tcs[tid];
  z.dx = a.cube_size[cube] / n;
  z.e = e; z.dT = dT; z.dTau = dTau; z.mu_L = mu_L; z.rho0 = rho0; z.P0 = P0;
  if (!cell_int<T, VISCOUS>(a, z)) {
    const CellIn<T> zr = z;  // (the copy lives in local memory, z in registers)
    cell_ref<T, VISCOUS>(a, zr);
  }
}

template <int T>
static cudaError_t launch_t(const FluxArgs &a, int ncubes, cudaStream_t s) {
  const int nt = a.ph.n / T;
  const size_t smem = FluxSmem<T>::bytes;
  const unsigned grid = (unsigned)(ncubes * nt * nt * nt);
  if (grid == 0) return cudaSuccess;
  cudaError_t e;
  if (a.ph.mu_L != 0.0) {
    e = cudaFuncSetAttribute(k_flux_fp64<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem);
    if (e != cudaSuccess) return e;
    k_flux_fp64<T, true><<<grid, T * T * T, smem, s>>>(a);
  } else {
    e = cudaFuncSetAttribute(k_flux_fp64<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem);
    if (e != cudaSuccess) return e;
    k_flux_fp64<T, false><<<grid, T * T * T, smem, s>>>(a);
  }
  return cudaGetLastError();
}

// Cubes [a.cube0, a.cube0 + ncubes) of the flat list.
cudaError_t launch_flux_fp64(const FluxArgs &a, int ncubes, cudaStream_t s) {
  if (a.ph.n % 4 != 0) return cudaErrorInvalidValue;
  if (flux_tile(a.ph.n, a.tile) == 8) return launch_t<8>(a, ncubes, s);
  return launch_t<4>(a, ncubes, s);
}

}  // namespace bcmg
