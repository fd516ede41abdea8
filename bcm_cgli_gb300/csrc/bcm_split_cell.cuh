// Per-face and per-cell arithmetic of the split-precision stage, shared by its
// kernels (bcm_flux_split.cu, bcm_flux_march.cu): both form every value with
// the same expressions.
#pragma once

#include <cuda_runtime.h>

#include "bcm_common.cuh"
#include "bcm_kernels.h"

namespace bcmg {

struct PrimF {
  float U, V, W, Tp;  // velocity, T - T0
};

// Asynchronous 4-byte global -> shared copy (cp.async) and the wait for all
// of a thread's copies; an L2 prefetch hint.
__device__ __forceinline__ void cp_async4(void *smem_dst, const void *gmem_src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}
__device__ __forceinline__ void prefetch_l2(const void *p) {
  asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p));
}

// Delta-form preconditioned Roe flux (same formulas as face_flux in
// bcm_common.cuh, evaluated on deltas from the reference state).  Returns the
// flux with P replaced by p' in the momentum terms (P0 cancels in every face
// difference) and dPp = 0.5*(p'_L + p'_R).
template <int AX>
__device__ __forceinline__ void face_flux_delta(const float *ML, const float *MR, float e,
                                                float rho0, float P0, float *F, float &dPp) {
  const float K = 1.4f, Km1 = 0.4f;
  float dU1 = MR[0] - ML[0], dU2 = MR[1] - ML[1], dU3 = MR[2] - ML[2], dU4 = MR[3] - ML[3],
        dU5 = MR[4] - ML[4];
  float _rho = rho0 + ML[0];
  float _ir = 1.0f / _rho;
  float _U = ML[1] * _ir, _V = ML[2] * _ir, _W = ML[3] * _ir;
  float _VV = _U * _U + _V * _V + _W * _W;
  float _pp = (ML[4] - 0.5f * _rho * _VV) * Km1;  // p' = p - P0
  float _P = P0 + _pp;
  float _C = K * _P * _ir;
  float _H = 0.5f * _VV + _C * (1.0f / Km1);
  float rho_ = rho0 + MR[0];
  float ir_ = 1.0f / rho_;
  float U_ = MR[1] * ir_, V_ = MR[2] * ir_, W_ = MR[3] * ir_;
  float VV_ = U_ * U_ + V_ * V_ + W_ * W_;
  float pp_ = (MR[4] - 0.5f * rho_ * VV_) * Km1;
  float P_ = P0 + pp_;
  float C_ = K * P_ * ir_;
  float H_ = 0.5f * VV_ + C_ * (1.0f / Km1);
  float temp5 = sqrtf(_rho), temp6 = sqrtf(rho_);
  float it4 = 1.0f / (temp5 + temp6);
  float rho = temp5 * temp6;
  float U = (temp5 * _U + temp6 * U_) * it4;
  float V = (temp5 * _V + temp6 * V_) * it4;
  float W = (temp5 * _W + temp6 * W_) * it4;
  float VV = U * U + V * V + W * W;
  float H = (temp5 * _H + temp6 * H_) * it4;
  float C = (H - 0.5f * VV) * Km1;
  float q = VV / C;
  float beta = q > e ? q : e;
  const float un = AX == 0 ? U : (AX == 1 ? V : W);
  const float _un = AX == 0 ? _U : (AX == 1 ? _V : _W);
  const float un_ = AX == 0 ? U_ : (AX == 1 ? V_ : W_);
  float temp = 0.5f * (1.0f + beta) * un;
  float Sp = 0.5f * sqrtf(4.0f * beta * C + un * un * (1.0f - beta) * (1.0f - beta));
  float iS = 1.0f / Sp;
  float dp = pp_ - _pp;
  float temp1 = dp / (rho * beta * C);
  float tS = temp * iS;
  float temp2 = tS * (un_ - _un);
  float temp3 = 0.5f * (1.0f - beta) * un * temp * iS;
  float an = fabsf(un);
  float deltaU = (Sp - temp3 - beta * an) * temp1 + temp2;
  float deltaP = tS * dp + (Sp - an + temp3) * rho * (un_ - _un);
  float dr = deltaU * rho;
  float Fav1 = an * dU1 + dr;
  float Fav2 = an * dU2 + dr * U;
  float Fav3 = an * dU3 + dr * V;
  float Fav4 = an * dU4 + dr * W;
  if (AX == 0) Fav2 += deltaP;
  if (AX == 1) Fav3 += deltaP;
  if (AX == 2) Fav4 += deltaP;
  float Fav5 = an * dU5 + dr * H + deltaP * un;
  F[0] = 0.5f * ((_rho * _un + rho_ * un_) - Fav1);
  F[1] = AX == 0 ? 0.5f * ((_rho * _U * _U + _pp + rho_ * U_ * U_ + pp_) - Fav2)
                 : 0.5f * ((_rho * _U * _un + rho_ * U_ * un_) - Fav2);
  F[2] = AX == 1 ? 0.5f * ((_rho * _V * _V + _pp + rho_ * V_ * V_ + pp_) - Fav3)
                 : 0.5f * ((_rho * _V * _un + rho_ * V_ * un_) - Fav3);
  F[3] = AX == 2 ? 0.5f * ((_rho * _W * _W + _pp + rho_ * W_ * W_ + pp_) - Fav4)
                 : 0.5f * ((_rho * _W * _un + rho_ * W_ * un_) - Fav4);
  F[4] = 0.5f * ((_un * (3.5f * _P + 0.5f * _rho * _VV) + un_ * (3.5f * P_ + 0.5f * rho_ * VV_)) -
                 Fav5);
  dPp = 0.5f * (_pp + pp_);
}

// Packed FP32 pairs: Blackwell's FFMA2 / FADD2 / FMUL2 do the arithmetic of
// two independent evaluations (lane .x and lane .y) in one instruction, so
// a thread evaluating two faces at once issues about half the FP32
// instructions.  Subtraction is a - b = fma(b, -1, a) (exact: b * -1 is
// exact); reciprocals and square roots stay per lane (no packed form).
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 rcp2(float2 a) { return make_float2(1.0f / a.x, 1.0f / a.y); }
__device__ __forceinline__ float2 sqrt2(float2 a) { return make_float2(sqrtf(a.x), sqrtf(a.y)); }

// face_flux_delta for two faces of one axis at once (same formulas; lane .x
// and .y are the two faces).
template <int AX>
__device__ __forceinline__ void face_flux_delta2(const float2 *ML, const float2 *MR, float e,
                                                 float rho0, float P0, float2 *F, float2 &dPp) {
  const float2 K = f2(1.4f), Km1 = f2(0.4f), half = f2(0.5f);
  const float2 dU1 = sub2(MR[0], ML[0]), dU2 = sub2(MR[1], ML[1]), dU3 = sub2(MR[2], ML[2]),
               dU4 = sub2(MR[3], ML[3]), dU5 = sub2(MR[4], ML[4]);
  const float2 r0 = f2(rho0), p0 = f2(P0);
  const float2 _rho = add2(r0, ML[0]);
  const float2 _ir = rcp2(_rho);
  const float2 _U = mul2(ML[1], _ir), _V = mul2(ML[2], _ir), _W = mul2(ML[3], _ir);
  const float2 _VV = fma2(_W, _W, fma2(_V, _V, mul2(_U, _U)));
  const float2 _pp = mul2(fma2(mul2(f2(-0.5f), _rho), _VV, ML[4]), Km1);
  const float2 _P = add2(p0, _pp);
  const float2 _C = mul2(mul2(K, _P), _ir);
  const float2 _H = fma2(_C, f2(2.5f), mul2(half, _VV));
  const float2 rho_ = add2(r0, MR[0]);
  const float2 ir_ = rcp2(rho_);
  const float2 U_ = mul2(MR[1], ir_), V_ = mul2(MR[2], ir_), W_ = mul2(MR[3], ir_);
  const float2 VV_ = fma2(W_, W_, fma2(V_, V_, mul2(U_, U_)));
  const float2 pp_ = mul2(fma2(mul2(f2(-0.5f), rho_), VV_, MR[4]), Km1);
  const float2 P_ = add2(p0, pp_);
  const float2 C_ = mul2(mul2(K, P_), ir_);
  const float2 H_ = fma2(C_, f2(2.5f), mul2(half, VV_));
  const float2 temp5 = sqrt2(_rho), temp6 = sqrt2(rho_);
  const float2 it4 = rcp2(add2(temp5, temp6));
  const float2 rho = mul2(temp5, temp6);
  const float2 U = mul2(fma2(temp6, U_, mul2(temp5, _U)), it4);
  const float2 V = mul2(fma2(temp6, V_, mul2(temp5, _V)), it4);
  const float2 W = mul2(fma2(temp6, W_, mul2(temp5, _W)), it4);
  const float2 VV = fma2(W, W, fma2(V, V, mul2(U, U)));
  const float2 H = mul2(fma2(temp6, H_, mul2(temp5, _H)), it4);
  const float2 C = mul2(fma2(f2(-0.5f), VV, H), Km1);
  const float2 q = mul2(VV, rcp2(C));
  const float2 beta = make_float2(fmaxf(q.x, e), fmaxf(q.y, e));
  const float2 un = AX == 0 ? U : (AX == 1 ? V : W);
  const float2 _un = AX == 0 ? _U : (AX == 1 ? _V : _W);
  const float2 un_ = AX == 0 ? U_ : (AX == 1 ? V_ : W_);
  const float2 omb = sub2(f2(1.0f), beta);
  const float2 temp = mul2(mul2(half, add2(f2(1.0f), beta)), un);
  const float2 Sp = mul2(half, sqrt2(fma2(mul2(f2(4.0f), beta), C, mul2(mul2(un, un), mul2(omb, omb)))));
  const float2 iS = rcp2(Sp);
  const float2 dp = sub2(pp_, _pp);
  const float2 temp1 = mul2(dp, rcp2(mul2(mul2(rho, beta), C)));
  const float2 tS = mul2(temp, iS);
  const float2 dun = sub2(un_, _un);
  const float2 temp2 = mul2(tS, dun);
  const float2 temp3 = mul2(mul2(mul2(mul2(half, omb), un), temp), iS);
  const float2 an = make_float2(fabsf(un.x), fabsf(un.y));
  const float2 deltaU = fma2(sub2(sub2(Sp, temp3), mul2(beta, an)), temp1, temp2);
  const float2 deltaP = fma2(mul2(add2(sub2(Sp, an), temp3), rho), dun, mul2(tS, dp));
  const float2 dr = mul2(deltaU, rho);
  float2 Fav1 = fma2(an, dU1, dr);
  float2 Fav2 = fma2(an, dU2, mul2(dr, U));
  float2 Fav3 = fma2(an, dU3, mul2(dr, V));
  float2 Fav4 = fma2(an, dU4, mul2(dr, W));
  if (AX == 0) Fav2 = add2(Fav2, deltaP);
  if (AX == 1) Fav3 = add2(Fav3, deltaP);
  if (AX == 2) Fav4 = add2(Fav4, deltaP);
  const float2 Fav5 = fma2(deltaP, un, fma2(an, dU5, mul2(dr, H)));
  const float2 _rhoun = mul2(_rho, _un), rhoun_ = mul2(rho_, un_);
  F[0] = mul2(half, sub2(add2(_rhoun, rhoun_), Fav1));
  F[1] = AX == 0 ? mul2(half, sub2(add2(fma2(_rhoun, _U, _pp), fma2(rhoun_, U_, pp_)), Fav2))
                 : mul2(half, sub2(fma2(rhoun_, U_, mul2(_rhoun, _U)), Fav2));
  F[2] = AX == 1 ? mul2(half, sub2(add2(fma2(_rhoun, _V, _pp), fma2(rhoun_, V_, pp_)), Fav3))
                 : mul2(half, sub2(fma2(rhoun_, V_, mul2(_rhoun, _V)), Fav3));
  F[3] = AX == 2 ? mul2(half, sub2(add2(fma2(_rhoun, _W, _pp), fma2(rhoun_, W_, pp_)), Fav4))
                 : mul2(half, sub2(fma2(rhoun_, W_, mul2(_rhoun, _W)), Fav4));
  const float2 EL = fma2(mul2(half, _rho), _VV, mul2(f2(3.5f), _P));
  const float2 ER = fma2(mul2(half, rho_), VV_, mul2(f2(3.5f), P_));
  F[4] = mul2(half, sub2(fma2(un_, ER, mul2(_un, EL)), Fav5));
  dPp = mul2(half, add2(_pp, pp_));
}

template <int AX, bool FWD>
__device__ __forceinline__ void visc_face_f(float mu_L, float T0, const PrimF &c, const PrimF &o,
                                            float inv, const PrimF &a0, const PrimF &a1,
                                            const PrimF &a2, const PrimF &a3, const PrimF &b0,
                                            const PrimF &b1, const PrimF &b2, const PrimF &b3,
                                            float *L) {
  float Tm = T0 + 0.5f * (c.Tp + o.Tp);
  float temp = Tm / T0;
  float mu_E = mu_L * temp * sqrtf(temp) * (T0 + 110.f) / (Tm + 110.f);
  float gn[4];
  if (FWD) {
    gn[0] = (o.U - c.U) * inv; gn[1] = (o.V - c.V) * inv;
    gn[2] = (o.W - c.W) * inv; gn[3] = (o.Tp - c.Tp) * inv;
  } else {
    gn[0] = (c.U - o.U) * inv; gn[1] = (c.V - o.V) * inv;
    gn[2] = (c.W - o.W) * inv; gn[3] = (c.Tp - o.Tp) * inv;
  }
  const float q = 0.25f * inv;
  float ga[3], gb[3];
  ga[0] = (a0.U + a1.U - a2.U - a3.U) * q;
  ga[1] = (a0.V + a1.V - a2.V - a3.V) * q;
  ga[2] = (a0.W + a1.W - a2.W - a3.W) * q;
  gb[0] = (b0.U + b1.U - b2.U - b3.U) * q;
  gb[1] = (b0.V + b1.V - b2.V - b3.V) * q;
  gb[2] = (b0.W + b1.W - b2.W - b3.W) * q;
  float d[3][3];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    d[AX][m] = gn[m];
    d[AX == 0 ? 1 : 0][m] = ga[m];
    d[AX == 2 ? 1 : 2][m] = gb[m];
  }
  float div = d[0][0] + d[1][1] + d[2][2];
  float Um = 0.5f * (c.U + o.U), Vm = 0.5f * (c.V + o.V), Wm = 0.5f * (c.W + o.W);
  float s1, s2, s3;
  if (AX == 0) {
    s1 = mu_E * (2.f * d[0][0] - (2.f / 3.f) * div);
    s2 = mu_E * (d[1][0] + d[0][1]);
    s3 = mu_E * (d[2][0] + d[0][2]);
  } else if (AX == 1) {
    s1 = mu_E * (d[1][0] + d[0][1]);
    s2 = mu_E * (2.f * d[1][1] - (2.f / 3.f) * div);
    s3 = mu_E * (d[2][1] + d[1][2]);
  } else {
    s1 = mu_E * (d[2][0] + d[0][2]);
    s2 = mu_E * (d[2][1] + d[1][2]);
    s3 = mu_E * (2.f * d[2][2] - (2.f / 3.f) * div);
  }
  L[0] = s1;
  L[1] = s2;
  L[2] = s3;
  L[3] = Um * s1 + Vm * s2 + Wm * s3 + mu_E * (float)(BCMG_CV * BCMG_K / BCMG_PR) * gn[3];
}

// Reconstruction of the split path: the stencils of recon() (bcm_common.cuh)
// with the 1/60 and 1/6 factors folded into the coefficients (one multiply
// fewer per value; the FP64 path keeps the reference's form).
template <typename Ld>
__device__ __forceinline__ void recon_split(int ord, Ld ld, float *ML, float *MR) {
  if (ord == 5) {
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      const float a = ld(-3, v), b = ld(-2, v), c = ld(-1, v), d = ld(0, v), f = ld(1, v),
                  g = ld(2, v);
      ML[v] = (2.f / 60) * a - (13.f / 60) * b + (47.f / 60) * c + (27.f / 60) * d -
              (3.f / 60) * f;
      MR[v] = (-3.f / 60) * b + (27.f / 60) * c + (47.f / 60) * d - (13.f / 60) * f +
              (2.f / 60) * g;
    }
  } else if (ord == 3) {
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      const float b = ld(-2, v), c = ld(-1, v), d = ld(0, v), f = ld(1, v);
      ML[v] = (-1.f / 6) * b + (5.f / 6) * c + (2.f / 6) * d;
      MR[v] = (2.f / 6) * c + (5.f / 6) * d - (1.f / 6) * f;
    }
  } else {
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      ML[v] = ld(-1, v);
      MR[v] = ld(0, v);
    }
  }
}

// Constants of a cube's case (kernel arguments for a single case).
struct SplitConst {
  float rho0, P0, RT0 /* R * T0 */, ef, T0, mu_L, i2dt, dT, dTau;
  double rho0d, E0d;  // mirror reference state (FP64)
};
__device__ __forceinline__ SplitConst split_const(const FluxSplitArgs &a, int cube) {
  SplitConst z = {a.rho0f, a.P0f,   a.RT0f, a.ef,       a.T0f,  a.mu_Lf,
                  a.i2dtf, a.dTf,   a.dTauf, a.mir.rho0, a.mir.E0};
  if (a.bt.cube_case) {
    const CaseConst *cq = a.bt.cases + __ldg(a.bt.cube_case + cube);
    z = {cq->rho0f, cq->P0f,  cq->RT0f,  cq->ef,   cq->T0f, cq->mu_Lf,
         cq->i2dtf, cq->dTf,  cq->dTauf, cq->rho0, cq->E0};
  }
  return z;
}

// Primitives (u, v, w, T - T0) of a cell's deltas.
__device__ __forceinline__ PrimF prim_split(const SplitConst &z, const float *q) {
  const float iR = 1.0f / 287.0f;
  float r = q[0], m1 = q[1], m2 = q[2], m3 = q[3], e = q[4];
  float rho = z.rho0 + r;
  float ir = 1.0f / rho;
  PrimF pr;
  pr.U = m1 * ir;
  pr.V = m2 * ir;
  pr.W = m3 * ir;
  float pp = (e - 0.5f * rho * (pr.U * pr.U + pr.V * pr.V + pr.W * pr.W)) * 0.4f;
  pr.Tp = (pp - r * z.RT0) * ir * iR;  // T - T0 = (p' - rho' R T0) / (rho R)
  return pr;
}

// A cell's FP64 state, the previous level and the level difference, as
// loaded; split_source forms the BDF2 source (times -2 dT) from the FP64
// time-level differences, then FP32.
//
// CVT: which conversions of a cell's stage go to the integer pipes (bit 0: FP64
// to FP32, bit 1: FP32 to FP64; the same bits as the hardware's, which take a
// slot of the FP64 pipe each).  Per stage of a 30-stage step, ns a cell, CVT 0,
// 1, 2, 3: march n = 8 0.314 0.320 0.314 0.323, n = 12 (1,728 cubes) 0.193 0.204
// 0.193 0.213, n = 16 (2,744) 0.142 0.132 0.136 0.133, n = 20 0.187 0.177 0.180
// 0.181, n = 24 0.149 0.142 0.145 0.147, n = 28 0.180 0.169 0.173 0.175, n = 32
// 0.140 0.124 0.130 0.121, edges without a kernel of their own (36) 0.175
// 0.174 0.171 0.179; tiles of 4^3 (4,096) 0.745 0.671 0.667 0.673, of 8^3 (4,096)
// 0.215 0.219 0.211 0.220.
template <int CVT>
__device__ __forceinline__ float split_f(double x) {
  return (CVT & 1) ? to_float_int(x) : __double2float_rn(x);
}
template <int CVT>
__device__ __forceinline__ double split_d(float x) {
  return (CVT & 2) ? to_double_int(x) : (double)x;
}
struct SplitLevels {
  double x[5], y[5];
  float d2[5];
};
__device__ __forceinline__ void split_load(const FluxSplitArgs &a, size_t go, SplitLevels &l) {
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    l.x[v] = a.U1_[5 * go + v];  // only this thread reads or writes these cells
    l.y[v] = __ldg(a.U1 + 5 * go + v);
    l.d2[v] = __ldg(a.D2 + 5 * go + v);
  }
}
// (fused operations written out where the operands come from different
// places in the kernels, so that both round alike)
template <int CVT>
__device__ __forceinline__ void split_source(const SplitLevels &l, float *src) {
#pragma unroll
  for (int v = 0; v < 5; ++v)
    src[v] = __fmaf_rn(3.0f, split_f<CVT>(l.x[v] - l.y[v]), -l.d2[v]);
}

// The rest of a cell's stage, given its inviscid balance acc, state xq and
// source src: viscous balance (P(di, dj, dk) are the primitives around it),
// preconditioner, state update, norm terms, next mirror value.  qm are the
// cell's deltas, go its offset; push(array, values) copies a new value into
// the same-level neighbours' ghost layers.  NORMS: stage 3 (the sums take 14
// registers).
template <bool VISCOUS, bool NORMS, int CVT, typename Prims, typename Push>
__device__ __forceinline__ void split_cell(const FluxSplitArgs &a, const SplitConst &z, int cube,
                                           float inv, Prims P, const float *qm, const float *acc,
                                           const double *xq, const float *src,
                                           float dPdx, float dPdz, size_t go, bool fluid,
                                           float *Mw, double *s5, Push push) {
  const PrimF &c = P(0, 0, 0);
  float vF[5] = {0, 0, 0, 0, 0};
  if (VISCOUS) {
    const float T0 = z.T0;
    const float mu_L = z.mu_L;
    float Lb[4], Lf[4], Mb[4], Mf[4], Nb[4], Nf[4];
    visc_face_f<0, false>(mu_L, T0, c, P(-1, 0, 0), inv, P(0, 1, 0), P(-1, 1, 0), P(0, -1, 0),
                          P(-1, -1, 0), P(0, 0, 1), P(-1, 0, 1), P(0, 0, -1), P(-1, 0, -1), Lb);
    visc_face_f<0, true>(mu_L, T0, c, P(1, 0, 0), inv, P(0, 1, 0), P(1, 1, 0), P(0, -1, 0),
                         P(1, -1, 0), P(0, 0, 1), P(1, 0, 1), P(0, 0, -1), P(1, 0, -1), Lf);
    visc_face_f<1, false>(mu_L, T0, c, P(0, -1, 0), inv, P(1, 0, 0), P(1, -1, 0), P(-1, 0, 0),
                          P(-1, -1, 0), P(0, 0, 1), P(0, -1, 1), P(0, 0, -1), P(0, -1, -1), Mb);
    visc_face_f<1, true>(mu_L, T0, c, P(0, 1, 0), inv, P(1, 0, 0), P(1, 1, 0), P(-1, 0, 0),
                         P(-1, 1, 0), P(0, 0, 1), P(0, 1, 1), P(0, 0, -1), P(0, 1, -1), Mf);
    visc_face_f<2, false>(mu_L, T0, c, P(0, 0, -1), inv, P(1, 0, 0), P(1, 0, -1), P(-1, 0, 0),
                          P(-1, 0, -1), P(0, 1, 0), P(0, 1, -1), P(0, -1, 0), P(0, -1, -1), Nb);
    visc_face_f<2, true>(mu_L, T0, c, P(0, 0, 1), inv, P(1, 0, 0), P(1, 0, 1), P(-1, 0, 0),
                         P(-1, 0, 1), P(0, 1, 0), P(0, 1, 1), P(0, -1, 0), P(0, -1, 1), Nf);
#pragma unroll
    for (int v = 1; v < 5; ++v)
      vF[v] = ((Lf[v - 1] - Lb[v - 1]) + (Mf[v - 1] - Mb[v - 1]) + (Nf[v - 1] - Nb[v - 1])) * inv;
  }

  double *u = a.U1_ + 5 * go;
  float Rk[5];
  double un[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) Rk[v] = __fmaf_rn(-src[v], z.i2dt, -acc[v]) + vF[v];
  if (fluid && a.RK == 0) {
    // residual only: the LU-SGS right-hand side
#pragma unroll
    for (int v = 0; v < 5; ++v) a.R32[5 * go + v] = Rk[v];
  } else if (fluid) {
    const float K = 1.4f, Km1 = 0.4f;
    const float dT = z.dT, dTau = z.dTau;
    const float rho = z.rho0 + qm[0];
    const float Uc = c.U, Vc = c.V, Wc = c.W;
    const float VV = Uc * Uc + Vc * Vc + Wc * Wc;
    const float Pc = z.P0 + (qm[4] - 0.5f * rho * VV) * Km1;
    const float Tt = Pc / rho;  // P/rho (:2302)
    const float C = K * Tt;
    const float qv = VV / C;
    const float beta = qv > z.ef ? qv : z.ef;
    // The inverse preconditioner (:2315-2390) is diagonal plus rank one: with X =
    // (1, u, v, w, H), Y = (V^2/2, -u, -v, -w, 1) and C = K T it is alpha (I +
    // g (K-1)/C X Y^T), alpha = 2 dT / (2 dT + 3 dTau), g = 2 dT (beta-1) / (2 dT +
    // 3 beta dTau).  In the energy, whose terms cancel to a part beta, h = 1 + g
    // is formed as the product it is.  Its 25 entries written out take some 130
    // operations more a cell (1 to 4% of the stage) and cancel in FP32.
    const float iden = 1.0f / (2 * dT + 3 * beta * dTau);
    const float g = 2 * dT * (beta - 1) * iden, h = beta * (2 * dT + 3 * dTau) * iden;
    const float alpha = 2 * dT / (2 * dT + 3 * dTau);
    // Stage update Q += w dQ (w = 1, 1/4, 2/3): the reference's RK
    // combinations with Q1 = Q2 = Q on fluid cells at stage entry.
    const float w = a.RK == 1 ? 1.0f : (a.RK == 2 ? 0.25f : 2.0f / 3.0f);
    const float wa = w * dTau * alpha, VV2 = 0.5f * VV;
    const float kin =
        __fmaf_rn(-Uc, Rk[1], __fmaf_rn(-Vc, Rk[2], __fmaf_rn(-Wc, Rk[3], VV2 * Rk[0])));
    const float gp = g * Km1 * (Rk[4] + kin) / C;
    const float dq[5] = {wa * (Rk[0] + gp), wa * __fmaf_rn(Uc, gp, Rk[1]),
                         wa * __fmaf_rn(Vc, gp, Rk[2]), wa * __fmaf_rn(Wc, gp, Rk[3]),
                         wa * __fmaf_rn(h, Rk[4], __fmaf_rn(g, kin, VV2 * gp))};
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      un[r] = xq[r] + split_d<CVT>(dq[r]);
      u[r] = un[r];
    }
    // Same-level interface copy of this cell, done here.  No CTA reads the
    // FP64 state of another cell during the stage, so the write races with
    // nothing.
    push(a.U1_, un);
    if (NORMS && a.RK == 3) {
      // Change norms of p, u, v, w, T from the increment, in FP32; summed
      // in FP64 (BCM_Flux...cpp:2530-2566).
      // (the momentum's deltas are the rounded values of xq)
      const float rf = rho, m1 = qm[1], m2 = qm[2], m3 = qm[3];
      const float dr = dq[0], e1 = dq[1], e2 = dq[2], e3 = dq[3], dE = dq[4];
      const float den = 1.0f / (rf * (rf + dr));
      const float dU = (e1 * rf - m1 * dr) * den;
      const float dVv = (e2 * rf - m2 * dr) * den;
      const float dW = (e3 * rf - m3 * dr) * den;
      const float mm = m1 * m1 + m2 * m2 + m3 * m3;
      const float dKE =
          0.5f * ((2.f * (m1 * e1 + m2 * e2 + m3 * e3) + e1 * e1 + e2 * e2 + e3 * e3) * rf - mm * dr) * den;
      const float dP = Km1 * (dE - dKE);
      const float dTt = (dP * rf - Pc * dr) * den;
      s5[0] += split_d<CVT>(dP * dP);
      s5[1] += split_d<CVT>(dU * dU);
      s5[2] += split_d<CVT>(dVv * dVv);
      s5[3] += split_d<CVT>(dW * dW);
      s5[4] += split_d<CVT>(dTt * dTt);
    }
  } else {
    // Force integrands on non-fluid cells (:2395-2398); their sum over the
    // case is er[6], er[7].
    const double dx = a.cube_size[cube] / a.ph.n;
    const double dV = dx * dx * dx;
    const double r0 = -((double)(-dPdx * inv) + (double)vF[1]) * dV;
    const double r1 = -((double)(-dPdz * inv) + (double)vF[3]) * dV;
    a.Residual1[5 * go + 0] = r0;
    a.Residual1[5 * go + 1] = r1;
    if (NORMS) {
      s5[5] += r0;
      s5[6] += r1;
    }
  }
  if (Mw) {
    // The cell's mirror value after the stage into the next buffer (the
    // staged value where the cell did not change), and into the same-level
    // neighbour's ghost layers: every cell of those layers pushes, since the
    // next buffer's ghost layers hold values two stages old.
    float m5[5];
    if (fluid) {
#pragma unroll
      for (int v = 0; v < 5; ++v)
        m5[v] = split_f<CVT>(v == 0 ? un[v] - z.rho0d : (v == 4 ? un[v] - z.E0d : un[v]));
    } else {
  #pragma unroll
      for (int v = 0; v < 5; ++v) m5[v] = qm[v];
    }
    float *mw = Mw + 5 * go;
#pragma unroll
    for (int v = 0; v < 5; ++v) mw[v] = m5[v];
    push(Mw, m5);
  }
}

}  // namespace bcmg
