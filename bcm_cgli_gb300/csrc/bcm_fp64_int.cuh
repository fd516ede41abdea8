// Correctly rounded FP64 division, square root and multiplication on the
// integer pipes.
//
// A warp's FP64 instruction takes 73 cycles of an SM sub-partition's FP64 pipe
// (measured at 1.92 GHz; two lanes an SM and cycle would be 64), a division eight
// of them (584) and a square root as many.  The same results from 32-bit integer
// instructions cost 72 cycles per division that shares its divisor's
// reciprocal (48 more for the reciprocal) and 54 per multiplication, and run
// beside the FP64 pipe: a multiplication here and an FP64 addition side by
// side take 73 cycles together, on the FP64 pipe one after the other 144.
//
// Every result is the IEEE round-to-nearest-even one, bit for bit, for the
// operands in the stated ranges:
//  * the reciprocal of the divisor's 53-bit significand to 62 bits: a
//    hardware FP32 seed and two Newton steps in fixed point;
//  * quotient: the 54-bit truncated quotient from the reciprocal is exact or
//    one too small; the exact remainder (low 64 bits of an integer product
//    suffice, it is smaller than twice the divisor) decides; a quotient of
//    53-bit significands never lies on a rounding boundary, so the 54th bit
//    rounds;
//  * square root: an FP32 seed, two residual corrections in fixed point, the
//    54-bit truncated root fixed by its exact remainder in the same way;
//  * product: the 106-bit integer product rounded to nearest even.
// Operands out of range (subnormals, infinities, NaN, exponents that could
// leave the normal range) clear the sticky flag `ok` instead of branching,
// so independent operations interleave; the caller then discards its
// results and redoes them on the FP64 pipe.  Exact zeros are in range.
//
// The functions are also compiled for the host, where the tests compare them
// with the host's own arithmetic.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define BCMG_HD __host__ __device__ __forceinline__
#else
#define BCMG_HD inline
#endif

namespace bcmg {

#ifdef __CUDA_ARCH__
BCMG_HD uint32_t d_hi(double x) { return (uint32_t)__double2hiint(x); }
BCMG_HD uint32_t d_lo(double x) { return (uint32_t)__double2loint(x); }
BCMG_HD double d_make(uint32_t hi, uint32_t lo) { return __hiloint2double((int)hi, (int)lo); }
BCMG_HD uint32_t shl_pair(uint32_t lo, uint32_t hi, uint32_t s) { return __funnelshift_l(lo, hi, s); }
BCMG_HD uint32_t shr_pair(uint32_t lo, uint32_t hi, uint32_t s) { return __funnelshift_r(lo, hi, s); }
BCMG_HD uint32_t mul_hi(uint32_t a, uint32_t b) { return __umulhi(a, b); }
BCMG_HD float f_bits(uint32_t b) { return __uint_as_float(b); }
BCMG_HD float seed_rcp(float x) { return __fdividef(1.0f, x); }
BCMG_HD float seed_rsqrt(float x) { return rsqrtf(x); }
BCMG_HD double fma64(double a, double b, double c) { return __fma_rn(a, b, c); }
#else
BCMG_HD uint64_t d_bits(double x) { uint64_t b; std::memcpy(&b, &x, 8); return b; }
BCMG_HD uint32_t d_hi(double x) { return (uint32_t)(d_bits(x) >> 32); }
BCMG_HD uint32_t d_lo(double x) { return (uint32_t)d_bits(x); }
BCMG_HD double d_make(uint32_t hi, uint32_t lo) {
  const uint64_t b = ((uint64_t)hi << 32) | lo;
  double x;
  std::memcpy(&x, &b, 8);
  return x;
}
BCMG_HD uint32_t shl_pair(uint32_t lo, uint32_t hi, uint32_t s) {
  return (uint32_t)(((((uint64_t)hi << 32) | lo) << (s & 31)) >> 32);
}
BCMG_HD uint32_t shr_pair(uint32_t lo, uint32_t hi, uint32_t s) {
  return (uint32_t)((((uint64_t)hi << 32) | lo) >> (s & 31));
}
BCMG_HD uint32_t mul_hi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
BCMG_HD float f_bits(uint32_t b) { float x; std::memcpy(&x, &b, 4); return x; }
#ifndef BCMG_SEED_SCALE  // a test scales the seeds to model the hardware's error
#define BCMG_SEED_SCALE 1.0f
#endif
BCMG_HD float seed_rcp(float x) { return 1.0f / x * BCMG_SEED_SCALE; }
BCMG_HD float seed_rsqrt(float x) { return 1.0f / std::sqrt(x) * BCMG_SEED_SCALE; }
BCMG_HD double fma64(double a, double b, double c) { return std::fma(a, b, c); }
#endif
BCMG_HD uint64_t mul_wide(uint32_t a, uint32_t b, uint64_t c) { return (uint64_t)a * b + c; }

constexpr uint32_t kExpMask = 0x7ff00000u, kExpOne = 0x00100000u, kFracMask = 0x000fffffu;

// A divisor: the 62-bit reciprocal of its significand (at most 50 units
// below 2^114 / m, never above), the significand and the sign/exponent word.
struct Recip {
  uint64_t R;
  uint32_t mh, ml, hi;
};

// The same for a compile-time divisor, given by its bits.
template <uint64_t bits>
struct RecipConst {
  static constexpr uint64_t m = (bits & 0xfffffffffffffull) | (1ull << 52);
  static constexpr uint64_t R = (uint64_t)((((unsigned __int128)1) << 114) / m) - 4;
  BCMG_HD static Recip get() {
    return Recip{R, (uint32_t)(m >> 32), (uint32_t)m, (uint32_t)(bits >> 32) & 0xfff00000u};
  }
};

// A factor of a product: its significand (shifted left by 5 for mul), its
// exponent and sign words.
struct Factor {
  uint32_t m1, m0, e, sign;
  bool zero;
};
// A compile-time factor, given by its bits.
template <uint64_t bits>
BCMG_HD Factor const_factor() {
  constexpr uint64_t m = ((bits & 0xfffffffffffffull) | (1ull << 52)) << 5;
  return Factor{(uint32_t)(m >> 32), (uint32_t)m, (uint32_t)(bits >> 32) & kExpMask,
                (uint32_t)(bits >> 32), false};
}

// The sticky flag and the operations.
struct IntFp {
  bool ok = true;

  // exponent field in [lo, hi)
  BCMG_HD static bool within(uint32_t expw, uint32_t lo, uint32_t hi) {
    return expw - (lo << 20) < ((hi - lo) << 20);
  }

  // divisors: 2^-255 .. 2^256
  BCMG_HD Recip recip(double b) {
    const uint32_t bh = d_hi(b), bl = d_lo(b);
    ok &= within(bh & kExpMask, 768, 1280);
    Recip k;
    k.hi = bh & ~kFracMask;
    k.mh = (bh & kFracMask) | kExpOne;
    k.ml = bl;
    const uint64_t m = ((uint64_t)k.mh << 32) | k.ml;  // d = m 2^-52 in [1, 2)
    const float d = f_bits(0x3f800000u | shl_pair(bl, bh & kFracMask, 3));
    const uint32_t r0 = (uint32_t)(seed_rcp(d) * 16777216.0f);  // 2^24 / d
    const uint64_t e1 = 0ull - m * r0;  // 2^76 (1 - d r0), mod 2^64
    const uint64_t r1 =
        ((uint64_t)r0 << 24) +
        (uint64_t)(((int64_t)(int32_t)r0 * (int64_t)(int32_t)((int64_t)e1 >> 24)) >> 28);  // 2^48
    const uint64_t e2 = 0ull - m * r1;  // 2^100 (1 - d r1), mod 2^64
    k.R = (r1 << 14) +
          (uint64_t)(((int64_t)(int32_t)(r1 >> 18) * (int64_t)(int32_t)((int64_t)e2 >> 27)) >> 41) -
          4;  // 2^62
    return k;
  }

  // numerators: exact zero or 2^-511 .. 2^513
  BCMG_HD double div(double a, const Recip &k) {
    const uint32_t ah = d_hi(a), al = d_lo(a), ea = ah & kExpMask;
    const bool zero = ((ah & 0x7fffffffu) | al) == 0;
    ok &= zero | within(ea, 512, 1536);
    const uint32_t mah = (ah & kFracMask) | kExpOne;
    const uint32_t A1 = shl_pair(al, mah, 10), A0 = al << 10;
    const uint32_t R1 = (uint32_t)(k.R >> 32), R0 = (uint32_t)k.R;
    const uint64_t v = mul_wide(A1, R0, mul_wide(A0, R1, mul_hi(A0, R0)));
    const uint64_t q = mul_wide(A1, R1, v >> 32);  // 2^60 ma / mb, in (2^59, 2^61)
    const uint32_t qh = (uint32_t)(q >> 32), g = qh >> 28, s = 6u + g;
    const uint32_t th = qh >> s, tl = shr_pair((uint32_t)q, qh, s);  // 54 bits
    // remainder ma 2^(60 - s) - t mb, mod 2^64
    const uint64_t p = (uint64_t)tl * k.ml;
    const uint32_t ph = (uint32_t)(p >> 32) + tl * k.mh + th * k.ml;
    const uint64_t rho =
        ((uint64_t)(al << (22u - g)) << 32) - (((uint64_t)ph << 32) | (uint32_t)p);
    const uint64_t mb = ((uint64_t)k.mh << 32) | k.ml;
    const uint64_t t = (((uint64_t)th << 32) | tl) + (rho >= mb ? 2u : 1u);
    const uint32_t ex = ea - (k.hi & kExpMask) + (1021u << 20) + (g << 20);
    const uint32_t sign = (ah ^ k.hi) & 0x80000000u;
    return d_make((zero ? 0u : (uint32_t)(t >> 33) + ex) | sign, zero ? 0u : (uint32_t)(t >> 1));
  }

  // 2^-511 .. 2^513
  BCMG_HD double root(double x) {
    const uint32_t xh = d_hi(x), xl = d_lo(x), be = xh >> 20;
    ok &= within(xh, 512, 1536);  // a set sign bit is out of range too
    const uint32_t sh = (be & 1u) ^ 1u;  // odd exponent: significand doubled
    const uint32_t mh = shl_pair(xl, (xh & kFracMask) | kExpOne, sh), ml = xl << sh;
    const float mf = f_bits((0x3f800000u + (sh << 23)) | shl_pair(xl, xh & kFracMask, 3));
    const float rf = seed_rsqrt(mf);
    const int32_t Y = (int32_t)(rf * 16777216.0f);           // 2^24 / sqrt
    const uint32_t s0 = (uint32_t)(mf * rf * 8388608.0f);    // 2^23 sqrt
    const uint64_t m = ((uint64_t)mh << 32) | ml;
    const int32_t d0 = (int32_t)((int64_t)(m - (((uint64_t)s0 * s0) << 6)) >> 4);
    const uint64_t s1 = ((uint64_t)s0 << 25) + (uint64_t)(((int64_t)d0 * (int64_t)Y) >> 25);  // 2^48
    const int32_t d1 = (int32_t)((int64_t)((m << 44) - s1 * s1) >> 26);
    const uint64_t s2 = (s1 << 12) + (uint64_t)(((int64_t)d1 * (int64_t)Y) >> 35) - 8;  // 2^60
    uint64_t t = s2 >> 7;  // 54 bits
    const uint64_t rho = ((uint64_t)(ml << 22) << 32) - t * t;
    t += rho >= 2 * t + 1 ? 2u : 1u;
    return d_make((uint32_t)(t >> 33) + (((be + 1021u - sh) >> 1) << 20), (uint32_t)(t >> 1));
  }

  // A factor: exact zero or 2^-503 .. 2^505.
  BCMG_HD Factor factor(double a) {
    const uint32_t ah = d_hi(a), al = d_lo(a);
    Factor f;
    f.e = ah & kExpMask;
    f.zero = ((ah & 0x7fffffffu) | al) == 0;
    ok &= f.zero | within(f.e, 520, 1528);
    f.m1 = shl_pair(al, (ah & kFracMask) | kExpOne, 5);
    f.m0 = al << 5;
    f.sign = ah;
    return f;
  }
  // Product with another factor in the same range.
  BCMG_HD double mul(const Factor &a, double b) {
    const uint32_t bh = d_hi(b), bl = d_lo(b), eb = bh & kExpMask;
    const bool zb = ((bh & 0x7fffffffu) | bl) == 0, z = a.zero | zb;
    ok &= zb | within(eb, 520, 1528);
    const uint32_t B1 = shl_pair(bl, (bh & kFracMask) | kExpOne, 6), B0 = bl << 6;
    const uint64_t p0 = (uint64_t)a.m0 * B0;
    const uint64_t v = mul_wide(a.m1, B0, mul_wide(a.m0, B1, p0 >> 32));
    const uint64_t H = mul_wide(a.m1, B1, v >> 32);  // bits 64.. of the product: 52 or 53
    const uint32_t Hh = (uint32_t)(H >> 32), Hl = (uint32_t)H, vl = (uint32_t)v;
    const uint32_t s = (Hh >> 20) ^ 1u;
    const uint32_t mh = shl_pair(Hl, Hh, s), ml = shl_pair(vl, Hl, s);
    const uint32_t r = (vl << s) | ((uint32_t)p0 != 0u ? 1u : 0u);  // rounding bits, sticky
    const uint64_t m =
        (((uint64_t)mh << 32) | ml) + (r + 0x7fffffffu + (ml & 1u) < r ? 1u : 0u);
    const uint32_t ex = a.e + eb - ((1023u + s) << 20);
    return d_make((z ? 0u : (uint32_t)(m >> 32) + ex) | ((a.sign ^ bh) & 0x80000000u),
                  z ? 0u : (uint32_t)m);
  }
  BCMG_HD double mul(double a, double b) { return mul(factor(a), b); }

  // A significand for products with small integers: exact zero or
  // 2^-503 .. 2^505.
  BCMG_HD Factor plain(double a) {
    const uint32_t ah = d_hi(a), al = d_lo(a);
    Factor f;
    f.e = ah & kExpMask;
    f.zero = ((ah & 0x7fffffffu) | al) == 0;
    ok &= f.zero | within(f.e, 520, 1528);
    f.m1 = (ah & kFracMask) | kExpOne;
    f.m0 = al;
    f.sign = ah;
    return f;
  }
  // C a for a small odd integer C: the product has at most 59 bits, so two
  // 32-bit products hold it.
  template <int C>
  BCMG_HD double times(const Factor &a) {
    constexpr int k = C < 4 ? 1 : (C < 8 ? 2 : (C < 16 ? 3 : (C < 32 ? 4 : 5)));  // 2^k < C
    static_assert(C > (1 << k) && C < (2 << k), "an odd integer from 3 to 63");
    const uint64_t p0 = (uint64_t)a.m0 * C;
    const uint32_t ph = a.m1 * C + (uint32_t)(p0 >> 32), pl = (uint32_t)p0;
    const uint32_t g = ph >> (21 + k), s = k + g;  // bits beyond the 53rd
    // round to nearest even at bit s: add half a unit less one, plus the
    // last kept bit
    const uint32_t add = ((1u << (k - 1)) << g) - 1u + ((pl >> s) & 1u);
    const uint64_t t = (((uint64_t)ph << 32) | pl) + add;
    const uint32_t th = (uint32_t)(t >> 32);
    const uint32_t hi = (th >> s) + a.e + (s << 20) - kExpOne;
    return d_make((a.zero ? 0u : hi) | (a.sign & 0x80000000u),
                  a.zero ? 0u : shr_pair((uint32_t)t, th, s));
  }

  // x / 2: exact zero or any normal number from 2^-511
  BCMG_HD double half(double x) {
    const uint32_t h = d_hi(x), l = d_lo(x);
    const bool zero = ((h & 0x7fffffffu) | l) == 0;
    ok &= zero | within(h & kExpMask, 512, 2047);
    return d_make(zero ? h : h - kExpOne, l);
  }

  // max(q, e) as q > e ? q : e, for e > 0 (signed order of the bits)
  BCMG_HD double floor_at(double q, double e) {
    const int64_t qb = (int64_t)(((uint64_t)d_hi(q) << 32) | d_lo(q));
    const int64_t eb = (int64_t)(((uint64_t)d_hi(e) << 32) | d_lo(e));
    ok &= ((d_hi(q) & kExpMask) != kExpMask) & (eb >= 0) & ((d_hi(e) & kExpMask) != kExpMask);
    return qb > eb ? q : e;
  }
};

}  // namespace bcmg
