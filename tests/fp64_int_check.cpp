// Host check of bcm_fp64_int.cuh: counts results that differ from the host's
// own IEEE arithmetic, and operands out of range that keep the flag set.
static float g_seed_scale = 1.0f;
#define BCMG_SEED_SCALE g_seed_scale
#include "../bcm_cgli_gb300/csrc/bcm_fp64_int.cuh"

#include <limits>

using namespace bcmg;

namespace {
uint64_t mix(uint64_t &s) {
  s += 0x9E3779B97F4A7C15ull;
  uint64_t z = s;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
double from_bits(uint64_t b) { double x; std::memcpy(&x, &b, 8); return x; }
bool same(double x, double y) {
  uint64_t a, b;
  std::memcpy(&a, &x, 8);
  std::memcpy(&b, &y, 8);
  return a == b;
}
// operands of one kind: 0 random significands, 1 few leading bits, 2 equal or
// one or two units apart, 3 all ones less a little, 4 few trailing bits,
// 5 zeros and powers of two
void operands(int kind, uint64_t &s, int elo, int ehi, double &a, double &b) {
  uint64_t ma = mix(s) >> 12, mb = mix(s) >> 12;
  const uint64_t r = mix(s), top = 0xfffffffffffffull;
  if (kind == 1) { ma &= 0xfffull << 40; mb &= 0xfffull << 40; }
  if (kind == 2) ma = (mb + (r >> 62)) & top;
  if (kind == 3) { mb = top - (r >> 60); if (r & 1) ma = top - (r >> 58 & 15); }
  if (kind == 4) { ma &= 0x3ffffff; mb &= 0x3ffffff; }
  if (kind == 5) { ma = mb = 0; }
  const uint64_t ea = elo + (mix(s) >> 16) % (ehi - elo), eb = elo + (mix(s) >> 16) % (ehi - elo);
  a = from_bits(((r >> 8 & 1) << 63) | ea << 52 | ma);
  b = from_bits(((r >> 9 & 1) << 63) | eb << 52 | mb);
  if (kind == 5 && (r >> 10 & 3) == 0) a = (r >> 12 & 1) ? -0.0 : 0.0;
}
}  // namespace

// op 0 div, 1 root, 2 mul, 3 half, 4 floor_at, 5 division by constants,
// 6 products with constants
extern "C" long fp64_int_bad(int op, int kind, long count, double seed_err) {
  uint64_t s = 977 * (uint64_t)op + 31 * (uint64_t)kind + 1;
  long bad = 0;
  for (long i = 0; i < count; ++i) {
    double a, b, x = 0, y = 0;
    g_seed_scale = (float)(1.0 + seed_err * (double)((int)(i % 5) - 2) / 2.0);
    IntFp o;
    if (op == 0) {
      operands(kind, s, 768, 1280, a, b);
      x = o.div(a, o.recip(b));
      y = a / b;
    } else if (op == 1) {
      operands(kind, s, 512, 1536, a, b);
      a = std::fabs(a);
      if (kind == 2) {  // squares and their neighbours
        const double c = from_bits((d_bits(a) & ~0x3ffffffull & ~(0x7ffull << 52)) | (1023ull + i % 2) << 52);
        a = from_bits(d_bits(c * c) + (uint64_t)(i / 2 % 3) - 1);
      }
      if (a == 0) continue;
      x = o.root(a);
      y = std::sqrt(a);
    } else if (op == 2) {
      operands(kind, s, 520, 1528, a, b);
      x = o.mul(a, b);
      y = a * b;
    } else if (op == 3) {
      operands(kind, s, 512, 2047, a, b);
      x = o.half(a);
      y = 0.5 * a;
    } else if (op == 4) {
      operands(kind, s, 900, 1100, a, b);
      b = std::fabs(b);
      x = o.floor_at(a, b);
      y = a > b ? a : b;
    } else if (op == 6) {
      operands(kind, s, 520, 1528, a, b);
      const Factor f = o.plain(a);
      bad += !same(o.times<3>(f), 3 * a) + !same(o.times<13>(f), 13 * a);
      bad += !same(o.times<27>(f), 27 * a) + !same(o.times<47>(f), 47 * a);
      bad += !same(o.times<5>(f), 5 * a) + !same(o.times<63>(f), 63 * a);
      x = o.mul(const_factor<__builtin_bit_cast(uint64_t, 1. / 60)>(), a);
      y = 1. / 60 * a;
    } else {
      operands(kind, s, 768, 1280, a, b);
      x = o.div(a, RecipConst<__builtin_bit_cast(uint64_t, 1.4 - 1)>::get());
      y = a / (1.4 - 1);
      bad += !same(o.div(a, RecipConst<__builtin_bit_cast(uint64_t, 287.0)>::get()), a / 287.0);
      bad += !same(o.div(a, RecipConst<__builtin_bit_cast(uint64_t, 0.72)>::get()), a / 0.72);
    }
    bad += !o.ok || !same(x, y);
  }
  return bad;
}

// out-of-range operands that are not flagged
extern "C" long fp64_int_unflagged(void) {
  typedef std::numeric_limits<double> L;
  const double big[] = {L::infinity(), -L::infinity(), L::quiet_NaN(), L::denorm_min(), 1e-310,
                        L::max(), L::min()};
  long n = 0;
  for (double v : big) {
    { IntFp o; o.recip(v); n += o.ok; }
    { IntFp o; o.div(v, o.recip(1.5)); n += o.ok; }
    { IntFp o; o.root(v); n += o.ok; }
    { IntFp o; o.mul(v, 1.5); n += o.ok; }
    { IntFp o; o.mul(1.5, v); n += o.ok; }
    { IntFp o; o.plain(v); n += o.ok; }
    { IntFp o; if (v != L::max()) { o.half(v); n += o.ok; } }
  }
  { IntFp o; o.recip(0.0); n += o.ok; }
  { IntFp o; o.root(0.0); n += o.ok; }
  { IntFp o; o.root(-1.0); n += o.ok; }
  { IntFp o; o.floor_at(L::quiet_NaN(), 0.1); n += o.ok; }
  { IntFp o; o.floor_at(1.0, -0.1); n += o.ok; }
  return n;
}
