// tri_test_host.cpp -- the quotients and sign tests of csrc/tri_test.cuh on the CPU, for
// tests/test_tri_test.py: its double-precision intrinsics are correctly rounded
// operations, so the host's own are the same.
//
// argv: seed count.  stdout: "ok NEAR" (NEAR: quotients next to halfway between two
// doubles) or "error ...".
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>

static inline double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
static inline double __dmul_rn(double a, double b) { return a * b; }
static inline double __ddiv_rn(double a, double b) { return a / b; }
static inline int64_t __double_as_longlong(double x) {
  int64_t v;
  memcpy(&v, &x, 8);
  return v;
}
static inline int __double2hiint(double x) { return (int)(__double_as_longlong(x) >> 32); }
using std::fabs;
using std::isfinite;

#include "tri_test.cuh"

using namespace cvtgb;

static uint64_t state;
static uint64_t rnd() {  // splitmix64 (S. Vigna)
  uint64_t z = (state += 0x9e3779b97f4a7c15ull);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
static double bits(uint64_t v) {
  double x;
  memcpy(&x, &v, 8);
  return x;
}
// a double of any exponent (exp < 0) or one in [2^(exp), 2^(exp + 1))
static double some(int exp) {
  const uint64_t e = exp < 0 ? rnd() % 2047 : (uint64_t)exp;
  uint64_t m = rnd() & 0xfffffffffffffull;
  if (rnd() % 4 == 0) m &= ~0ull << (rnd() % 52);           // few bits
  if (rnd() % 4 == 0) m |= 0xfffffffffffffull >> (rnd() % 52);  // many ones
  return bits((rnd() & (1ull << 63)) | (e << 52) | m);
}

int main(int argc, char **argv) {
  state = argc > 1 ? strtoull(argv[1], nullptr, 10) : 1;
  const long count = argc > 2 ? atol(argv[2]) : 100000;
  long near = 0;
  for (long k = 0; k < count; ++k) {
    const int kind = (int)(k % 4);
    double num, den = fabs(some(kind == 3 ? -1 : 623 + (int)(rnd() % 801)));
    if (kind == 0) {
      num = some(623 + (int)(rnd() % 801));
    } else if (kind < 3) {
      // D Q = N 2^54 + s, D and Q odd, Q of 54 bits: N / D is Q less s / D units in the
      // 54th place, next to halfway between two doubles
      const uint64_t D = (1ull << 52) | (rnd() >> 12) | 1ull, mask = (1ull << 54) - 1;
      const int64_t small = (int64_t)(2 * (rnd() % 32) + 1) * (rnd() & 1 ? 1 : -1);
      uint64_t inv = D;  // D^-1 mod 2^64 (Newton)
      for (int it = 0; it < 6; ++it) inv *= 2 - D * inv;
      const uint64_t Q = ((uint64_t)small * inv) & mask;
      if (Q < (1ull << 53)) continue;
      const uint64_t N = (uint64_t)(((__int128)D * Q - small) >> 54);
      num = ldexp((double)N, (int)(rnd() % 700) - 400);
      den = ldexp((double)D, (int)(rnd() % 700) - 400);
      if (rnd() & 1) num = -num;
      ++near;
    } else {
      num = rnd() % 16 ? some(-1) : 0.0 * some(1023);
    }
    if (den == 0) continue;
    const double y = 1.0 / den, want = num / den, got = div_by(num, den, y);
    if (__double_as_longlong(got) != __double_as_longlong(want) && !(got != got && want != want))
      return printf("error div %a / %a = %a, not %a\n", num, den, got, want), 0;
    if (!std::isnan(num)) {
      if (below_zero(num) != (num < 0)) return printf("error below %a\n", num), 0;
      if (quot_negative(num, den) && !(want < 0)) return printf("error sign %a / %a\n", num, den), 0;
    }
  }
  printf("ok %ld\n", near);
}
