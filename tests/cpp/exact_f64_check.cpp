// Checks the integer-pipe double operations of exact_f64.cuh against the
// host's IEEE operations, bit for bit, with their single-precision seeds
// disturbed by up to three units in the last place (the device's approximations
// are within one or two).  argv[1]: random cases.  Built and run by
// tests/test_exact_f64.py.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

static std::mt19937_64 rng(7);
static float disturb(float y) {
  uint32_t u;
  std::memcpy(&u, &y, 4);
  u += (int)(rng() % 7) - 3;
  std::memcpy(&y, &u, 4);
  return y;
}
#define XF_SEED(y) disturb(y)
#include "exact_f64.cuh"

using namespace om::xf;

static long bad = 0;
static void same(const char *what, double a, double b, double got, double want) {
  if (bits(got) == bits(want) || (got != got && want != want)) return;
  if (bad++ < 10) std::printf("%s(%a, %a): %a, not %a\n", what, a, b, got, want);
}

static void check(double a, double b) {
  same("div", a, b, div(a, b), a / b);
  same("sqrt", a, 0, sqrt_rn(a), std::sqrt(a));
  same("half", a, 0, half(a), a / 2.0);
  same("plus_zero", a, 0, plus_zero(a), 0.0 + a);
  same("plus_none", a, b, plus_none(a, b), a + b * 0.0);
  same("positive", a, 0, positive(a), 0.0 < a);
  same("less", a, b, less(a, b), a < b);
  same("lesseq", a, b, lesseq(a, b), a <= b);
  same("absmaller", a, b, absmaller(a, b),
       a * b <= 0.0 ? 0.0 : (std::fabs(a) < std::fabs(b) ? a : b));
}

int main(int, char **argv) {
  const double inf = HUGE_VAL;
  const double edge[] = {0.0, -0.0, inf, -inf, inf - inf, 1, -1, 2, 3, 4, 5e-324, -5e-324, 1e-2,
                         2.2250738585072014e-308, 1.7976931348623157e308, 0x1.fffffffffffffp0,
                         0x1.fffffffffffffp1, 0x1.0000000000001p0, 0x1.0000000000001p1, 0x1p-480,
                         0x1.fffffffffffffp-481, 0x1p479, 0x1p480, 1e-160, 1e160, -1e200};
  for (double a : edge)
    for (double b : edge) check(a, b);
  const uint64_t frac = 0x000fffffffffffffull;
  for (long i = 0, n = std::atol(argv[1]); i < n; ++i) {
    uint64_t u = rng(), v = rng();
    const int kind = (int)(rng() % 8);
    if (kind < 6) {  // ordinary magnitudes
      u = (u & ~(2047ull << 52)) | (uint64_t)(1003 + rng() % 40) << 52;
      v = (v & ~(2047ull << 52)) | (uint64_t)(1003 + rng() % 40) << 52;
    }
    if (kind == 1) u |= frac >> (rng() % 40), v |= frac >> (rng() % 40);
    if (kind == 2) u &= ~(frac >> (rng() % 40)), v &= ~(frac >> (rng() % 40));
    if (kind == 3) {  // quotients next to exact ones
      const double q = from_bits((rng() & frac) | 1023ull << 52);
      u = bits(q * from_bits(v)) + rng() % 3 - 1;
    }
    if (kind == 4) {  // squares and their neighbours
      const double r = from_bits(u);
      u = bits(r * r) + rng() % 3 - 1;
    }
    if (kind == 5) v = rng() & 1 ? u : u ^ 1ull << 63;
    check(from_bits(u), from_bits(v));
  }
  if (bad) std::printf("%ld differ\n", bad);
  return bad != 0;
}
