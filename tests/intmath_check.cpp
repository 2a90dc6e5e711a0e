// intmath.h against the C library on the host: every pair of a list of special
// values, then n generated pairs (any exponents, near ones, short and nearly
// full significands).  Prints the number of differences.
#include <cinttypes>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../rocflu_gb300/csrc/intmath.h"

using namespace rflu;

static long bad = 0;
static bool same(double x, double y) { return bitsOf(x) == bitsOf(y) || (std::isnan(x) && std::isnan(y)); }
static void check(double a, double b) {
  if (!same(intDiv(a, b), a / b) || !same(intDiv(1.0, b), 1.0 / b) || !same(intSqrt(a), std::sqrt(a)) ||
      isLess(a, b) != (a < b) || isLessEq(a, b) != (a <= b) || isPos(a) != (a > 0.0) || isNeg(a) != (a < 0.0)) {
    if (bad++ < 5) std::printf("differs: %a %a\n", a, b);
  }
}
int main(int argc, char **argv) {
  const long n = argc > 1 ? std::atol(argv[1]) : 100000;
  const double sp[] = {0.0, -0.0, 1.0, -1.0, INFINITY, -INFINITY, NAN, 5e-324, -5e-324, 2.2250738585072014e-308,
                       1.7976931348623157e308, 1e-310, 4.0, 2.0, 0.25, 3.0, 1e-160, -1e160, 1.0 + 0x1p-52,
                       2.0 - 0x1p-52, 0x1.fffffffffffffp-1};
  for (double a : sp)
    for (double b : sp) check(a, b);
  std::mt19937_64 g(7);
  for (long t = 0; t < n; ++t) {
    uint64_t ea = g() % 2047, eb = g() % 2047, ma = g() >> 12, mb = g() >> 12;
    if (t % 2) { ea = 1000 + g() % 40; eb = 1000 + g() % 40; }
    if (t % 5 == 0) ma &= ~((1ull << (g() % 52)) - 1);
    if (t % 7 == 0) mb = (g() % 2) ? (1ull << (g() % 52)) : 0xfffffffffffffull - (g() % 4);
    if (t % 11 == 0) { const uint64_t r = (g() >> 38) | 1; ma = (r * r) & 0xfffffffffffffull; }  // near squares
    const uint64_t s = 1ull << 63;
    check(ofBits((g() & s) | ea << 52 | ma), ofBits((g() & s) | eb << 52 | mb));
  }
  std::printf("%ld\n", bad);
  return 0;
}
