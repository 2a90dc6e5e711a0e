// Sums of products of doubles on the integer pipe.
//
// The GB300 runs one FP64 instruction per sub-partition in about 64 cycles and
// a 32x32+64-bit integer multiply-add in 2.3 (measured), so a sum of products
// whose terms share a scale is formed in fixed point: every factor becomes a
// 56-bit integer in units of its block's largest magnitude, is split into two
// 28-bit halves, and the partial products are accumulated exactly in 64-bit
// integers (Karatsuba: three multiplies per product).  The only rounding is
// that of the factors to their units, 2^-55 of the block's largest magnitude,
// and of the result to a double; a sum in FP64 rounds every term and every
// partial sum at 2^-53 of their size.  Where a block's terms are of like size
// the fixed point is the more accurate; fixCellWeights says which cells' are.
//
// Host and device code (no CUDA types): tests/test_fixedsum_cpu.py and
// tests/test_fixedsum_cells_cpu.py compare it with exact rational sums.
#pragma once
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define RFLU_HD __host__ __device__
#else
#define RFLU_HD
#endif

namespace rflu {

// A finite double as (signed mantissa << 2) * 2^(e - 1077), e its biased
// exponent; e = 0 only for zero.  kFixBad marks what the fixed-point sums do
// not take (denormals, infinities, NaN, magnitudes outside about 2^-500 ..
// 2^500): it is larger than every other e, so that it survives a maximum.
constexpr int kFixBad = 4095, kFixEmin = 523, kFixEmax = 1523;
constexpr int kFixMaxTerms = 64;   // terms per sum that cannot overflow
constexpr int kFixBadScale = 1 << 20;

struct FixNum {
  int64_t m;
  int e;
};
RFLU_HD inline FixNum fixOf(double x) {
  uint64_t b;
#ifdef __CUDA_ARCH__
  b = (uint64_t)__double_as_longlong(x);
#else
  std::memcpy(&b, &x, 8);
#endif
  FixNum r;
  const int e = (int)((b >> 52) & 0x7ff);
  const int64_t m = (int64_t)(((b & 0xfffffffffffffull) | 0x10000000000000ull) << 2);
  const bool zero = (b << 1) == 0;
  r.m = zero ? 0 : ((int64_t)b < 0 ? -m : m);
  r.e = zero ? 0 : (e < kFixEmin || e > kFixEmax) ? kFixBad : e;
  return r;
}

// The number in units of 2^(eMax - 1077), eMax >= e (rounded down).
RFLU_HD inline int64_t fixAt(int64_t m, int e, int eMax) {
  const int s = eMax - e;
  return m >> (s < 63 ? s : 63);
}

// A weight in units of 2^(x - 55) with |w| < 2^x, in two signed halves: w =
// (hi * 2^28 + lo) units, |hi| <= 2^27, -2^27 <= lo < 2^27.
struct FixHalves {
  int hi, lo;
};
RFLU_HD inline FixHalves fixSplit(int64_t v) {
  FixHalves h;
  h.hi = (int)((v + (1 << 27)) >> 28);
  h.lo = (int)((uint32_t)v - ((uint32_t)h.hi << 28));
  return h;
}

// One sum of products; the weights' halves and the differences' halves are
// formed once per member and used in 15 sums.  |difference| <= 2^56 units.
struct FixSum {
  int64_t hh, ss, ll;
};
RFLU_HD inline void fixAdd(FixSum &a, int wh, int wl, int ws, int dh, int dl, int ds) {
  a.hh += (int64_t)wh * dh;
  a.ll += (int64_t)wl * dl;
  a.ss += (int64_t)ws * ds;  // ws = wh + wl, ds = dh + dl: hh + ll + the cross terms
}

RFLU_HD inline int fixClz(uint64_t x) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)x);
#else
  return __builtin_clzll(x);
#endif
}

// The sum as a double: units of 2^scale; rounded to nearest.
RFLU_HD inline double fixResult(const FixSum &a, int scale) {
  const int64_t mid = a.ss - a.hh - a.ll;
  // a.hh * 2^56 + mid * 2^28 + a.ll as h * 2^56 + low, 0 <= low < 2^56
  const int64_t m1 = mid + (a.ll >> 28);
  int64_t h = a.hh + (m1 >> 28);
  uint64_t low = ((uint64_t)(m1 & 0xfffffff) << 28) | (uint64_t)(a.ll & 0xfffffff);
  const bool neg = h < 0;
  if (neg) {
    h = low ? ~h : -h;
    low = low ? (1ull << 56) - low : 0;
  }
  const uint64_t H = (uint64_t)h, L = low << 8;
  if ((H | L) == 0) return 0.0;
  int lz;
  uint64_t top;
  if (H) {
    lz = fixClz(H);
    top = (H << lz) | (lz ? L >> (64 - lz) : 0);
  } else {
    const int l = fixClz(L);
    lz = 64 + l;
    top = L << l;
  }
  // top's leading bit stands for 2^(119 - lz) units
  const int e = 119 - lz + scale + 1022;
  const uint64_t bits = ((uint64_t)e << 52) + (top >> 11) + ((top >> 10) & 1) + (neg ? 1ull << 63 : 0);
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)bits);
#else
  double d;
  std::memcpy(&d, &bits, 8);
  return d;
#endif
}

// The smallest exponent of a block's largest weight: below it the smallest
// result (values of 2^-500) would leave the normal doubles.
constexpr int kFixWeightEmin = 610;

// |w| < 2^x for the largest magnitude of a block of weights: its biased
// exponent minus 1022; kFixBadScale for what the sums do not take (or none).
RFLU_HD inline int fixScale(int eMax) {
  return (eMax < kFixWeightEmin || eMax == kFixBad) ? kFixBadScale : eMax - 1022;
}
// A weight of that block in units of 2^(x - 55), rounded to nearest.
RFLU_HD inline int64_t fixWeight(double w, int eMax) {
  const FixNum f = fixOf(w);
  const int s = eMax - f.e;
  if (s > 60) return 0;
  return s == 0 ? f.m : ((f.m >> (s - 1)) + 1) >> 1;
}

// The exponent of the largest of a cell's least-squares weights, their block's,
// or kFixNoWeights where the cell's sums stay in FP64.
//
// A weight is rounded to 2^-56 of the block's largest, so a cell loses digits
// where its weights differ widely: those along a cell's long axis are smaller by
// its aspect ratio, and a member whose weights are all small carries a large
// difference, whose product's digits FP64 keeps.  The sums take the cells whose
// components' largest weights lie within kFixCompSpread exponents of each other
// and whose members' largest weights within kFixMemberSpread.  Error against 128
// bits on hexahedra (26 members) and jittered tetrahedra (40), smooth, random and
// discontinuous fields, in units of sum |w||d|: root mean square of cubic cells
// 2e-17 to 7e-17 (hexahedra) and 2e-17 to 1.1e-16 (tetrahedra) against the FP64
// sum's 5e-17 to 1.1e-16 and 6e-17 to 1.4e-16 (largest 2.9e-16 and 8.9e-16 against
// 6.2e-16 and 8.5e-16); of cells of aspect 2 at most the FP64 sum's.  Beyond, the
// fixed point falls behind: aspect 8 in x 5e-16 against 1.2e-16, aspect 1e4
// 5e-13, with an exponent per component too.  (Members up to 2^5 apart would
// leave out 11 of 196,608 jittered tetrahedra, whose warps' FP64 loops held up
// every launch: tangent and adjoint 2595 -> 2681 us.)
constexpr int kFixCompSpread = 2, kFixMemberSpread = 6;
constexpr int kFixNoWeights = -1;
template <typename R>
RFLU_HD inline int fixCellWeights(const R *wx, const R *wy, const R *wz, int n) {
  int e[3] = {0, 0, 0}, top = 0, low = kFixBad;
  for (int k = 0; k < n; ++k) {
    const int x = fixOf((double)wx[k]).e, y = fixOf((double)wy[k]).e, z = fixOf((double)wz[k]).e;
    const int xy = x > y ? x : y, m = xy > z ? xy : z;
    e[0] = x > e[0] ? x : e[0];
    e[1] = y > e[1] ? y : e[1];
    e[2] = z > e[2] ? z : e[2];
    top = m > top ? m : top;
    low = m < low ? m : low;
  }
  int least = e[0] < e[1] ? e[0] : e[1];
  least = e[2] < least ? e[2] : least;
  if (n < 1 || n > kFixMaxTerms || fixScale(top) == kFixBadScale || top - least > kFixCompSpread ||
      top - low > kFixMemberSpread)
    return kFixNoWeights;
  return top;
}

}  // namespace rflu
