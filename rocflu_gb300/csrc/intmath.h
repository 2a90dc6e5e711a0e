// FP64 division and square root, and comparisons, on the integer pipe.
//
// On the GB300 an IEEE division is eight FP64 instructions, a square root
// about ten, at 64 cycles of a sub-partition each.  Here the significand's
// reciprocal (or reciprocal root) starts from the FP32 unit's approximation
// and takes one cubic step (Householder's method of order two: with e = 1 - x
// y0, y = y0 (1 + e + e^2); for the root, e = 1 - x y0^2, y = y0 (1 + e/2 +
// 3 e^2/8)) in 64-bit integers, 2^-60 or better; the quotient or root is one
// 64-bit product, and its remainder, an exact integer, settles the rounding:
// the results are the IEEE operations' bits.  Zero, denormal, infinite and NaN
// operands and results outside the normal range go to the IEEE operation.
//
// Host and device code (no CUDA types): tests/test_intmath_cpu.py compares it
// with the C library's operations bit by bit, rflu_gpu_check_conversions
// compares the device's.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define RFLU_HD __host__ __device__
#else
#define RFLU_HD
#endif

namespace rflu {

RFLU_HD inline uint64_t bitsOf(double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t b;
  std::memcpy(&b, &x, 8);
  return b;
#endif
}
RFLU_HD inline double ofBits(uint64_t b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double x;
  std::memcpy(&x, &b, 8);
  return x;
#endif
}
RFLU_HD inline uint64_t mulHi(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

// x > 0, x < 0 and a < b as the FP64 pipe's comparisons decide them (false for
// NaN, -0 equal to +0).
RFLU_HD inline bool isPos(double x) { return bitsOf(x) - 1 < 0x7ff0000000000000ull; }
RFLU_HD inline bool isNeg(double x) { return bitsOf(x) - 0x8000000000000001ull < 0x7ff0000000000000ull; }
RFLU_HD inline bool isLess(double a, double b) {
  const int64_t x = (int64_t)bitsOf(a), y = (int64_t)bitsOf(b);
  const int64_t sx = x >> 63, sy = y >> 63;
  const int64_t mx = x & 0x7fffffffffffffffll, my = y & 0x7fffffffffffffffll;
  const int64_t kx = (mx ^ sx) - sx, ky = (my ^ sy) - sy;
  constexpr int64_t inf = 0x7ff0000000000000ll;
  return kx < ky && mx <= inf && my <= inf;
}
RFLU_HD inline bool isLessEq(double a, double b) {
  const int64_t x = (int64_t)bitsOf(a), y = (int64_t)bitsOf(b);
  const int64_t sx = x >> 63, sy = y >> 63;
  const int64_t mx = x & 0x7fffffffffffffffll, my = y & 0x7fffffffffffffffll;
  const int64_t kx = (mx ^ sx) - sx, ky = (my ^ sy) - sy;
  constexpr int64_t inf = 0x7ff0000000000000ll;
  return kx <= ky && mx <= inf && my <= inf;
}

// A double as an integer in the doubles' order (-0 just below +0; NaN beyond the
// infinities), and back: minima and maxima of many values as integer ones.
RFLU_HD inline int64_t orderKey(double x) {
  const int64_t b = (int64_t)bitsOf(x);
  return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}
RFLU_HD inline double ofKey(int64_t k) { return ofBits((uint64_t)(k ^ ((k >> 63) & 0x7fffffffffffffffll))); }
constexpr int64_t kKeyInf = 0x7ff0000000000000ll;  // orderKey(infinity); a NaN's key is above it or below -1 - it

// The FP32 approximations the iterations start from, as 32-bit fractions of
// an argument's significand: f has the leading 24 bits; results in (1/2, 1].
RFLU_HD inline uint32_t seedFraction(float r) {
  uint32_t b;
#ifdef __CUDA_ARCH__
  b = __float_as_uint(r);
#else
  std::memcpy(&b, &r, 4);
#endif
  return b >= 0x3f800000u ? 0xffffffffu : ((b & 0x7fffffu) | 0x800000u) << 8;
}
RFLU_HD inline uint32_t recipSeed(uint32_t floatBits) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(floatBits)));
  return seedFraction(r);
#else
  float f;
  std::memcpy(&f, &floatBits, 4);
  return seedFraction(1.0f / f);
#endif
}
RFLU_HD inline uint32_t rootSeed(uint32_t floatBits) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(floatBits)));
  return seedFraction(r);
#else
  float f;
  std::memcpy(&f, &floatBits, 4);
  return seedFraction(1.0f / std::sqrt(f));
#endif
}

// y0 (1 + d) for a 32-bit fraction y0 and |d| < 2^-20 in units of 2^-u, as a
// 64-bit fraction.
template <int u>
RFLU_HD inline uint64_t stepFraction(uint32_t y0, int64_t d) {
  const uint64_t lo = (uint64_t)y0 * (uint32_t)d;
  const int64_t hi = (int64_t)y0 * (int)(d >> 32);
  return ((uint64_t)y0 << 32) + (lo >> (u - 32)) + ((uint64_t)hi << (64 - u));
}

// 2^127 / m for m = 2^63 .. 2^64 - 1 (the reciprocal of m / 2^63 as a 64-bit
// fraction).
RFLU_HD inline uint64_t recipFraction(uint64_t m) {
  const uint32_t y0 = recipSeed(0x3f800000u | (uint32_t)((m >> 40) & 0x7fffff));
  const uint64_t p = (uint64_t)(uint32_t)(m >> 32) * y0 + (((uint64_t)(uint32_t)m * y0) >> 32);
  const int64_t e = (int64_t)(0x8000000000000000ull - p);  // 1 - x y0 in units of 2^-63
  const int es = (int)(e >> 20);
  return stepFraction<63>(y0, e + (((int64_t)es * es) >> 23));
}

// The double (-1)^neg 2^(e - 1075) q for a 53-bit q (or 2^53).
RFLU_HD inline double packDouble(uint64_t neg, int e, uint64_t q) {
  return ofBits((neg << 63) + ((uint64_t)(e - 1) << 52) + q);
}

#ifdef __CUDA_ARCH__
// out of line: the rare operands' code stays out of the kernels' main path
__device__ __noinline__ static double ieeeDiv(double a, double b) { return a / b; }
__device__ __noinline__ static double ieeeSqrt(double x) { return sqrt(x); }
#else
inline double ieeeDiv(double a, double b) { return a / b; }
inline double ieeeSqrt(double x) { return std::sqrt(x); }
#endif

// ma / mb 2^52 (or 2^53 when ma < mb) to the nearest integer, for 53-bit
// significands; below: which of the two.
RFLU_HD inline uint64_t quotient53(uint64_t ma, uint64_t mb, bool &below) {
  below = ma < mb;
  const uint64_t hi = mulHi(ma << 11, recipFraction(mb << 11));  // ma / mb 2^63, a few units off
  uint64_t q = ((hi >> (below ? 9 : 10)) + 1) >> 1;
  // the remainder, |r| < mb: a quotient of two 53-bit integers is never
  // half-way between two 53-bit ones
  const int64_t r2 = (int64_t)(((ma << (below ? 53 : 52)) - q * mb) << 1);
  if (r2 > (int64_t)mb) ++q;
  else if (r2 < -(int64_t)mb) --q;
  return q;
}

RFLU_HD inline double intDiv(double a, double b) {
  const uint64_t x = bitsOf(a), y = bitsOf(b);
  const int ea = (int)((x >> 52) & 0x7ff), eb = (int)((y >> 52) & 0x7ff);
  const int e = ea - eb + 1023;
  const uint64_t neg = (x ^ y) >> 63;
  if ((unsigned)(eb - 1) < 2046u) {
    // a normal, the result normal before and after its rounding
    if ((unsigned)(ea - 1) < 2046u && (unsigned)(e - 2) < 2044u) {
      constexpr uint64_t one = 0x10000000000000ull;
      bool below;
      const uint64_t q = quotient53((x & (one - 1)) | one, (y & (one - 1)) | one, below);
      return packDouble(neg, below ? e - 1 : e, q);
    }
    if ((x << 1) == 0) return ofBits(neg << 63);  // a zero over a normal number
  }
  return ieeeDiv(a, b);
}

RFLU_HD inline double intSqrt(double a) {
  const uint64_t x = bitsOf(a);
  const int ex = (int)(x >> 52);  // with the sign: a negative number's is above 2046
  if ((unsigned)(ex - 1) < 2046u) {
    const int odd = (ex & 1) ^ 1;  // the unbiased exponent is odd
    const uint64_t m53 = (x & 0xfffffffffffffull) | 0x10000000000000ull;
    const uint64_t m = m53 << (10 + odd);  // v = m / 2^62 in [1, 4)
    const uint32_t y0 = rootSeed((uint32_t)(127 + odd) << 23 | (uint32_t)((x >> 29) & 0x7fffff));
    const uint64_t t = mulHi(m, (uint64_t)y0 * y0);
    const int64_t e = (int64_t)(0x4000000000000000ull - t);  // 1 - v y0^2 in units of 2^-62
    const int es = (int)(e >> 20);
    const uint64_t y = stepFraction<62>(y0, (e >> 1) + ((3 * ((int64_t)es * es)) >> 25));
    uint64_t s = ((mulHi(m, y) >> 9) + 1) >> 1;  // the root of v times 2^52
    // the remainder of m53 2^(52 + odd): the root of a 53-bit integer is never
    // half-way between two of them
    const int64_t r = (int64_t)((m53 << (52 + odd)) - s * s);
    if (r > (int64_t)s) ++s;
    else if (r <= -(int64_t)s) --s;
    return packDouble(0, ((ex - 1023 - odd) >> 1) + 1023, s);
  }
  if ((x << 1) == 0) return a;
  return ieeeSqrt(a);
}

}  // namespace rflu
