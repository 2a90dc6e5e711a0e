// Forward-mode dual numbers: a value and N directional derivatives.  The
// point-wise physics of physics.cuh is generic in its scalar type, so the same
// flux, reconstruction and limiter code evaluated on Dual<N> gives exact
// local Jacobians (tangent kernels) and, for N inputs of a face, the rows of
// the transposed flux Jacobian (adjoint kernels).  Comparisons and branch
// decisions use the value only: derivatives follow the active branch.
#pragma once
#include <cmath>

#include "intmath.h"

namespace rflu {

// Division, square root and comparisons as the point-wise code calls them.
// On the device FP64 ones run on the integer pipe with the IEEE operations'
// results (intmath.h): about 110 cycles of a sub-partition instead of 530 for
// a division and 100 instead of 650 for a root, 5 to 20 instead of 76 for a
// comparison.  Other scalar types use the language's operators.
template <typename A, typename B>
__host__ __device__ inline auto div_(const A &a, const B &b) -> decltype(a / b) { return a / b; }
template <typename S> __host__ __device__ inline bool less_(const S &a, const S &b) { return a < b; }
template <typename S> __host__ __device__ inline bool lessEq_(const S &a, const S &b) { return a <= b; }
template <typename S> __host__ __device__ inline bool pos_(const S &a) { return a > S(0); }
template <typename S> __host__ __device__ inline bool neg_(const S &a) { return a < S(0); }
template <typename S> __host__ __device__ inline bool nonZero_(const S &a) { return a != S(0); }
__host__ __device__ inline bool isNan_(double a) { return (bitsOf(a) << 1) > 0xffe0000000000000ull; }
__host__ __device__ inline float sqrt_(float x) { return sqrtf(x); }
#ifdef __CUDA_ARCH__
__device__ inline double div_(double a, double b) { return intDiv(a, b); }
__device__ inline double sqrt_(double x) { return intSqrt(x); }
__device__ inline bool less_(double a, double b) { return isLess(a, b); }
__device__ inline bool lessEq_(double a, double b) { return isLessEq(a, b); }
__device__ inline bool pos_(double a) { return isPos(a); }
__device__ inline bool neg_(double a) { return isNeg(a); }
__device__ inline bool nonZero_(double a) { return (bitsOf(a) << 1) != 0; }
#else
__host__ inline double sqrt_(double x) { return std::sqrt(x); }
#endif

// T is the arithmetic type of value and derivatives: double in the FP64
// modes, float for the mixed mode's flux and limiter Jacobians.
template <int N, typename T = double>
struct Dual {
  T v;
  T d[N];
  __host__ __device__ Dual() : v(T(0)) {
#pragma unroll
    for (int k = 0; k < N; ++k) d[k] = T(0);
  }
  __host__ __device__ Dual(double x) : v(T(x)) {  // NOLINT: constants promote implicitly
#pragma unroll
    for (int k = 0; k < N; ++k) d[k] = T(0);
  }
  __host__ __device__ static Dual seed(double x, int k) {
    Dual r(x);
    r.d[k] = T(1);
    return r;
  }
  // rounding between arithmetic types (the mixed mode's FP64 first-order
  // paths feeding FP32 fluxes)
  template <typename U>
  __host__ __device__ explicit Dual(const Dual<N, U> &o) : v(T(o.v)) {
#pragma unroll
    for (int k = 0; k < N; ++k) d[k] = T(o.d[k]);
  }
};

#define RFLU_DUAL_BINOP(op, expr_d)                                                                \
  template <int N, typename T>                                                                     \
  __host__ __device__ inline Dual<N, T> operator op(const Dual<N, T> &a, const Dual<N, T> &b) {    \
    Dual<N, T> r;                                                                                  \
    r.v = a.v op b.v;                                                                    \
    _Pragma("unroll") for (int k = 0; k < N; ++k) r.d[k] = expr_d;                       \
    return r;                                                                            \
  }
RFLU_DUAL_BINOP(+, a.d[k] + b.d[k])
RFLU_DUAL_BINOP(-, a.d[k] - b.d[k])
RFLU_DUAL_BINOP(*, a.d[k] * b.v + a.v * b.d[k])
#undef RFLU_DUAL_BINOP

// With a number that carries no derivative (a geometric factor, a parameter of
// the gas): the products with its zero derivatives are not formed.
template <typename D> struct Same { using type = D; };
template <int N, typename T>
__host__ __device__ inline Dual<N, T> operator*(const Dual<N, T> &a, const typename Same<T>::type &b) {
  Dual<N, T> r;
  r.v = a.v * b;
#pragma unroll
  for (int k = 0; k < N; ++k) r.d[k] = a.d[k] * b;
  return r;
}
template <int N, typename T>
__host__ __device__ inline Dual<N, T> operator*(const typename Same<T>::type &a, const Dual<N, T> &b) { return b * a; }
template <int N, typename T>
__host__ __device__ inline Dual<N, T> operator+(const Dual<N, T> &a, const typename Same<T>::type &b) {
  Dual<N, T> r = a;
  r.v = a.v + b;
  return r;
}
template <int N, typename T>
__host__ __device__ inline Dual<N, T> operator+(const typename Same<T>::type &a, const Dual<N, T> &b) { return b + a; }
template <int N, typename T>
__host__ __device__ inline Dual<N, T> operator-(const Dual<N, T> &a, const typename Same<T>::type &b) {
  Dual<N, T> r = a;
  r.v = a.v - b;
  return r;
}
template <int N, typename T>
__host__ __device__ inline Dual<N, T> operator-(const typename Same<T>::type &a, const Dual<N, T> &b) {
  Dual<N, T> r;
  r.v = a - b.v;
#pragma unroll
  for (int k = 0; k < N; ++k) r.d[k] = -b.d[k];
  return r;
}
template <int N, typename T>
__host__ __device__ inline Dual<N, T> operator/(const typename Same<T>::type &a, const Dual<N, T> &b) {
  Dual<N, T> r;
  const T ib = div_(T(1), b.v);
  r.v = div_(a, b.v);
  const T s = -(r.v * ib);
#pragma unroll
  for (int k = 0; k < N; ++k) r.d[k] = s * b.d[k];
  return r;
}

template <int N, typename T>
__host__ __device__ inline Dual<N, T> operator/(const Dual<N, T> &a, const Dual<N, T> &b) {
  Dual<N, T> r;
  const T ib = div_(T(1), b.v);
  r.v = div_(a.v, b.v);
#pragma unroll
  for (int k = 0; k < N; ++k) r.d[k] = (a.d[k] - r.v * b.d[k]) * ib;
  return r;
}
template <int N, typename T>
__host__ __device__ inline Dual<N, T> operator-(const Dual<N, T> &a) {
  Dual<N, T> r;
  r.v = -a.v;
#pragma unroll
  for (int k = 0; k < N; ++k) r.d[k] = -a.d[k];
  return r;
}
template <int N, typename T> __host__ __device__ inline bool operator<(const Dual<N, T> &a, const Dual<N, T> &b) { return less_(a.v, b.v); }
template <int N, typename T> __host__ __device__ inline bool operator>(const Dual<N, T> &a, const Dual<N, T> &b) { return less_(b.v, a.v); }
template <int N, typename T> __host__ __device__ inline bool operator<=(const Dual<N, T> &a, const Dual<N, T> &b) { return lessEq_(a.v, b.v); }
template <int N, typename T> __host__ __device__ inline bool operator>=(const Dual<N, T> &a, const Dual<N, T> &b) { return lessEq_(b.v, a.v); }
template <int N, typename T> __host__ __device__ inline bool operator==(const Dual<N, T> &a, const Dual<N, T> &b) { return a.v == b.v; }
template <int N, typename T> __host__ __device__ inline bool operator!=(const Dual<N, T> &a, const Dual<N, T> &b) { return a.v != b.v; }

template <int N, typename T>
__host__ __device__ inline Dual<N, T> sqrt_(const Dual<N, T> &a) {
  Dual<N, T> r;
  r.v = sqrt_(a.v);
  const T h = pos_(r.v) ? div_(T(0.5), r.v) : T(0);
#pragma unroll
  for (int k = 0; k < N; ++k) r.d[k] = a.d[k] * h;
  return r;
}
// x ** y with y a constant of the gas model: d(x^y) = y x^(y-1) dx
template <int N, typename T>
__host__ __device__ inline Dual<N, T> powConstExp(const Dual<N, T> &a, const Dual<N, T> &y) {
  Dual<N, T> r;
  r.v = pow(a.v, y.v);
  const T s = y.v * pow(a.v, y.v - T(1));
#pragma unroll
  for (int k = 0; k < N; ++k) r.d[k] = a.d[k] * s;
  return r;
}
template <int N, typename T>
__host__ __device__ inline Dual<N, T> fabs_(const Dual<N, T> &a) {
  return neg_(a.v) ? -a : a;
}
template <int N, typename T>
__host__ __device__ inline Dual<N, T> copysign_(const Dual<N, T> &a, const Dual<N, T> &b) {
  // d/db copysign(a, b) = 0 away from b = 0
  const bool flip = (signbit(a.v) != signbit(b.v));
  return flip ? -a : a;
}

template <typename S> struct ValueOf { __host__ __device__ static double get(const S &x) { return (double)x; } };
template <int N, typename T> struct ValueOf<Dual<N, T>> {
  __host__ __device__ static double get(const Dual<N, T> &x) { return (double)x.v; }
};

}  // namespace rflu
