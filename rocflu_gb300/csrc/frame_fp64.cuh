// The eigen-frame of RFLU_PREC_FP64's velocity limiter.
//
// Device code; the same source compiles for the host, where
// tests/test_frame_cpu.py compares it with symmetricEigen3 in wider arithmetic.
#pragma once
#include <algorithm>
#include <cmath>

#include "convert.cuh"
#include "intmath.h"
#include "physics.cuh"

#if defined(__CUDACC__)
#define RFLU_FRAME_FN __device__ inline
#else
#define RFLU_FRAME_FN inline
#endif

namespace rflu {

#if defined(__CUDACC__)
RFLU_FRAME_FN float fastDivide(float a, float b) { return __fdividef(a, b); }
RFLU_FRAME_FN float fastRoot(float x) { return rsqrtf(x); }
#else
RFLU_FRAME_FN float fastDivide(float a, float b) { return a / b; }
RFLU_FRAME_FN float fastRoot(float x) { return 1.f / std::sqrt(x); }
using std::max;
#endif

// FP32: cyclic Jacobi rotations as symmetricEigen3 takes them, each angle's
// tangent from one division and its cosine from one reciprocal root, to
// off-diagonals of 3e-8: the start of strainFrame64's FP64 sweep.  The mixed
// mode's own frame stays with symmetricEigen3: with these rotations 10 steps of
// 2.1 M cells took 16.0 -> 15.7 ms but ended 8.8e-8 from the FP64 result
// instead of 3.7e-8, at either tolerance.
RFLU_FRAME_FN void jacobi3(float &r0, float &r1, float &r2, float r01, float r02, float r12, float *vec) {
  const float total = r0 * r0 + r1 * r1 + r2 * r2 + 2.f * (r01 * r01 + r02 * r02 + r12 * r12);
#pragma unroll
  for (int k = 0; k < 9; ++k) vec[k] = 0.f;
  vec[0] = vec[4] = vec[8] = 1.f;
  const float tol = 8.8e-16f * total;
  // rotation in the plane of p and q; o the third axis
  auto rotate = [&](float &pp, float &qq, float &pq, float &op, float &oq, float *vp, float *vq) {
    const float d = qq - pp, b = 2.f * pq, h = d * d + b * b;
    if (pq == 0.f || !(h > 0.f)) return;  // nothing to turn, or both squares underflow
    const float t = fastDivide(b, d + copysignf(sqrtf(h), d));
    const float c = fastRoot(t * t + 1.f), s = t * c;
    pp = pp - t * pq;
    qq = qq + t * pq;
    pq = 0.f;
    const float a = op;
    op = c * a - s * oq;
    oq = s * a + c * oq;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float x = vp[k];
      vp[k] = c * x - s * vq[k];
      vq[k] = s * x + c * vq[k];
    }
  };
  for (int sweep = 0; sweep < 50; ++sweep) {
    if (r01 * r01 + r02 * r02 + r12 * r12 <= tol) break;
    rotate(r0, r1, r01, r02, r12, vec, vec + 3);
    rotate(r0, r2, r02, r01, r12, vec, vec + 6);
    rotate(r1, r2, r12, r01, r02, vec + 3, vec + 6);
  }
}

// Eigenvalues (ascending) and eigenvectors (columns) of a symmetric matrix in
// RFLU_PREC_FP64, to symmetricEigen3's tolerance (off-diagonals below 1e-12 of
// the matrix): the rotations run in FP32 on the scaled matrix first (jacobi3),
// their product is orthonormalised in FP64 and the matrix turned by it, which
// leaves off-diagonals near 1e-7, and one FP64 sweep of small angles ends it:
// some 155 FP64 instructions, counted in the source, instead of 90 per sweep and
// four or five sweeps.  What is left off the diagonal, of the matrix's norm and
// in 128-bit arithmetic over 40,000 normal matrices: root mean square 2.5e-15,
// largest 1.2e-13 (symmetricEigen3 1.1e-13 and 1e-12).  Two steps of 13,824 cells
// end 9.5e-17 from a computation with converged axes, with symmetricEigen3's
// 5.0e-16.
RFLU_FRAME_FN void strainFrame64(const double *m, double *vec, double *val) {
  const double s00 = m[0], s11 = m[4], s22 = m[8], s01 = m[3], s02 = m[6], s12 = m[7];
  auto expOf = [](double x) { return (int)(bitsOf(x) >> 52) & 0x7ff; };
  const int e = max(max(max(expOf(s00), expOf(s11)), max(expOf(s22), expOf(s01))), max(expOf(s02), expOf(s12)));
  // zero, or far from one: the rotations' squares of remainders 2^-53 and
  // 2^-106 of the matrix stay normal numbers between 2^-200 and 2^200
  if (e < 823 || e > 1223) {
    symmetricEigen3(m, vec, val);
    return;
  }
  // in [0, 2) of the largest entry's power of two, cut to 24 bits
  auto scaled = [&](double x) {
    const uint64_t b = bitsOf(x);
    const int k = expOf(x) - e + 127;
    return k <= 0 ? 0.f
                  : cvt::fromBits((unsigned)(b >> 32) & 0x80000000u | (unsigned)k << 23 | (unsigned)(b >> 29) & 0x7fffffu);
  };
  float f0 = scaled(s00), f1 = scaled(s11), f2 = scaled(s22), vf[9];
  jacobi3(f0, f1, f2, scaled(s01), scaled(s02), scaled(s12), vf);
  double *a = vec, *b = vec + 3, *c = vec + 6;
#pragma unroll
  for (int k = 0; k < 6; ++k) vec[k] = f2d(vf[k]);
  // a, then b, orthonormal from near it: 1/sqrt(1 + x) = 1 - x/2 + 3 x^2/8
  auto unit = [](double *v) {
    const double x = v[0] * v[0] + v[1] * v[1] + v[2] * v[2] - 1.0;
    const double s = x * (0.375 * x - 0.5) + 1.0;
    v[0] = v[0] * s;
    v[1] = v[1] * s;
    v[2] = v[2] * s;
  };
  unit(a);
  const double ab = a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
#pragma unroll
  for (int k = 0; k < 3; ++k) b[k] = b[k] - ab * a[k];
  unit(b);
  c[0] = a[1] * b[2] - a[2] * b[1];
  c[1] = a[2] * b[0] - a[0] * b[2];
  c[2] = a[0] * b[1] - a[1] * b[0];
  double r[3], r01, r02, r12;
  {
    auto times = [&](const double *v, double *y) {
      y[0] = s00 * v[0] + s01 * v[1] + s02 * v[2];
      y[1] = s01 * v[0] + s11 * v[1] + s12 * v[2];
      y[2] = s02 * v[0] + s12 * v[1] + s22 * v[2];
    };
    auto dot = [](const double *x, const double *y) { return x[0] * y[0] + x[1] * y[1] + x[2] * y[2]; };
    double y[3];
    times(a, y);
    r[0] = dot(a, y);
    r01 = dot(b, y);
    r02 = dot(c, y);
    times(b, y);
    r[1] = dot(b, y);
    r12 = dot(c, y);
    times(c, y);
    r[2] = dot(c, y);
  }
  auto rotate = [](double &pp, double &qq, double &pq, double &op, double &oq, double *vp, double *vq) {
    if (!nonZero_(pq)) return;
    const double d = qq - pp;
    double t, cs;
    const int ed = (int)(bitsOf(d) >> 52) & 0x7ff, ep = (int)(bitsOf(pq) >> 52) & 0x7ff;
    if (ed - ep >= 17) {  // |pq / d| < 2^-16: the angle's tangent to 2^-64 from its series
      const double x = div_(pq, d);
      t = x - x * (x * x);
      cs = 1.0 - 0.5 * (t * t);
    } else {
      const double bb = 2.0 * pq, h = d * d + bb * bb;
      if (!isPos(h)) return;  // both squares underflow: nothing beside the matrix
      t = div_(bb, d + copysign_(sqrt_(h), d));
      cs = div_(1.0, sqrt_(t * t + 1.0));
    }
    const double sn = t * cs, x = op;
    pp = pp - t * pq;
    qq = qq + t * pq;
    pq = 0.0;
    op = cs * x - sn * oq;
    oq = sn * x + cs * oq;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double y = vp[k];
      vp[k] = cs * y - sn * vq[k];
      vq[k] = sn * y + cs * vq[k];
    }
  };
  const double tol = 1.0e-24 * (r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
  for (int sweep = 0; sweep < 50; ++sweep) {
    if (lessEq_(r01 * r01 + r02 * r02 + r12 * r12, tol)) break;
    rotate(r[0], r[1], r01, r02, r12, a, b);
    rotate(r[0], r[2], r02, r01, r12, a, c);
    rotate(r[1], r[2], r12, r01, r02, b, c);
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) val[k] = r[k];
  sortAxes(val, vec);
}

}  // namespace rflu
