// strainFrame64 (frame_fp64.cuh) on the host.  Mode "sizes": matrices of small
// integers times 2^e over the doubles' range; prints how many frames hold a
// value that is not finite, are not orthonormal to 1e-14, or leave more than
// 1.01e-12 of the norm off the diagonal.  Mode "residual": normal matrices and
// shears; prints per family the root mean square and the largest off-diagonal
// remainder, of the norm, of symmetricEigen3 and of strainFrame64, and the
// orthonormality of both.
#define __host__
#define __device__
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>

#include "frame_fp64.cuh"

using namespace rflu;

#if defined(__x86_64__)
typedef __float128 Wide;
#else
typedef long double Wide;  // 128 bits on aarch64
#endif

// what V^T M V holds off its diagonal, and V^T V off the identity
template <typename Wide>
static void remainders(const double *m, const double *v, double &off, double &orth) {
  Wide mo = 0, mq = 0;
  for (int i = 0; i < 3; ++i)
    for (int j = i; j < 3; ++j) {
      Wide s = 0, o = i == j ? -1 : 0;
      for (int x = 0; x < 3; ++x) {
        o += (Wide)v[x + 3 * i] * v[x + 3 * j];
        for (int y = 0; y < 3; ++y) s += (Wide)v[x + 3 * i] * m[x + 3 * y] * v[y + 3 * j];
      }
      if (i != j) mo = std::max(mo, s < 0 ? -s : s);
      mq = std::max(mq, o < 0 ? -o : o);
    }
  off = (double)mo;
  orth = (double)mq;
}
static double norm(const double *m) {
  double top = 0.0, s = 0.0;
  for (int k = 0; k < 9; ++k) top = std::max(top, std::fabs(m[k]));
  if (top == 0.0) return 0.0;
  for (int k = 0; k < 9; ++k) s += (m[k] / top) * (m[k] / top);
  return top * std::sqrt(s);
}

int main(int, char **argv) {
  std::mt19937_64 rng(1);
  std::normal_distribution<double> N;
  if (!std::strcmp(argv[1], "sizes")) {
    long wrong = 0;
    for (int e = -1060; e <= 900; e += (e >= -520 && e < -460) ? 3 : 20)
      for (int t = 0; t < 20000; ++t) {
        double a[3], b[3], m[9], v[9], l[3];
        for (double &x : a) x = (int)(rng() % 7) - 3;
        for (double &x : b) x = (int)(rng() % 5) - 2;
        const double q = std::sqrt(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]), c = 1.0 + (rng() % 1000) / 1000.0;
        if (q == 0.0) continue;
        for (int i = 0; i < 3; ++i)
          for (int j = 0; j < 3; ++j)
            m[i + 3 * j] = std::ldexp(c * (0.5 * (a[i] * b[j] + a[j] * b[i]) / q + (t % 3 == 0) * (i == j)), e);
        strainFrame64(m, v, l);
        bool ok = true;
        for (double x : v) ok = ok && std::isfinite(x);
        for (double x : l) ok = ok && std::isfinite(x);
        double off = 0.0, orth = 0.0;
        if (ok) remainders<long double>(m, v, off, orth);
        // below 2^-480 the squares of 1e-12 of the matrix leave the doubles, in
        // symmetricEigen3's test too
        wrong += !ok || orth > 1e-14 || (e >= -480 && e < 500 && off > 1.01e-12 * norm(m));
      }
    std::printf("%ld\n", wrong);
    return 0;
  }
  for (int fam = 0; fam < 2; ++fam) {
    double rms[2] = {0, 0}, top[2] = {0, 0}, bad[2] = {0, 0};
    const int T = 40000;
    for (int t = 0; t < T; ++t) {
      double a[9], m[9];
      for (int k = 0; k < 9; ++k) a[k] = N(rng) * (fam && k % 3 ? 1e-3 : 1.0);
      for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) m[i + 3 * j] = 0.5 * (a[i + 3 * j] + a[j + 3 * i]);
      for (int w = 0; w < 2; ++w) {
        double v[9], l[3], off, orth;
        if (w) strainFrame64(m, v, l);
        else symmetricEigen3(m, v, l);
        remainders<Wide>(m, v, off, orth);
        off /= norm(m);
        rms[w] += off * off / T;
        top[w] = std::max(top[w], off);
        bad[w] = std::max(bad[w], orth);
      }
    }
    std::printf("%.3e %.3e %.3e %.3e %.3e %.3e\n", std::sqrt(rms[0]), std::sqrt(rms[1]), top[0], top[1], bad[0], bad[1]);
  }
  return 0;
}
