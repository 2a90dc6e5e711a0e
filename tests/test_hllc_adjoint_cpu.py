"""The hand-written reverse sweep of the second-order HLLC flux against the
transposed Jacobian from forward-mode dual numbers on the flux code itself
(both compiled for the host): both supersonic sides, both sides of the
contact, equal states."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rocflu_gb300", "csrc")

HARNESS = r"""
#define __host__
#define __device__
#include <cstdio>
#include <random>
#include "physics.cuh"
#include "dual.cuh"
#include "hllc_adjoint.cuh"
using namespace rflu;
int main() {
  std::mt19937_64 rng(6);
  std::uniform_real_distribution<double> U(-1.0, 1.0);
  const double g = 1.4;
  double worst = 0.0;
  int seen[4] = {0, 0, 0, 0};
  for (int trial = 0; trial < 4000; ++trial) {
    double L[6] = {1.0 + 0.3 * U(rng), 0.5 * U(rng), 0.5 * U(rng), 0.5 * U(rng), 1.0 + 0.3 * U(rng), 0.0};
    double R[6] = {1.0 + 0.3 * U(rng), 0.5 * U(rng), 0.5 * U(rng), 0.5 * U(rng), 1.0 + 0.3 * U(rng), 0.0};
    if (trial % 3 == 0) { L[1] = 2.0 * U(rng); R[1] = L[1] + 0.3 * U(rng); }
    if (trial % 4 == 0) { L[1] = R[1] = 2.5; }
    if (trial % 4 == 1) { L[1] = R[1] = -2.5; }
    if (trial % 7 == 0) for (int k = 0; k < 5; ++k) R[k] = L[k];
    L[5] = 1.0 / (L[0] * (1.0 + 0.1 * U(rng)));
    R[5] = 1.0 / (R[0] * (1.0 + 0.1 * U(rng)));
    double n[3] = {1.0 + 0.3 * U(rng), U(rng), U(rng)};
    double m = sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
    for (double &x : n) x /= m;
    const double nm = 0.3 + 0.5 * (U(rng) + 1.0);
    double fbar[5], Lb[6], Rb[6];
    for (double &x : fbar) x = U(rng);
    hllc2Adjoint(g, n[0], n[1], n[2], nm, L, L[5], R, R[5], fbar, Lb, Rb);
    typedef Dual<12> D;
    D a[6], b[6], f[5];
    for (int k = 0; k < 6; ++k) { a[k] = D::seed(L[k], k); b[k] = D::seed(R[k], 6 + k); }
    D G(g);
    D el = perfEo(a[0], G, a[4], a[1], a[2], a[3]), al = sqrt_(G * a[4] / a[0]);
    D er = perfEo(b[0], G, b[4], b[1], b[2], b[3]), ar = sqrt_(G * b[4] / b[0]);
    D Hl = el + a[5] * a[4], Hr = er + b[5] * b[4];
    hllcFlux(G, D(n[0]), D(n[1]), D(n[2]), D(nm), a[0], a[1], a[2], a[3], a[4], el, al, Hl, b[0], b[1], b[2], b[3],
             b[4], er, ar, Hr, f);
    double q = L[1] * n[0] + L[2] * n[1] + L[3] * n[2];
    seen[q > 1.9 ? 0 : q < -1.9 ? 1 : q > 0 ? 2 : 3]++;
    for (int j = 0; j < 12; ++j) {
      double s = 0.0;
      for (int k = 0; k < 5; ++k) s += fbar[k] * f[k].d[j];
      double h = (j < 6) ? Lb[j] : Rb[j - 6];
      double err = fabs(s - h) / (1.0 + fabs(s));
      if (!(err <= worst)) worst = err;
    }
  }
  for (int s : seen) if (s < 100) worst = 1.0;
  printf("%.3e\n", worst);
  return 0;
}
"""


def test_hllc_reverse_sweep_matches_dual_jacobian(tmp_path):
    src = tmp_path / "hllc_adj.cpp"
    src.write_text(HARNESS)
    exe = tmp_path / "hllc_adj"
    subprocess.run(["g++", "-O1", "-std=c++17", "-w", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert float(out) < 1e-12, out
