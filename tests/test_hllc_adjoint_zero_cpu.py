"""The hand-written reverse sweep of the HLLC flux (compiled for the host)
where a side's pressure is zero, hence its sound speed: the derivative of a
root at zero counts as zero, as in the dual numbers it is compared with.  Also
over ordinary states, with every entry required to be finite.  (States whose
flux has no derivative, 0/0 where neither side has pressure, are skipped.)"""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rocflu_gb300", "csrc")

HARNESS = r"""
#define __host__
#define __device__
#include <cmath>
#include <cstdio>
#include <random>
#include "physics.cuh"
#include "dual.cuh"
#include "hllc_adjoint.cuh"
using namespace rflu;
int main() {
  std::mt19937_64 rng(8);
  std::uniform_real_distribution<double> U(-1.0, 1.0);
  const double g = 1.4;
  for (int kind = 0; kind < 4; ++kind) {  // ordinary; p = 0 left, right, on both sides
    double worst = 0.0;
    long bad = 0, skipped = 0;
    for (int trial = 0; trial < 2000; ++trial) {
      double L[6] = {1.0 + 0.3 * U(rng), 1.5 * U(rng), 0.5 * U(rng), 0.5 * U(rng), 1.0 + 0.3 * U(rng), 0.0};
      double R[6] = {1.0 + 0.3 * U(rng), 1.5 * U(rng), 0.5 * U(rng), 0.5 * U(rng), 1.0 + 0.3 * U(rng), 0.0};
      if (kind & 1) L[4] = 0.0;
      if (kind & 2) R[4] = 0.0;
      L[5] = 1.0 / L[0];
      R[5] = 1.0 / R[0];
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
      double want[12];
      bool finite = true;
      for (int j = 0; j < 12; ++j) {
        want[j] = 0.0;
        for (int k = 0; k < 5; ++k) want[j] += fbar[k] * f[k].d[j];
        finite = finite && std::isfinite(want[j]);
      }
      if (!finite) { ++skipped; continue; }
      for (int j = 0; j < 12; ++j) {
        const double h = j < 6 ? Lb[j] : Rb[j - 6];
        if (!std::isfinite(h)) { ++bad; continue; }
        worst = fmax(worst, fabs(want[j] - h) / (1.0 + fabs(want[j])));
      }
    }
    printf("%ld %ld %.3e\n", bad, skipped, worst);
  }
}
"""


def test_reverse_sweep_at_zero_pressure(tmp_path):
    src = tmp_path / "hllc_zero.cpp"
    src.write_text(HARNESS)
    exe = tmp_path / "hllc_zero"
    subprocess.run(["g++", "-O1", "-std=c++17", "-w", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")
    for line in out[:4]:
        bad, skipped, worst = line.split()
        assert int(bad) == 0 and int(skipped) < 1000 and float(worst) < 1e-10, out
