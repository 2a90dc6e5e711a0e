// A cell's least-squares sums in fixed point with the scale of its own weights
// (fixCellWeights), and as the FP64 loop forms them, over the cells read from
// standard input: per line the member count, the own value, then (value, wx, wy,
// wz) per member, as hexadecimal floats.  Prints "fp64" for a cell the fixed
// point leaves to the loop, then the three sums of the loop; else "fixed", the
// three fixed-point sums and the loop's.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <vector>

#include "../rocflu_gb300/csrc/fixedsum.h"

using namespace rflu;

int main() {
  int n;
  while (std::scanf("%d", &n) == 1) {
    double own;
    if (std::scanf("%la", &own) != 1) return 1;
    std::vector<double> q(n), w[3];
    for (auto &x : w) x.resize(n);
    for (int k = 0; k < n; ++k)
      if (std::scanf("%la %la %la %la", &q[k], &w[0][k], &w[1][k], &w[2][k]) != 4) return 1;
    int eq = fixOf(own).e;
    for (double x : q) eq = std::max(eq, fixOf(x).e);
    const int top = fixCellWeights(w[0].data(), w[1].data(), w[2].data(), n);
    const bool fixed = top != kFixNoWeights && eq != kFixBad;
    std::printf(fixed ? "fixed" : "fp64");
    if (fixed)
      for (int c = 0; c < 3; ++c) {
        FixSum a{0, 0, 0};
        const FixNum o = fixOf(own);
        for (int k = 0; k < n; ++k) {
          const FixNum x = fixOf(q[k]);
          const FixHalves d = fixSplit(fixAt(x.m, x.e, eq) - fixAt(o.m, o.e, eq)), h = fixSplit(fixWeight(w[c][k], top));
          fixAdd(a, h.hi, h.lo, h.hi + h.lo, d.hi, d.lo, d.hi + d.lo);
        }
        std::printf(" %a", fixResult(a, fixScale(top) - 55 + eq - 1077));
      }
    for (int c = 0; c < 3; ++c) {
      double s = 0.0;
      for (int k = 0; k < n; ++k) s = std::fma(w[c][k], q[k] - own, s);
      std::printf(" %a", s);
    }
    std::puts("");
  }
  return 0;
}
