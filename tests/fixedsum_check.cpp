// Sums of fixedsum.h over the terms read from standard input: per line the
// term count, the own value, then (value, weight) pairs, as hexadecimal
// floats; prints each sum, or "bad" where the fixed point does not take it.
#include <algorithm>
#include <cstdio>
#include <vector>

#include "../rocflu_gb300/csrc/fixedsum.h"

using namespace rflu;

int main() {
  int n;
  while (std::scanf("%d", &n) == 1) {
    double own;
    if (std::scanf("%la", &own) != 1) return 1;
    std::vector<double> q(n), w(n);
    for (int k = 0; k < n; ++k)
      if (std::scanf("%la %la", &q[k], &w[k]) != 2) return 1;
    int eq = fixOf(own).e, ew = 0;
    for (int k = 0; k < n; ++k) {
      eq = std::max(eq, fixOf(q[k]).e);
      ew = std::max(ew, fixOf(w[k]).e);
    }
    const int scale = fixScale(ew);
    if (n > kFixMaxTerms || eq == kFixBad || scale == kFixBadScale) {
      std::puts("bad");
      continue;
    }
    FixSum a{0, 0, 0};
    const FixNum o = fixOf(own);
    for (int k = 0; k < n; ++k) {
      const FixNum x = fixOf(q[k]);
      const FixHalves d = fixSplit(fixAt(x.m, x.e, eq) - fixAt(o.m, o.e, eq)), h = fixSplit(fixWeight(w[k], ew));
      fixAdd(a, h.hi, h.lo, h.hi + h.lo, d.hi, d.lo, d.hi + d.lo);
    }
    std::printf("%a\n", fixResult(a, scale - 55 + eq - 1077));
  }
  return 0;
}
