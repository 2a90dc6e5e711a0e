"""Threads that read a value through one slot (rocflu_gb300/csrc/shared_slot.h):
each gets what its own copy brought, never a mixture of two."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rocflu_gb300", "csrc")

HARNESS = r"""
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#include "shared_slot.h"
struct Pair { volatile long a, b; Pair &operator=(const Pair &p) { a = p.a; std::this_thread::yield(); b = p.b; return *this; } };
int main() {
  Pair storage{0, 0};
  rflu::SharedSlot<Pair> s;
  s.slot = &storage;
  std::atomic<long> torn{0}, errors{0};
  std::vector<std::thread> team;
  for (int t = 0; t < 4; ++t)
    team.emplace_back([&, t] {
      for (long k = 0; k < 2000; ++k) {
        Pair out{-1, -1};
        const long v = 10000 * t + k;
        const int rc = s.read(&out, [&](Pair *p) {
          if (k % 50 == 49) return 7;  // a failed copy: no value
          p->a = v;
          std::this_thread::yield();
          p->b = v;
          return 0;
        });
        if (rc) errors += (rc == 7 && out.a == -1);
        else if (out.a != v || out.b != v) ++torn;
      }
    });
  for (auto &t : team) t.join();
  std::printf("%ld %ld\n", torn.load(), errors.load());
}
"""


def test_reads_are_whole(tmp_path):
    src = tmp_path / "slot.cpp"
    src.write_text(HARNESS)
    exe = tmp_path / "slot"
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60).stdout.split() == ["0", "160"]
