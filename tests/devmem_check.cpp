// DeviceArrays on a budget of bytes read from the command line.  Standard
// input: lines "need n", "want n" or "scratch n" (bytes); prints per line
// whether the memory was had, the optional arrays then held and the times they
// were dropped; last the bytes that were never given back.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>

#include "../rocflu_gb300/csrc/devmem.h"

static std::size_t budget, used;
static std::map<void *, std::size_t> live;
struct Mem {
  static void *take(std::size_t n) {
    if (used + n > budget) return nullptr;
    void *p = std::malloc(n);
    live[p] = n;
    used += n;
    return p;
  }
  static void give(void *p) {
    used -= live.at(p);
    live.erase(p);
    std::free(p);
  }
};

int main(int, char **argv) {
  budget = std::strtoull(argv[1], nullptr, 10);
  std::vector<void *> scratch;
  {
    rflu::DeviceArrays<Mem> a;
    int held = 0, drops = 0;
    a.beforeDrop = [&] { held = 0; ++drops; };
    char what[16];
    std::size_t n;
    while (std::scanf("%15s %zu", what, &n) == 2) {
      void *p = nullptr;
      if (!std::strcmp(what, "need")) p = a.need(n);
      else if (!std::strcmp(what, "scratch")) { if ((p = a.takeNeeded(n))) scratch.push_back(p); }
      else if ((p = a.want(n))) ++held;
      std::printf("%d %d %d\n", p != nullptr, held, drops);
    }
    std::printf("%zu\n", a.bytes());
  }
  for (void *p : scratch) Mem::give(p);
  std::printf("%zu\n", used);
  return 0;
}
