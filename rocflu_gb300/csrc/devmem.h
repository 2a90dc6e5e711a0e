// Device arrays of one context: the ones it needs, and the ones that only make
// it faster and are given back when a needed one finds no memory.
//
// Host code without CUDA types (Mem takes and gives the memory):
// tests/test_devmem_cpu.py runs it on a small budget.
#pragma once
#include <algorithm>
#include <cstddef>
#include <functional>
#include <vector>

namespace rflu {

// Mem::take(bytes): memory or null; Mem::give(p) frees it.
template <typename Mem>
class DeviceArrays {
 public:
  // Called before the optional arrays are freed: the owner waits for the work
  // that reads them and forgets their addresses.
  std::function<void()> beforeDrop;

  ~DeviceArrays() {
    for (const Array &a : needed) Mem::give(a.p);
    for (const Array &a : optional) Mem::give(a.p);
  }
  void *need(std::size_t bytes) {
    void *p = takeNeeded(bytes);
    if (p) needed.push_back({p, bytes});
    return p;
  }
  // Memory that the caller frees itself.
  void *takeNeeded(std::size_t bytes) {
    void *p = Mem::take(bytes);
    if (!p && dropOptional()) p = Mem::take(bytes);
    return p;
  }
  void *want(std::size_t bytes) {
    void *p = Mem::take(bytes);
    if (p) optional.push_back({p, bytes});
    return p;
  }
  // Frees one optional array.
  void release(void *p) {
    for (auto a = optional.begin(); a != optional.end(); ++a)
      if (a->p == p) {
        Mem::give(p);
        optional.erase(a);
        return;
      }
  }
  bool dropOptional() {
    if (optional.empty()) return false;
    if (beforeDrop) beforeDrop();
    for (const Array &a : optional) Mem::give(a.p);
    optional.clear();
    return true;
  }
  std::size_t bytes() const {
    std::size_t s = 0;
    for (const Array &a : needed) s += a.bytes;
    for (const Array &a : optional) s += a.bytes;
    return s;
  }

 private:
  struct Array {
    void *p;
    std::size_t bytes;
  };
  std::vector<Array> needed, optional;
};

}  // namespace rflu
