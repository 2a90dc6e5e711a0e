// A slot of (pinned) host memory through which several host threads read a
// device value: one copy at a time, so that none reads another's half-written.
//
// Host code without CUDA types: tests/test_shared_slot_cpu.py runs it with
// threads.
#pragma once
#include <mutex>

namespace rflu {

template <typename T>
class SharedSlot {
 public:
  T *slot = nullptr;
  // copy(slot) fills the slot, waits for it and returns 0, or its error.
  template <typename Copy>
  int read(T *out, Copy &&copy) {
    std::lock_guard<std::mutex> one(busy);
    if (const int rc = copy(slot)) return rc;
    *out = *slot;
    return 0;
  }

 private:
  std::mutex busy;
};

}  // namespace rflu
