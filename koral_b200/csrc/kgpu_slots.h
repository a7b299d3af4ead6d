// Slots of a small fixed set that calls hold while they run.  Any number of
// host threads may take and give back; a slot is never held twice.
#pragma once
#include <atomic>

namespace kgpu {

class Slots {
 public:
  static constexpr int N = 64;
  // a free slot, or -1 when all are held
  int take() {
    unsigned long long m = held_.load(std::memory_order_relaxed);
    while (~m) {
      const int i = __builtin_ctzll(~m);
      if (held_.compare_exchange_weak(m, m | 1ull << i, std::memory_order_acquire, std::memory_order_relaxed)) return i;
    }
    return -1;
  }
  void give(int i) { held_.fetch_and(~(1ull << i), std::memory_order_release); }

 private:
  std::atomic<unsigned long long> held_{0};
};

}  // namespace kgpu
