// Threads that take and give slots as fast as they can; counts every time a
// slot was found in two hands.
#include <atomic>
#include <thread>
#include <vector>

#include "../../koral_b200/csrc/kgpu_slots.h"

extern "C" int slots_all_distinct() {
  kgpu::Slots s;
  bool seen[kgpu::Slots::N] = {};
  for (int i = 0; i < kgpu::Slots::N; i++) {
    const int k = s.take();
    if (k < 0 || k >= kgpu::Slots::N || seen[k]) return 0;
    seen[k] = true;
  }
  if (s.take() != -1) return 0;
  s.give(17);
  return s.take() == 17 && s.take() == -1;
}

extern "C" long slots_collisions(int threads, int rounds) {
  kgpu::Slots s;
  std::atomic<int> holder[kgpu::Slots::N] = {};
  std::atomic<long> bad{0};
  std::vector<std::thread> t;
  for (int i = 0; i < threads; i++)
    t.emplace_back([&] {
      for (int r = 0; r < rounds; r++) {
        const int k = s.take();
        if (k < 0) continue;
        if (holder[k].fetch_add(1) != 0) bad++;
        holder[k].fetch_sub(1);
        s.give(k);
      }
    });
  for (auto &x : t) x.join();
  for (int k = 0; k < kgpu::Slots::N; k++)
    if (holder[k] != 0) bad++;
  for (int k = 0; k < kgpu::Slots::N; k++)
    if (s.take() < 0) bad++;   // all came back
  return bad;
}
