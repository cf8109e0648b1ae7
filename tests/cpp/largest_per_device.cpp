// LargestPerDevice (superlinear_gb300/csrc) against a fake of the setting it guards.
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>

#include "../../superlinear_gb300/csrc/largest_per_device.h"

#define CHECK(x)                                              \
  do {                                                        \
    if (!(x)) {                                               \
      std::printf("failed, line %d: %s\n", __LINE__, #x);     \
      return 1;                                               \
    }                                                         \
  } while (0)

int main() {
  sus2g::LargestPerDevice largest;
  std::size_t set[3] = {};
  int calls = 0, result = 0;
  auto raise = [&](int device, std::size_t size) {
    return largest.raise(device, size, [&](std::size_t n) {
      ++calls;
      if (result == 0) set[device] = n;
      return result;
    });
  };
  result = 7;
  CHECK(raise(0, 50) == 7 && calls == 1 && set[0] == 0);  // a failure is not remembered
  result = 0;
  CHECK(raise(0, 50) == 0 && raise(0, 50) == 0 && raise(0, 20) == 0 && calls == 2 && set[0] == 50);
  CHECK(raise(2, 30) == 0 && calls == 3 && set[2] == 30 && set[1] == 0);  // each device has its own
  CHECK(raise(0, 60) == 0 && raise(2, 20) == 0 && set[0] == 60 && set[2] == 30);
  // threads of different sizes: the setting covers each one's size from its return on
  for (int round = 0; round < 200; ++round) {
    sus2g::LargestPerDevice shared;
    std::atomic<std::size_t> now{0};
    std::atomic<int> refused{0};
    std::vector<std::thread> threads;
    for (std::size_t size : {40, 10, 30, 20})
      threads.emplace_back([&, size] {
        shared.raise(1, size, [&](std::size_t n) { now.store(n); return 0; });
        for (int k = 0; k < 50; ++k)
          if (now.load() < size) refused.store(1);
      });
    for (auto& t : threads) t.join();
    CHECK(!refused.load() && now.load() == 40);
  }
  std::printf("ok\n");
  return 0;
}
