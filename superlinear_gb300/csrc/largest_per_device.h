// A limit that is raised per device and never lowered.
#pragma once
#include <cstddef>
#include <mutex>
#include <vector>

namespace sus2g {

// The largest size that a setting has been given on each device, shared by host threads.
class LargestPerDevice {
 public:
  // act(size) when the device's setting is smaller yet; returns act's result (zero: done) or zero.  A
  // failure is not remembered.  When this returns zero the setting is at least `size` and stays so.
  template <typename Act>
  int raise(int device, std::size_t size, Act&& act) {
    std::lock_guard<std::mutex> lock(mutex_);
    if (static_cast<std::size_t>(device) >= largest_.size()) largest_.resize(static_cast<std::size_t>(device) + 1, 0);
    if (size <= largest_[device]) return 0;
    const int result = act(size);
    if (result == 0) largest_[device] = size;
    return result;
  }

 private:
  std::mutex mutex_;
  std::vector<std::size_t> largest_;
};

}  // namespace sus2g
