// Device memory that an evaluation can do without.
#pragma once
#include <cstddef>

namespace sus2g {

// Grows a buffer that a kernel works without, more slowly.  A refused size is remembered and not
// asked for again until another one is wanted: the kernels of one evaluation, which share the
// buffer, then agree on whether it is there, and a full device is not asked at every launch.
class OptionalSize {
 public:
  // Whether the buffer of `have` bytes holds `want`, after grow(want) (true: grown) where it must.
  template <typename Grow>
  bool holds(std::size_t have, std::size_t want, Grow&& grow) {
    if (want <= have) return true;
    if (want == refused_) return false;
    if (grow(want)) return true;
    refused_ = want;
    return false;
  }

 private:
  std::size_t refused_ = 0;
};

}  // namespace sus2g
