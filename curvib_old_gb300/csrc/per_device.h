// What holds for one device alone (a kernel's attributes, whether it can be launched
// with a cluster), formed once on each device of the process.
#pragma once
#include <atomic>

namespace cvb {

class PerDevice {
  static constexpr int kKept = 64;  // ordinals beyond are formed every time
  std::atomic<unsigned long long> formed_{0}, result_{0};

 public:
  // form() on device dev, or what it returned there before.  Two threads may both be
  // first: form gives the same each time.
  template <typename F>
  bool get(int dev, F form) {
    if (dev < 0 || dev >= kKept) return form();
    const unsigned long long bit = 1ULL << dev;
    if (formed_.load() & bit) return (result_.load() & bit) != 0;
    const bool r = form();
    if (r) result_.fetch_or(bit);
    formed_.fetch_or(bit);
    return r;
  }
};

}  // namespace cvb
