// The library's scratch pools, one per device (host code; Api holds the
// runtime's calls, so that the bookkeeping can be tested without a GPU).
#pragma once

#include <mutex>

namespace piv {

template <class Api>
class ScratchPools {
 public:
  // The pool of the current device, created on first use; Pool() where there is none.
  typename Api::Pool get() {
    int dev = 0;
    if (!Api::device(&dev) || dev < 0 || dev >= kMax) return typename Api::Pool();
    std::lock_guard<std::mutex> lock(mu_);
    if (!pools_[dev] && !Api::create(dev, &pools_[dev])) pools_[dev] = typename Api::Pool();
    return pools_[dev];
  }

  // Gives back the idle memory of device `dev`'s pool, whichever device is current.
  void trim(int dev) {
    if (dev < 0 || dev >= kMax) return;
    std::lock_guard<std::mutex> lock(mu_);
    if (pools_[dev]) Api::trim(pools_[dev]);
  }

 private:
  static constexpr int kMax = 64;
  std::mutex mu_;
  typename Api::Pool pools_[kMax] = {};
};

}  // namespace piv
