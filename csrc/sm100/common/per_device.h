// Launch settings that belong to a device: a function attribute set on one GPU says nothing about
// the next one that the same process uses, and neither does an occupancy answer.
#pragma once

#include <mutex>

namespace ka {

// Set up once per device ordinal, from whichever thread comes first; a set-up that fails is tried
// again by the next call. Meant for function-local statics.
class PerDevice {
 public:
  // The value that `setup` gave for device `dev`; what is not positive is a failure and is returned as it is.
  template <typename F>
  int get(int dev, F&& setup) {
    if (dev < 0 || dev >= kMaxDevices) return -1;
    std::lock_guard<std::mutex> lock(mu_);
    if (value_[dev] > 0) return value_[dev];
    const int v = setup();
    if (v > 0) value_[dev] = v;
    return v;
  }

 private:
  static constexpr int kMaxDevices = 64;
  std::mutex mu_;
  int value_[kMaxDevices] = {};
};

}  // namespace ka
