// Set-up that the CUDA runtime keeps per device (a kernel's shared-memory limit), done once on each.
#pragma once
#include <mutex>

namespace cphf {

class PerDevice {
 public:
  // true once `set` has succeeded for the device (one thread at a time; a failure is tried again)
  template <class F>
  bool once(int device, F&& set) {
    if (device < 0 || device >= kDevices) return set();
    std::lock_guard<std::mutex> lock(mu_);
    if (!done_[device]) done_[device] = set();
    return done_[device];
  }

 private:
  static constexpr int kDevices = 64;
  std::mutex mu_;
  bool done_[kDevices] = {};
};

}  // namespace cphf
