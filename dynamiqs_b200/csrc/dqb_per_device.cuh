// Set-up that holds for one device: a kernel's attributes (its shared-memory limit and
// carveout) belong to a function on a device, so a process that uses several GPUs sets
// them on each.  No CUDA header is needed (tests/test_per_device.py).
#pragma once

#include <mutex>

namespace dqb {

class PerDevice {
 public:
  static constexpr int kMax = 64;

  // Runs `setup`, which says whether it succeeded, unless it has succeeded for `device`
  // before.  Whether it has now.
  template <class F>
  bool run(int device, F setup) {
    if (device < 0 || device >= kMax) return false;
    std::lock_guard<std::mutex> lock(mu_);
    if (!done_[device]) done_[device] = setup();
    return done_[device];
  }

 private:
  std::mutex mu_;
  bool done_[kMax] = {};
};

}  // namespace dqb
