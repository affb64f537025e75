// A kernel's attributes (shared memory above 48 KB, cluster sizes) belong to the device that is current when they are
// set: they are set once for each device that a process launches the kernel on.
#pragma once

#include <cuda_runtime.h>

#include <mutex>

namespace xgb {

class PerDevice {
 public:
  static constexpr int kMost = 64;
  // the current device's index
  static int current() {
    int dev = 0;
    return cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kMost ? dev : 0;
  }
  // f() on the first call with each current device (again if it threw)
  template <class F>
  void once(F&& f) {
    std::call_once(done_[current()], static_cast<F&&>(f));
  }

 private:
  std::once_flag done_[kMost];
};

}  // namespace xgb
