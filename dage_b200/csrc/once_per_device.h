// once_per_device.h -- setup that must run once on every device of a process.
//
// Kernel attributes and __constant__ tables belong to the device that is
// current when they are set, so a flag per process leaves a second device
// without them (its launches above 48 KB of shared memory are refused).
#pragma once

#include <mutex>
#include <set>

namespace dage {

class OncePerDevice {
 public:
  // f() for a device that has not had a successful f() yet; returns its
  // status (0: done).  A failed f() runs again at the next call.
  template <class F>
  int run(int device, F &&f) {
    std::lock_guard<std::mutex> lock(mu_);
    if (done_.count(device)) return 0;
    const int rc = f();
    if (rc == 0) done_.insert(device);
    return rc;
  }

 private:
  std::mutex mu_;
  std::set<int> done_;
};

}  // namespace dage
