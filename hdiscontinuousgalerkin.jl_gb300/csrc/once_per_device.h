// What has to be done once on every device: a kernel's attributes (cudaFuncSetAttribute) belong to the current device, so
// a second device of the process needs them again.
#pragma once
#include <mutex>
#include <set>

class OncePerDevice {
 public:
  // Calls set() unless an earlier call for this device has returned; one that throws is made again.  Callers wait for it.
  template <class F> void operator()(int device, F set) {
    std::lock_guard<std::mutex> lk(mu_);
    if (done_.count(device)) return;
    set();
    done_.insert(device);
  }

 private:
  std::mutex mu_;
  std::set<int> done_;
};
