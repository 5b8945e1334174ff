// Work that is done once for each device of the process, such as a kernel's
// shared-memory limit: cudaFuncSetAttribute holds for the current device only.
#pragma once

#include <mutex>
#include <vector>

namespace hd {

class OncePerDevice {
 public:
  // f() if it has not yet returned for this device; if it throws, the next call
  // tries again
  template <class F> void run(int device, F &&f) {
    std::lock_guard<std::mutex> lk(mu_);
    if (done_.size() <= (size_t)device) done_.resize((size_t)device + 1, 0);
    if (done_[device]) return;
    f();
    done_[device] = 1;
  }

 private:
  std::mutex mu_;
  std::vector<char> done_;
};

}  // namespace hd
