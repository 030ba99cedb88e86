// What has to be told once per device: a kernel's limits belong to the device's context, a process may use several devices, and
// several threads may launch at once.
#pragma once
#include <mutex>
#include <unordered_map>
#include <vector>

namespace nrt {

class OncePerDevice {
 public:
  // `tell` (0: done) for a key and device that it has not succeeded for yet; its result, 0 where there is nothing left to do
  template <class F>
  int operator()(const void* key, int device, F&& tell) {
    std::lock_guard<std::mutex> lock(mu_);
    std::vector<bool>& told = told_[key];
    if (device < (int)told.size() && told[device]) return 0;
    const int rc = tell();
    if (rc == 0) {
      if (device >= (int)told.size()) told.resize(device + 1);
      told[device] = true;
    }
    return rc;
  }

 private:
  std::mutex mu_;
  std::unordered_map<const void*, std::vector<bool>> told_;            // by device
};

}  // namespace nrt
