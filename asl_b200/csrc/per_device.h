// What a launch finds out once and keeps, per CUDA device: a kernel's limit of
// dynamic shared memory and its resident blocks belong to a device, and a
// program may run solvers on several (aslb_set_device). Host only.
#pragma once
#include <atomic>

namespace aslb {

class PerDevice {
 public:
  // The positive number kept for a device, or what find(number) gives on its
  // first use there (an error code, 0 for none; errors are not kept). Threads
  // that come first together each call find.
  template <class Find>
  auto get(int device, int& number, Find find) -> decltype(find(number)) {
    std::atomic<int>* kept = device >= 0 && device < kDevices ? &kept_[device] : nullptr;
    number = kept ? kept->load(std::memory_order_acquire) : 0;
    if (number > 0) return decltype(find(number))(0);
    const auto error = find(number);
    if (kept && !error && number > 0) kept->store(number, std::memory_order_release);
    return error;
  }

 private:
  static constexpr int kDevices = 64;
  std::atomic<int> kept_[kDevices] = {};
};

}  // namespace aslb
