// How much dynamic shared memory a kernel has been allowed, device by device: the driver keeps that limit per device, and a
// process may use several, from several threads.
#pragma once
#include <atomic>
#include <mutex>

namespace cdeep {

class SmemLimit {
 public:
  // Sees to it that the limit on `device` is at least `bytes`. `set(bytes)` asks the driver and returns 0 where that
  // worked; it is called only for a limit that grows. Returns what `set` returned, else 0.
  template <typename Set>
  int raise(int device, int bytes, Set set) {
    if (device < 0 || device >= kDevices) return set(bytes);
    std::atomic<int>& allowed = allowed_[device];
    if (bytes <= allowed.load(std::memory_order_acquire)) return 0;
    std::lock_guard<std::mutex> lock(mu_);        // a smaller limit must not be set behind a larger one
    if (bytes <= allowed.load(std::memory_order_relaxed)) return 0;
    const int e = set(bytes);
    if (e == 0) allowed.store(bytes, std::memory_order_release);
    return e;
  }

 private:
  static constexpr int kDevices = 64;
  std::atomic<int> allowed_[kDevices] = {};
  std::mutex mu_;
};

}  // namespace cdeep
