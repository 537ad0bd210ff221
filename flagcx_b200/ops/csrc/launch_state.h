// launch_state.h -- what the launchers of fused_elementwise.cu remember between calls, safe with
// several threads and devices.  No CUDA here: the calls to make come in as functions whose result
// is 0 on success.
#pragma once
#include <atomic>
#include <cstdint>

namespace fcxops {

// Runs `set` until it has succeeded once on a device (device 64 and above: every time).
class OncePerDevice {
 public:
  template <typename F>
  auto operator()(int device, F &&set) -> decltype(set()) {
    const uint64_t bit = device >= 0 && device < 64 ? uint64_t(1) << device : 0;
    if (done_.load(std::memory_order_acquire) & bit) return decltype(set())(0);
    const auto e = set();
    if (e == decltype(set())(0)) done_.fetch_or(bit, std::memory_order_release);
    return e;
  }

 private:
  std::atomic<uint64_t> done_{0};
};

} // namespace fcxops
