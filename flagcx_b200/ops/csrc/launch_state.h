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

// How many clusters of a launch shape run at once on a device: the last answer is kept, another
// shape or device asks again.  ask(&n) is the driver's call.
class ClusterCount {
 public:
  template <typename F>
  auto operator()(int device, int sharedBytes, int ctas, F &&ask, int *clusters) -> decltype(ask(clusters)) {
    const uint64_t key = (uint64_t)(uint16_t)device << 32 | (uint64_t)(uint32_t)sharedBytes << 8 | (uint64_t)(uint8_t)ctas;
    uint64_t k = last_.load(std::memory_order_relaxed);
    if (k >> 16 != key) {
      int n = 0;
      const auto e = ask(&n);
      if (e != decltype(ask(clusters))(0)) return e;
      k = key << 16 | (uint64_t)(n < 1 ? 1 : n > 0xffff ? 0xffff : n);
      last_.store(k, std::memory_order_relaxed);
    }
    *clusters = (int)(k & 0xffff);
    return decltype(ask(clusters))(0);
  }

 private:
  std::atomic<uint64_t> last_{0}; // device 16 bits, shared memory 24, CTAs per cluster 8, answer 16
};

} // namespace fcxops
