// "Done on this device": a kernel's attributes (shared memory beyond 48 KB, clusters of
// more than 8 CTAs) belong to one device's context, so a flag for the process would
// leave a second device without them.
#pragma once

#include <atomic>
#include <cstdint>

namespace tnad {

class PerDevice {
 public:
  // device numbers from 64 on are never marked: what is done once is done each time
  bool has(int dev) const { return in(dev) && (done_.load(std::memory_order_acquire) >> dev & 1u) != 0; }
  void mark(int dev) {
    if (in(dev)) done_.fetch_or(std::uint64_t(1) << dev, std::memory_order_release);
  }

 private:
  static bool in(int dev) { return dev >= 0 && dev < 64; }
  std::atomic<std::uint64_t> done_{0};
};

}  // namespace tnad
