// What has been done once per kernel and device, for any number of kernels (host code only).
#pragma once

#include <cstdint>
#include <mutex>
#include <unordered_map>

namespace dil {

class OncePerDevice {
 public:
  static constexpr int kDevices = 64;      // one bit each; nothing is remembered for a device past them
  bool done(const void* fn, int dev) {
    if (dev < 0 || dev >= kDevices) return false;
    std::lock_guard<std::mutex> lk(mu_);
    const auto it = bits_.find(fn);
    return it != bits_.end() && (it->second >> dev & 1);
  }
  void set(const void* fn, int dev) {
    if (dev < 0 || dev >= kDevices) return;
    std::lock_guard<std::mutex> lk(mu_);
    bits_[fn] |= uint64_t{1} << dev;
  }

 private:
  std::mutex mu_;
  std::unordered_map<const void*, uint64_t> bits_;
};

}  // namespace dil
