// pinned.cuh -- pinned host memory of the process's contexts.
//
// Blocks of two sizes: a context's mailbox and a piece of a field on its way to the
// host.  Allocating or freeing pinned memory takes milliseconds and waits for the
// device, so freed blocks are kept: four staging blocks while any context lives, and
// beyond that what picard_gpu_pool_keep allows (the largest value of a device, at
// most kPinnedKeepMost), which also bounds what stays after the last context is
// gone.  Any thread, any device.
#pragma once

#include <algorithm>
#include <cstddef>
#include <exception>
#include <mutex>
#include <vector>

namespace picard {

constexpr size_t kPinnedBlock[2] = {36 << 10, 4 << 20};
constexpr size_t kPinnedKeepMost = 64 << 20;
constexpr int kPinnedDevices = 64;

// Host: static void* alloc(size_t) (null: none left) and static void free(void*).
template <class Host>
class PinnedPool {
 public:
  void* get(int cls) {
    {
      std::lock_guard<std::mutex> lk(mu_);
      if (!idle_[cls].empty()) {
        void* p = idle_[cls].back();
        idle_[cls].pop_back();
        return p;
      }
    }
    return Host::alloc(kPinnedBlock[cls]);
  }
  void put(int cls, void* p) {
    if (!p) return;
    std::lock_guard<std::mutex> lk(mu_);
    try {
      idle_[cls].push_back(p);
    } catch (const std::exception&) {
      Host::free(p);
      return;
    }
    trim();
  }
  void context(int d) {
    std::lock_guard<std::mutex> lk(mu_);
    contexts_ += d;
    trim();
  }
  void set_keep(int device, size_t bytes) {
    std::lock_guard<std::mutex> lk(mu_);
    keep_[std::clamp(device, 0, kPinnedDevices - 1)] = std::min(bytes, kPinnedKeepMost);
    trim();
  }

 private:
  std::mutex mu_;
  std::vector<void*> idle_[2];
  size_t keep_[kPinnedDevices] = {};
  long long contexts_ = 0;

  void trim() {  // with mu_ held
    const size_t allowed =
        *std::max_element(keep_, keep_ + kPinnedDevices) + (contexts_ > 0 ? 4 * kPinnedBlock[1] : 0);
    for (int cls = 1; cls >= 0; --cls)
      while (!idle_[cls].empty() &&
             idle_[0].size() * kPinnedBlock[0] + idle_[1].size() * kPinnedBlock[1] > allowed) {
        Host::free(idle_[cls].back());
        idle_[cls].pop_back();
      }
  }
};

}  // namespace picard
