// A number that belongs to a device, such as an occupancy that holds once a kernel's attributes have been set there (function
// attributes are a device's, not the process's): made at the first use on each device, from whichever thread comes first.
#ifndef THC_PER_DEVICE_H
#define THC_PER_DEVICE_H

#include <atomic>
#include <mutex>

namespace thc {

class PerDevice {
 public:
  // make() > 0, called with `device` current; when it throws, nothing is remembered.
  template <class Make> int get(int device, Make make) {
    if (device < 0 || device >= kDevices) return make();
    if (const int v = value_[device].load(std::memory_order_acquire)) return v;
    std::lock_guard<std::mutex> l(m_);
    if (const int v = value_[device].load(std::memory_order_relaxed)) return v;
    const int v = make();
    value_[device].store(v, std::memory_order_release);
    return v;
  }

 private:
  static constexpr int kDevices = 64;
  std::atomic<int> value_[kDevices] = {};
  std::mutex m_;
};

}  // namespace thc

#endif
