// per_device.h — an answer that is asked of each device once.
#pragma once
#include <mutex>

namespace axc {

// get(dev, make): make() on the first call for device dev (the current one), its
// answer from then on; safe with several threads.  A process may go from one
// device to another (gpu_set_device), and a kernel's attributes are set on the
// current device only.
template <typename T>
class PerDevice {
 public:
  static constexpr int kDevices = 64;

  template <typename Make>
  T get(int dev, Make make) {
    if (dev < 0 || dev >= kDevices) return make();
    std::call_once(once_[dev], [&] { value_[dev] = make(); });
    return value_[dev];
  }

 private:
  std::once_flag once_[kDevices];
  T value_[kDevices] = {};
};

}  // namespace axc
