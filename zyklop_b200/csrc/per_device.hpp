// A value looked up once per device and kept.  The library serves several
// devices in one process, and what it asks of the runtime (occupancy, kernel
// attributes) belongs to the device that is current, so a function-local
// static would keep the first device's answer for all of them.  A lookup that
// throws is made again by the next call.
#pragma once
#include <map>
#include <mutex>

namespace zk {

template <class T>
class PerDevice {
 public:
  // the value of `dev`; `make` runs with that device current
  template <class Make>
  T get(int dev, Make make) {
    std::lock_guard<std::mutex> g(mu_);
    const auto it = of_.find(dev);
    return it != of_.end() ? it->second : of_.emplace(dev, make()).first->second;
  }

 private:
  std::mutex mu_;
  std::map<int, T> of_;
};

}  // namespace zk
