// A property of the current device that costs a driver call to find out, kept
// per device and context: what was granted to one device (a function's
// attributes among it) says nothing about the next.  Safe for any number of
// threads; two that ask at once may both ask the driver.
#pragma once

#include <map>
#include <mutex>
#include <utility>

namespace qcmg {

template <class T>
class DeviceMemo {
 public:
  // the value for (device, context): ask()'s, the first time
  template <class F>
  T get(int device, unsigned long long context, F&& ask) {
    const std::pair<int, unsigned long long> key(device, context);
    {
      std::lock_guard<std::mutex> lock(mu_);
      const auto it = known_.find(key);
      if (it != known_.end()) return it->second;
    }
    const T v = ask();
    std::lock_guard<std::mutex> lock(mu_);
    known_[key] = v;
    return v;
  }

 private:
  std::mutex mu_;
  std::map<std::pair<int, unsigned long long>, T> known_;
};

}  // namespace qcmg
