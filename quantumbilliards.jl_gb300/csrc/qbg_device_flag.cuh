// An answer kept per device. A kernel's attributes (opt-in shared memory,
// cluster sizes beyond 8, what the occupancy query says) belong to the device
// they were set on, so a process that moves to a second one asks again there.
// Plain C++: no CUDA header.
#pragma once
#include <atomic>

namespace qbg {

class DeviceFlag {
  static constexpr int N = 64;
  std::atomic<signed char> v_[N] = {};  // 0 not asked, 1 yes, -1 no

 public:
  // f() for this device, called until it has said what to keep; concurrent first
  // callers may each call it. A device beyond the table asks every time.
  template <class F>
  bool get(int dev, F f) {
    if (dev < 0 || dev >= N) return f();
    const signed char v = v_[dev].load();
    if (v) return v > 0;
    const bool yes = f();
    v_[dev].store(yes ? 1 : -1);
    return yes;
  }
};

}  // namespace qbg
