// Host-side preparation that the driver keeps for each device by itself, as kernel attributes: done once per device, by whichever threads
// get there first (it must stand being done twice).  One that failed is tried again by the next call.
#pragma once
#include <atomic>

namespace ogb {

class OncePerDevice {
 public:
  template <typename Prepare>
  int operator()(int device, Prepare&& prepare) {
    if (device < 0 || device >= kMost) return prepare();
    if (done_[device].load(std::memory_order_acquire)) return 0;
    const int rc = prepare();
    if (rc == 0) done_[device].store(true, std::memory_order_release);
    return rc;
  }

 private:
  static constexpr int kMost = 64;
  std::atomic<bool> done_[kMost] = {};
};

}  // namespace ogb
