// A positive number that a launcher works out once per device (a count of SMs, after what it has to set up there), not once per
// process: attributes of a kernel are a device's own, and a process may hold several.
#pragma once

#include <atomic>

#define HB_KEPT_DEVICES 64

struct HbPerDevice {
  std::atomic<int> kept[HB_KEPT_DEVICES];      // 0: not asked yet (static storage)
};

// The number kept for device `dev`, or what ask() gives: kept if positive, else asked again next time.  Two threads that come first
// together both ask.  Devices beyond the table are asked at every call.
template <typename Ask>
static inline int hb_per_device(HbPerDevice& p, int dev, Ask ask) {
  const bool in = dev >= 0 && dev < HB_KEPT_DEVICES;
  int v = in ? p.kept[dev].load(std::memory_order_acquire) : 0;
  if (v > 0) return v;
  v = ask();
  if (in && v > 0) p.kept[dev].store(v, std::memory_order_release);
  return v;
}
