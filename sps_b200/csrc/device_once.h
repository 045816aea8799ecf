// Settings that a process makes once for every device that it uses.
#pragma once

#include <atomic>
#include <cstdint>

namespace spsattn {

// Runs `set` (0 = done) unless it has succeeded on `device` before; `done` holds a bit per device.  Two
// threads may both run it the first time.  Devices past the 64th run it on every call.
template <typename F>
int once_per_device(std::atomic<uint64_t>& done, int device, F&& set) {
  const bool kept = device >= 0 && device < 64;
  const uint64_t bit = kept ? uint64_t{1} << device : 0;
  if (kept && (done.load(std::memory_order_acquire) & bit)) return 0;
  const int rc = set();
  if (rc == 0 && kept) done.fetch_or(bit, std::memory_order_release);
  return rc;
}

}  // namespace spsattn
