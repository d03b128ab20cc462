// Setting a kernel's attributes once per device, from any number of threads.
#pragma once
#include <atomic>
#include <cuda_runtime.h>

namespace pie {

// Function attributes (the dynamic shared-memory opt-in) are per device.  set() runs until it has succeeded once on the current one.
// A device counts as served only behind that: a thread whose first call comes while another's set() is under way sets them as
// well (which is harmless) and does not launch without them.
template <class Set>
inline cudaError_t once_per_device(std::atomic<unsigned long long>& served, Set set) {
  int dev = 0;
  cudaGetDevice(&dev);
  const unsigned long long bit = 1ull << (dev & 63);
  if (served.load(std::memory_order_acquire) & bit) return cudaSuccess;
  const cudaError_t e = set();
  if (e == cudaSuccess) served.fetch_or(bit, std::memory_order_release);
  return e;
}

}  // namespace pie
