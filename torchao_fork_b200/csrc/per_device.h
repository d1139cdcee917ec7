// What a launcher sets up or asks for once: a kernel's attributes and its occupancy belong to one device, so "once" is once per device, from any
// thread.  Devices beyond the table are served every time.
#pragma once
#include <atomic>

namespace ao {

constexpr int kDeviceTable = 64;

struct OncePerDevice {
  std::atomic<bool> done[kDeviceTable] = {};
  // set(), a status of 0 for success, unless it has succeeded for this device before
  template <typename F>
  int run(int device, F&& set) {
    const bool known = device >= 0 && device < kDeviceTable;
    if (known && done[device].load(std::memory_order_acquire)) return 0;
    const int status = set();
    if (status == 0 && known) done[device].store(true, std::memory_order_release);
    return status;
  }
};

struct NumberPerDevice {
  std::atomic<int> number[kDeviceTable] = {};   // 0: not asked for yet
  // ask(), not 0, unless it has been asked for this device before
  template <typename F>
  int get(int device, F&& ask) {
    const bool known = device >= 0 && device < kDeviceTable;
    int n = known ? number[device].load(std::memory_order_relaxed) : 0;
    if (n == 0) {
      n = ask();
      if (known) number[device].store(n, std::memory_order_relaxed);
    }
    return n;
  }
};

#ifdef __CUDACC__
// The kernel may use up to `bytes` of dynamic shared memory on the current device
template <typename Kernel>
inline bool dynamic_smem(OncePerDevice& once, Kernel* kernel, int bytes) {
  int device = -1;
  cudaGetDevice(&device);
  return once.run(device, [&] { return (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); }) == 0;
}
#endif

}  // namespace ao
