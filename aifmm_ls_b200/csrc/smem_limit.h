// smem_limit.h -- a kernel's opt-in to more than 48 KB of dynamic shared memory.
//
// The limit belongs to a kernel on a device and holds for every thread of the process,
// so it is raised once per device, to one value for all launches: a call that set what
// its own launch needs could lower it between another thread's call and launch.
#pragma once
#include <atomic>

class SmemLimit {
 public:
  // raise(): 0 once the current device (`device`) has the limit, else a CUDA error; it is
  // called until it has succeeded once for that device.
  template <typename Raise>
  int once(int device, Raise raise) {
    const bool kept = device >= 0 && device < kDevices;
    if (kept && done_[device].load(std::memory_order_acquire)) return 0;
    const int e = raise();
    if (e == 0 && kept) done_[device].store(true, std::memory_order_release);
    return e;
  }

 private:
  static constexpr int kDevices = 64;
  std::atomic<bool> done_[kDevices] = {};
};

#ifdef __CUDACC__
namespace {
// opt a kernel into the large dynamic shared memory on the current device
template <typename K>
int smem_limit(K kernel, SmemLimit& limit) {
  int device = 0;
  const cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return (int)e;
  return limit.once(device, [&] {
    return (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
  });
}
}  // namespace
#endif
