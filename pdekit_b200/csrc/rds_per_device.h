// A positive number per GPU of the process, found by a set-up call on first use: what a launch asks
// the device once (resident blocks, whether a cluster fits) or sets once per kernel and device (the
// shared-memory opt-in). cudaFuncSetAttribute and the attributes hold for one device only, so a
// value found on the first device must not serve a context on another.
#pragma once

#include <atomic>

#include <cuda_runtime_api.h>

namespace rds
{

class PerDevice
{
public:
  // The number of the current device; set_up(device, &number) finds it on the device's first call
  // and, should it fail, on the next. Threads that come first together may each run set_up.
  template <typename F>
  cudaError_t get(int *value, F &&set_up)
  {
    int dev             = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess)
      return e;
    if (dev >= kDevices)
      return set_up(dev, value);
    int v = value_[dev].load(std::memory_order_acquire);
    if (v == 0)
    {
      const cudaError_t f = set_up(dev, &v);
      if (f != cudaSuccess)
        return f;
      value_[dev].store(v, std::memory_order_release);
    }
    *value = v;
    return cudaSuccess;
  }

private:
  static constexpr int kDevices = 64;
  std::atomic<int> value_[kDevices]{};
};

} // namespace rds
