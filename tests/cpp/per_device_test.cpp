// PerDevice (rds_per_device.h) with a stand-in for cudaGetDevice: no GPU, no CUDA library. Exits 0
// when every check holds, else with the number of the first that does not.
#include "rds_per_device.h"

#include <atomic>
#include <thread>
#include <vector>

static thread_local int current     = 0;
static thread_local bool device_bad = false;

extern "C" cudaError_t cudaGetDevice(int *d)
{
  *d = current;
  return device_bad ? cudaErrorNoDevice : cudaSuccess;
}

static rds::PerDevice number;
static std::atomic<int> calls{0};

static cudaError_t ask(int *v)
{
  return number.get(v, [](int dev, int *n) {
    ++calls;
    *n = 100 + dev;
    return cudaSuccess;
  });
}

int main()
{
  int v = 0;
  // one set-up per device, and each device's own number
  for (int round = 0; round < 3; ++round)
    for (int dev : {0, 1, 7})
    {
      current = dev;
      if (ask(&v) != cudaSuccess || v != 100 + dev)
        return 1;
    }
  if (calls != 3)
    return 2;
  // a failed set-up is reported and tried again
  current      = 2;
  auto failing = [](int, int *n) {
    *n = 5;
    return cudaErrorInvalidValue;
  };
  if (number.get(&v, failing) != cudaErrorInvalidValue)
    return 3;
  if (ask(&v) != cudaSuccess || v != 102 || calls != 4)
    return 4;
  // no device
  device_bad = true;
  if (ask(&v) != cudaErrorNoDevice)
    return 5;
  device_bad = false;
  // beyond the table: asked every time
  current = 1000;
  for (int round = 0; round < 2; ++round)
    if (ask(&v) != cudaSuccess || v != 1100)
      return 6;
  if (calls != 6)
    return 7;
  // threads on devices of their own
  std::atomic<int> wrong{0};
  std::vector<std::thread> threads;
  for (int t = 0; t < 8; ++t)
    threads.emplace_back([t, &wrong] {
      current = 10 + t % 4;
      for (int i = 0; i < 1000; ++i)
      {
        int w = 0;
        if (ask(&w) != cudaSuccess || w != 110 + t % 4)
          ++wrong;
      }
    });
  for (std::thread &t : threads)
    t.join();
  return wrong == 0 ? 0 : 8;
}
