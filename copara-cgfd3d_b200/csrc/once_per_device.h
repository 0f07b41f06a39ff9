// once_per_device.h -- host-side set-up that belongs to a device.
#pragma once

#include <cuda_runtime.h>

#include <mutex>
#include <set>
#include <utility>

namespace cgfd {

// Work done once per (device, key): kernel attributes belong to the device that
// is current when they are set.  A failed run is tried again by the next call.
class OncePerDevice {
 public:
  template <typename F>  // cudaError_t()
  bool run(int key, F &&f) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    std::lock_guard<std::mutex> lk(m_);
    if (done_.count({dev, key})) return true;
    if (f() != cudaSuccess) return false;
    done_.insert({dev, key});
    return true;
  }

 private:
  std::mutex m_;
  std::set<std::pair<int, int>> done_;
};

// SMs of the current device
inline int sm_count() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

}  // namespace cgfd
