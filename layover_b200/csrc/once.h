// Something that is to happen once per device: `run(configure)` calls it for the device that is current unless it has succeeded for
// that device before, and returns whether it has. A thread that comes while another configures waits for it, so nobody goes on
// with a device that is not configured yet; a configuration that fails is tried again by the next call. Host code only.
#pragma once
#include <cuda_runtime_api.h>

#include <atomic>
#include <mutex>

struct LbPerDeviceOnce {
  static constexpr int MAX_DEVICES = 64;
  template <typename F>
  bool run(F configure) {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= MAX_DEVICES) return configure();   // again rather than not at all
    if (done[device].load(std::memory_order_acquire)) return true;
    std::lock_guard<std::mutex> lock(busy);
    if (done[device].load(std::memory_order_relaxed)) return true;
    if (!configure()) return false;
    done[device].store(true, std::memory_order_release);
    return true;
  }

 private:
  std::atomic<bool> done[MAX_DEVICES] = {};
  std::mutex busy;
};

// The common case: a kernel's limit of dynamic shared memory, raised once per device.
#define LB_ALLOW_SMEM(kernel, bytes)                                                                                        \
  [&] { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(bytes)) == cudaSuccess; }
