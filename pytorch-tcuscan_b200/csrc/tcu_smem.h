// tcu_smem.h -- opting kernels into more than 48 KB of dynamic shared memory.
#pragma once

#include <cuda_runtime_api.h>

#include <atomic>
#include <cstdint>
#include <initializer_list>

namespace tcu {

// Devices on which a launcher has raised its kernels' limit.  The attribute
// belongs to the current device, so one flag per process would leave every
// further device at 48 KB.  Two threads may both find a device missing and set
// the attribute twice, to the same value.
class DeviceSet {
 public:
  bool has(int dev) const { return dev >= 0 && dev < 64 && (bits_.load(std::memory_order_acquire) >> dev & 1u); }
  void add(int dev) {
    if (dev >= 0 && dev < 64) bits_.fetch_or(uint64_t(1) << dev, std::memory_order_release);
  }

 private:
  std::atomic<uint64_t> bits_{0};
};

// Raises the limit of the given kernels to `bytes` on the current device,
// unless `done` (one per launcher) holds it.
template <typename... Kernels>
inline cudaError_t allow_smem(DeviceSet& done, int bytes, Kernels... kernels) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || done.has(dev)) return e;
  for (const void* k : {reinterpret_cast<const void*>(kernels)...}) {
    e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
  }
  done.add(dev);
  return cudaSuccess;
}

}  // namespace tcu
