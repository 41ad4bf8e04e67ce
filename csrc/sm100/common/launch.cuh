// Host helpers of the launchers.
#pragma once

#include <cuda_runtime.h>

#include "per_device.h"

namespace ka {

// Opt `kernel` in to `bytes` of dynamic shared memory on the current device, once per device.
// `once` belongs to this kernel alone.
template <typename K>
bool smem_opt_in(PerDevice& once, K* kernel, int bytes) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  return once.get(dev, [&] {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess ? 1 : -1;
  }) > 0;
}

}  // namespace ka
