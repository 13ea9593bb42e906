// What a launcher sets or asks once per device.
#pragma once
#include <cuda_runtime.h>

#include "per_device.h"

namespace ssb {

// A kernel's leave to use more than 48 KB of dynamic shared memory; `done` belongs to the kernel.
template <class Kernel>
int allow_smem_once(OncePerDevice<>& done, Kernel kernel, int bytes) {
  int dev = 0, unused = 0;
  if (const cudaError_t e = cudaGetDevice(&dev)) return static_cast<int>(e);
  return done.get(dev, &unused, [&](int* value) {
    *value = 1;
    return static_cast<int>(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  });
}

}  // namespace ssb
