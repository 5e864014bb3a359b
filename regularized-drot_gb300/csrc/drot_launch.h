// drot_launch.h -- shared-memory opt-in of kernels that are launched with
// sizes that depend on the problem.
#pragma once

#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <utility>

namespace drot {

// Allows `fn` all the dynamic shared memory that a block can have on the current
// device.  The attribute belongs to the function, not to a launch: set to the
// size of each launch, it made the launches of two host threads with problems of
// different sizes fail, when one thread lowered it between the other's setting
// and launch.  Here every thread sets the same value.
inline cudaError_t allow_shared_memory(const void* fn) {
  static std::mutex mu;
  static std::map<std::pair<int, const void*>, int> limits;
  int dev = 0;
  cudaError_t rc = cudaGetDevice(&dev);
  if (rc != cudaSuccess) return rc;
  int limit = 0;
  {
    std::lock_guard<std::mutex> lk(mu);
    int& known = limits[std::make_pair(dev, fn)];
    if (known == 0) {
      int optin = 0;
      cudaFuncAttributes at;
      rc = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
      if (rc == cudaSuccess) rc = cudaFuncGetAttributes(&at, fn);
      if (rc != cudaSuccess) return rc;
      known = optin - (int)at.sharedSizeBytes;
    }
    limit = known;
  }
  return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, limit);
}

}  // namespace drot
