// tp_launch.h -- launch sizing shared by the persistent kernels.
#pragma once
#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <tuple>

// Allows `bytes` of dynamic shared memory to a kernel and returns the blocks of it that the current
// device holds at once (0: it does not fit).  The limit is one value per kernel and device, whatever thread
// launches, so it is only ever raised: a thread with a smaller scene must not lower it between another's call
// here and its launch.  The occupancy query costs more than a launch, so its answer is kept per (kernel, device,
// block size, shared memory); a handful of combinations exist.
inline cudaError_t kernel_residency(const void *kernel, int threads, int bytes, int *blocks) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  static std::mutex mu;
  static std::map<std::pair<const void *, int>, int> limits;
  static std::map<std::tuple<const void *, int, int, int>, int> known;
  std::lock_guard<std::mutex> lock(mu);
  int &limit = limits[{kernel, dev}];
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes > limit ? bytes : limit);
  if (e != cudaSuccess) return e;
  if (bytes > limit) limit = bytes;
  const auto key = std::make_tuple(kernel, dev, threads, bytes);
  const auto it = known.find(key);
  if (it != known.end()) {
    *blocks = it->second;
    return cudaSuccess;
  }
  int sms = 0, per_sm = 0;
  e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, bytes);
  if (e != cudaSuccess) return e;
  *blocks = sms * per_sm;
  if (known.size() < 1024) known[key] = *blocks;
  return cudaSuccess;
}
