// Dynamic shared memory a kernel may be launched with.
//
// The limit (cudaFuncAttributeMaxDynamicSharedMemorySize) belongs to the kernel on its
// device, not to a launch, and solves of several sizes launch the same kernels from several
// threads: one that set the limit to its own need would lower it under a larger
// launch between that thread's call and its launch.  So the limit is only ever raised.
#include <map>
#include <mutex>
#include <utility>

#include "common.cuh"

namespace afq {

cudaError_t allow_smem(const void* kernel, size_t bytes) {
  static std::mutex mutex;
  static std::map<std::pair<int, const void*>, size_t> limits;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(mutex);
  size_t& limit = limits[{dev, kernel}];
  const size_t want = bytes > limit ? bytes : limit;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)want);
  if (e == cudaSuccess) limit = want;
  return e;
}

}  // namespace afq
