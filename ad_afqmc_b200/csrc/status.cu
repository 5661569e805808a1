// Device-side failure status of one workspace.
//
// The tensor-core kernels never spin without bound: every mbarrier wait polls
// a limited number of times (umma.cuh), and a wait that runs out sets an int
// flag in the caller's workspace and ends its CTA: nothing more is issued, what is in flight
// is waited for (bounded), TMEM is freed.  The launching call has returned
// AFQ_OK long before, since every entry point is asynchronous, so the walkers
// or energies of that call are garbage and the flag is the only record.
// afq_check_status reads and clears it (once per block is enough: the flag
// stays set until read); afq_status_flag gives its device address to code that
// copies it out inside a CUDA graph.  afq_test_wait_timeout makes a producer's
// wait run out on purpose, on a stage that nobody reads and with no copy or MMA in
// flight, so tests can exercise this path without a fault.
#include <cuda_runtime.h>

#include "afqmc_b200.h"
#include "layout.cuh"
#include "umma.cuh"

namespace afq {
namespace {

int flag_ptr(const afq_dims* d, void* work, size_t work_bytes, int** out) {
  Layout L;
  const int rc = make_layout(d, L);
  if (rc != AFQ_OK) return rc;
  if (!work) return AFQ_ERR_NULL;
  if ((reinterpret_cast<uintptr_t>(work) & 15u) != 0) return AFQ_ERR_ALIGN;
  if (work_bytes < (size_t)L.work * sizeof(double)) return AFQ_ERR_WORKSPACE;
  *out = reinterpret_cast<int*>(static_cast<double*>(work) + L.w_misc);
  return AFQ_OK;
}

// The producer side of a ring of two stages that nobody reads, with the GEMM
// pipelines' own wait and fill loop; a plain arrival stands for a copy that has landed.
// The third stage's wait runs out, which sets the flag.  Anything else than two
// stages issued, the second fill refused at its first wait and a drain of what was
// issued is reported as flag value 2.
__global__ void wait_timeout_kernel(int* flag, uint32_t polls) {
  __shared__ __align__(8) uint64_t full[2], empty[2];
  __shared__ int abort_s, issued;
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    abort_s = issued = 0;
    fence_barrier_init();
  }
  __syncwarp();
  Ring ring{full, empty, 2};
  auto issue = [&](int stage, int) {
    ++issued;
    mbar_arrive(&full[stage]);
  };
  const bool first = ring_fill(ring, 5, &abort_s, flag, issue, polls);
  const bool second = ring_fill(ring, 5, &abort_s, flag, issue, polls);
  ring_drain(ring, full);
  if (threadIdx.x == 0 && (first || second || issued != 2 || abort_s != 1)) atomicExch(flag, 2);
}

}  // namespace
}  // namespace afq

using namespace afq;

extern "C" {

int afq_check_status(const afq_dims* d, void* work, size_t work_bytes, void* stream) {
  int* flag = nullptr;
  int rc = flag_ptr(d, work, work_bytes, &flag);
  if (rc != AFQ_OK) return rc;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  int host = 0;
  if (cudaMemcpyAsync(&host, flag, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess)
    return AFQ_ERR_CUDA;
  if (cudaStreamSynchronize(st) != cudaSuccess) return AFQ_ERR_CUDA;
  if (host == 0) return AFQ_OK;
  if (cudaMemsetAsync(flag, 0, sizeof(int), st) != cudaSuccess) return AFQ_ERR_CUDA;
  if (cudaStreamSynchronize(st) != cudaSuccess) return AFQ_ERR_CUDA;
  return host == 2 ? AFQ_ERR_BOUNDS : AFQ_ERR_TIMEOUT;
}

int afq_status_flag(const afq_dims* d, void* work, size_t work_bytes, int32_t** flag) {
  if (!flag) return AFQ_ERR_NULL;
  int* p = nullptr;
  const int rc = flag_ptr(d, work, work_bytes, &p);
  if (rc != AFQ_OK) return rc;
  *flag = p;
  return AFQ_OK;
}

int afq_test_wait_timeout(const afq_dims* d, void* work, size_t work_bytes, uint32_t polls,
                          void* stream) {
  int* flag = nullptr;
  int rc = flag_ptr(d, work, work_bytes, &flag);
  if (rc != AFQ_OK) return rc;
  if (polls < 1 || polls > 4096) return AFQ_ERR_ARG;
  wait_timeout_kernel<<<1, 32, 0, reinterpret_cast<cudaStream_t>(stream)>>>(flag, polls);
  return cudaGetLastError() == cudaSuccess ? AFQ_OK : AFQ_ERR_CUDA;
}

}  // extern "C"
