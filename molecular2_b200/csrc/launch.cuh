// Kernel launches whose status is kept.
//
// The status is taken right after each launch: the next successful
// cudaFuncSetAttribute clears the error of a failed launch before it (seen on
// CUDA 12.9), so that one query after a row of launches reports nothing and a
// class would be missing from the sum.
#pragma once
#include <cuda_runtime.h>

namespace m2 {

// Launch with `smem` bytes of dynamic shared memory.
template <class... A, class... B>
inline cudaError_t launch_smem(void (*kernel)(A...), dim3 grid, int threads, size_t smem, cudaStream_t s,
                               const B&... args) {
  const cudaError_t st = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (st != cudaSuccess) return st;
  kernel<<<grid, threads, smem, s>>>(args...);
  return cudaGetLastError();
}

// First failure of a row of launches.
struct LaunchStatus {
  cudaError_t st = cudaSuccess;
  void operator()(cudaError_t s) {
    if (st == cudaSuccess) st = s;
  }
};

}  // namespace m2
