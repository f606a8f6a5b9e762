// Kernel launches whose status is kept.
//
// The status is taken right after each launch: the next successful
// cudaFuncSetAttribute clears the error of a failed launch before it (seen on
// CUDA 12.9), so that one query after a row of launches reports nothing and a
// class would be missing from the sum.
#pragma once
#include <cuda_runtime.h>

namespace m2 {

constexpr size_t SMEM_BLOCK_MAX = 227 * 1024;

// Launch with `smem` bytes of dynamic shared memory, of the `most` that any launch
// of this kernel asks for.  The limit belongs to the function in the whole process:
// one that followed the call would be lowered by another thread between its setting
// and the launch.
template <class... A, class... B>
inline cudaError_t launch_smem(void (*kernel)(A...), dim3 grid, int threads, size_t smem, size_t most, cudaStream_t s,
                               const B&... args) {
  const cudaError_t st = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
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
