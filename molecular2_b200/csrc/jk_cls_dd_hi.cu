// Kernel instantiations of the direct J/K build, bra class dd with ket dp, dd.
// Split across translation units only so that nvcc compiles them in parallel.
#include "jk_kernels.cuh"

namespace m2 {
cudaError_t launch_jk_bra_dd_hi(int B, const JKParams& P, dim3 grid, cudaStream_t s) {
  if (B == 4) return launch_jk_class<2, 2, 2, 1>(P, grid, s);
  if (B == 5) return launch_jk_class<2, 2, 2, 2>(P, grid, s);
  return cudaErrorInvalidValue;
}

}  // namespace m2
