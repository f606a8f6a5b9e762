// Kernel instantiations of the direct J/K build, bra class dd with ket ss .. ds.
// Split across translation units only so that nvcc compiles them in parallel.
#include "jk_kernels.cuh"

namespace m2 {
cudaError_t launch_jk_bra_dd_lo(int B, const JKParams& P, dim3 grid, cudaStream_t s) {
  if (B == 0) return launch_jk_class<2, 2, 0, 0>(P, grid, s);
  if (B == 1) return launch_jk_class<2, 2, 1, 0>(P, grid, s);
  if (B == 2) return launch_jk_class<2, 2, 1, 1>(P, grid, s);
  if (B == 3) return launch_jk_class<2, 2, 2, 0>(P, grid, s);
  return cudaErrorInvalidValue;
}

}  // namespace m2
