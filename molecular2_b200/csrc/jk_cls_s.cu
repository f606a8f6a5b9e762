// Kernel instantiations of the direct J/K build, bra classes ss, ps, pp.
// Split across translation units only so that nvcc compiles them in parallel.
#include "jk_kernels.cuh"

namespace m2 {
cudaError_t launch_jk_bra_s(int A, int B, const JKParams& P, dim3 grid, cudaStream_t s) {
  if (A == 0 && B == 0) return launch_jk_class<0, 0, 0, 0>(P, grid, s);
  if (A == 1 && B == 0) return launch_jk_class<1, 0, 0, 0>(P, grid, s);
  if (A == 1 && B == 1) return launch_jk_class<1, 0, 1, 0>(P, grid, s);
  if (A == 2 && B == 0) return launch_jk_class<1, 1, 0, 0>(P, grid, s);
  if (A == 2 && B == 1) return launch_jk_class<1, 1, 1, 0>(P, grid, s);
  if (A == 2 && B == 2) return launch_jk_class<1, 1, 1, 1>(P, grid, s);
  return cudaErrorInvalidValue;
}

}  // namespace m2
