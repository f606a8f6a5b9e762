// Kernel instantiations of the RHF gradient, bra classes ss, ps, pp.
// Split across translation units only so that nvcc compiles them in parallel.
#include "grad_kernels.cuh"

namespace m2 {
cudaError_t launch_grad2e_bra_s(int A, int B, const Grad2eParams& P, dim3 grid, cudaStream_t s) {
  if (A == 0 && B == 0) return launch_grad2e_class<0, 0, 0, 0>(P, grid, s);
  if (A == 1 && B == 0) return launch_grad2e_class<1, 0, 0, 0>(P, grid, s);
  if (A == 1 && B == 1) return launch_grad2e_class<1, 0, 1, 0>(P, grid, s);
  if (A == 2 && B == 0) return launch_grad2e_class<1, 1, 0, 0>(P, grid, s);
  if (A == 2 && B == 1) return launch_grad2e_class<1, 1, 1, 0>(P, grid, s);
  if (A == 2 && B == 2) return launch_grad2e_class<1, 1, 1, 1>(P, grid, s);
  return cudaErrorInvalidValue;
}

}  // namespace m2
