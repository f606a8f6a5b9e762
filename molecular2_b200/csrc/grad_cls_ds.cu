// Kernel instantiations of the RHF gradient, bra class ds.
// Split across translation units only so that nvcc compiles them in parallel.
#include "grad_kernels.cuh"

namespace m2 {
cudaError_t launch_grad2e_bra_ds(int B, const Grad2eParams& P, dim3 grid, cudaStream_t s) {
  if (B == 0) return launch_grad2e_class<2, 0, 0, 0>(P, grid, s);
  if (B == 1) return launch_grad2e_class<2, 0, 1, 0>(P, grid, s);
  if (B == 2) return launch_grad2e_class<2, 0, 1, 1>(P, grid, s);
  if (B == 3) return launch_grad2e_class<2, 0, 2, 0>(P, grid, s);
  return cudaErrorInvalidValue;
}

}  // namespace m2
