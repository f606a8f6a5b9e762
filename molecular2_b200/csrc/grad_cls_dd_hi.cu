// Kernel instantiations of the RHF gradient, bra class dd with ket dp, dd.
// Split across translation units only so that nvcc compiles them in parallel.
#include "grad_kernels.cuh"

namespace m2 {
cudaError_t launch_grad2e_bra_dd_hi(int B, const Grad2eParams& P, dim3 grid, cudaStream_t s) {
  if (B == 4) return launch_grad2e_class<2, 2, 2, 1>(P, grid, s);
  if (B == 5) return launch_grad2e_class<2, 2, 2, 2>(P, grid, s);
  return cudaErrorInvalidValue;
}

}  // namespace m2
