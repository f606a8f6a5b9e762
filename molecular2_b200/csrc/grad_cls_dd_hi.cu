// Kernel instantiations of the RHF gradient, bra class dd with ket dp, dd.
// Split across translation units only so that nvcc compiles them in parallel.
#include "grad_kernels.cuh"

namespace m2 {
void launch_grad2e_bra_dd_hi(int B, const Grad2eParams& P, dim3 grid, cudaStream_t s) {
  if (B == 4) launch_grad2e_class<2, 2, 2, 1>(P, grid, s);
  if (B == 5) launch_grad2e_class<2, 2, 2, 2>(P, grid, s);
}

}  // namespace m2
