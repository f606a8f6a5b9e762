// Kernel instantiations of the RHF gradient, bra class dp.
// Split across translation units only so that nvcc compiles them in parallel.
#include "grad_kernels.cuh"

namespace m2 {
void launch_grad2e_bra_dp(int B, const Grad2eParams& P, dim3 grid, cudaStream_t s) {
  if (B == 0) launch_grad2e_class<2, 1, 0, 0>(P, grid, s);
  if (B == 1) launch_grad2e_class<2, 1, 1, 0>(P, grid, s);
  if (B == 2) launch_grad2e_class<2, 1, 1, 1>(P, grid, s);
  if (B == 3) launch_grad2e_class<2, 1, 2, 0>(P, grid, s);
  if (B == 4) launch_grad2e_class<2, 1, 2, 1>(P, grid, s);
}

}  // namespace m2
