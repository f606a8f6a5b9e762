// Three-index derivative kernels of the density-fitted gradient for s and p
// fitting shells.  Split across translation units only so that nvcc compiles
// them in parallel.
#include "df_grad_kernels.cuh"

namespace m2 {

cudaError_t launch_grad3_s(int pc, const Grad3Params& P, cudaStream_t s) { return launch_grad3_l<0, true>(pc, P, s); }
cudaError_t launch_grad3_p(int pc, const Grad3Params& P, cudaStream_t s) { return launch_grad3_l<1, true>(pc, P, s); }

}  // namespace m2
