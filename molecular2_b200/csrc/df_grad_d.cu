// Three-index derivative kernels of the density-fitted gradient for pure d
// fitting shells.  Split across translation units only so that nvcc compiles
// them in parallel.
#include "df_grad_kernels.cuh"

namespace m2 {

cudaError_t launch_grad3_d_pure(int pc, const Grad3Params& P, cudaStream_t s) { return launch_grad3_l<2, true>(pc, P, s); }

}  // namespace m2
