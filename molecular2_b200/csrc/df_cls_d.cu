// Three-index (P|mn) kernel instantiations for pure d fitting shells.
// Split across translation units only so that nvcc compiles them in parallel.
#include "df_kernels.cuh"

namespace m2 {

cudaError_t launch_eri3_d_pure(int pc, const Eri3Params& P, bool j, cudaStream_t s) { return launch_eri3_l<2, true>(pc, P, j, s); }

}  // namespace m2
