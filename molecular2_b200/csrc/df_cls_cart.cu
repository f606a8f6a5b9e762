// Three-index (P|mn) kernel instantiations for Cartesian d and f fitting shells.
// Split across translation units only so that nvcc compiles them in parallel.
#include "df_kernels.cuh"

namespace m2 {

cudaError_t launch_eri3_d_cart(int pc, const Eri3Params& P, bool j, cudaStream_t s) { return launch_eri3_l<2, false>(pc, P, j, s); }
cudaError_t launch_eri3_f_cart(int pc, const Eri3Params& P, bool j, cudaStream_t s) { return launch_eri3_l<3, false>(pc, P, j, s); }

}  // namespace m2
