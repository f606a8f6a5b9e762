// Three-index (P|mn) kernel instantiations for s and p fitting shells.
// Split across translation units only so that nvcc compiles them in parallel.
#include "df_kernels.cuh"

namespace m2 {

cudaError_t launch_eri3_s(int pc, const Eri3Params& P, bool j, cudaStream_t s) { return launch_eri3_l<0, true>(pc, P, j, s); }
cudaError_t launch_eri3_p(int pc, const Eri3Params& P, bool j, cudaStream_t s) { return launch_eri3_l<1, true>(pc, P, j, s); }

}  // namespace m2
