// Schwarz bound kernels of the six pair classes (compute_schwarz_ints,
// molecular2 src/integrals.cpp:472-513).
#include "jk_kernels.cuh"

namespace m2 {

cudaError_t launch_schwarz(int la, int lb, const SchwarzParams& P, cudaStream_t s) {
  if (la == 0 && lb == 0) return launch_schwarz_class<0, 0>(P, s);
  if (la == 1 && lb == 0) return launch_schwarz_class<1, 0>(P, s);
  if (la == 1 && lb == 1) return launch_schwarz_class<1, 1>(P, s);
  if (la == 2 && lb == 0) return launch_schwarz_class<2, 0>(P, s);
  if (la == 2 && lb == 1) return launch_schwarz_class<2, 1>(P, s);
  if (la == 2 && lb == 2) return launch_schwarz_class<2, 2>(P, s);
  return cudaErrorInvalidValue;
}

}  // namespace m2
