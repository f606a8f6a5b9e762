// Schwarz bound kernels of the six pair classes (compute_schwarz_ints,
// molecular2 src/integrals.cpp:472-513).
#include "jk_kernels.cuh"

namespace m2 {

void launch_schwarz(int la, int lb, const SchwarzParams& P, int npair, cudaStream_t s) {
  dim3 grid((npair + 63) / 64);
  if (la == 0 && lb == 0) k_schwarz<0, 0><<<grid, 64, 0, s>>>(P);
  if (la == 1 && lb == 0) k_schwarz<1, 0><<<grid, 64, 0, s>>>(P);
  if (la == 1 && lb == 1) k_schwarz<1, 1><<<grid, 64, 0, s>>>(P);
  if (la == 2 && lb == 0) k_schwarz<2, 0><<<grid, 64, 0, s>>>(P);
  if (la == 2 && lb == 1) k_schwarz<2, 1><<<grid, 64, 0, s>>>(P);
  if (la == 2 && lb == 2) k_schwarz<2, 2><<<grid, 64, 0, s>>>(P);
}

}  // namespace m2
