// Two-index (metric) derivatives of the density-fitted gradient for every
// ordered pair of fitting groups (s, p, pure d, Cartesian d, pure f, Cartesian f).
#include "df_grad_kernels.cuh"

namespace m2 {

template <int LP, bool PP, int LQ, bool PQ>
static cudaError_t go(const Grad2Params& P, cudaStream_t s) {
  const int chunks = (P.Q.count + G2_THREADS - 1) / G2_THREADS;
  k_grad2<LP, PP, LQ, PQ><<<dim3(P.P.count, chunks), G2_THREADS, 0, s>>>(P);
  return cudaGetLastError();
}
template <int LP, bool PP>
static cudaError_t go_q(int gQ, const Grad2Params& P, cudaStream_t s) {
  if (gQ == 0) return go<LP, PP, 0, true>(P, s);
  if (gQ == 1) return go<LP, PP, 1, true>(P, s);
  if (gQ == 2) return go<LP, PP, 2, true>(P, s);
  if (gQ == 3) return go<LP, PP, 2, false>(P, s);
  if (gQ == 4) return go<LP, PP, 3, true>(P, s);
  if (gQ == 5) return go<LP, PP, 3, false>(P, s);
  return cudaErrorInvalidValue;
}

cudaError_t launch_grad2(int gP, int gQ, const Grad2Params& P, cudaStream_t s) {
  if (gP == 0) return go_q<0, true>(gQ, P, s);
  if (gP == 1) return go_q<1, true>(gQ, P, s);
  if (gP == 2) return go_q<2, true>(gQ, P, s);
  if (gP == 3) return go_q<2, false>(gQ, P, s);
  if (gP == 4) return go_q<3, true>(gQ, P, s);
  if (gP == 5) return go_q<3, false>(gQ, P, s);
  return cudaErrorInvalidValue;
}

}  // namespace m2
