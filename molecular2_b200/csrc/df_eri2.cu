// Two-index (P|Q) kernels for every pair of fitting groups.
#include "df_kernels.cuh"

namespace m2 {

template <int LP, bool PP, int LQ, bool PQ>
static cudaError_t go(const Eri2Params& P, cudaStream_t s) {
  k_eri2<LP, PP, LQ, PQ><<<dim3(P.P.count, (P.Q.count + E2_THREADS - 1) / E2_THREADS), E2_THREADS, 0, s>>>(P);
  return cudaGetLastError();
}

cudaError_t launch_eri2(int gP, int gQ, const Eri2Params& P, cudaStream_t s) {
  if (gP == 0 && gQ == 0) return go<0, true, 0, true>(P, s);
  if (gP == 1 && gQ == 0) return go<1, true, 0, true>(P, s);
  if (gP == 1 && gQ == 1) return go<1, true, 1, true>(P, s);
  if (gP == 2 && gQ == 0) return go<2, true, 0, true>(P, s);
  if (gP == 2 && gQ == 1) return go<2, true, 1, true>(P, s);
  if (gP == 2 && gQ == 2) return go<2, true, 2, true>(P, s);
  if (gP == 3 && gQ == 0) return go<2, false, 0, true>(P, s);
  if (gP == 3 && gQ == 1) return go<2, false, 1, true>(P, s);
  if (gP == 3 && gQ == 2) return go<2, false, 2, true>(P, s);
  if (gP == 3 && gQ == 3) return go<2, false, 2, false>(P, s);
  if (gP == 4 && gQ == 0) return go<3, true, 0, true>(P, s);
  if (gP == 4 && gQ == 1) return go<3, true, 1, true>(P, s);
  if (gP == 4 && gQ == 2) return go<3, true, 2, true>(P, s);
  if (gP == 4 && gQ == 3) return go<3, true, 2, false>(P, s);
  if (gP == 4 && gQ == 4) return go<3, true, 3, true>(P, s);
  if (gP == 5 && gQ == 0) return go<3, false, 0, true>(P, s);
  if (gP == 5 && gQ == 1) return go<3, false, 1, true>(P, s);
  if (gP == 5 && gQ == 2) return go<3, false, 2, true>(P, s);
  if (gP == 5 && gQ == 3) return go<3, false, 2, false>(P, s);
  if (gP == 5 && gQ == 4) return go<3, false, 3, true>(P, s);
  if (gP == 5 && gQ == 5) return go<3, false, 3, false>(P, s);
  return cudaErrorInvalidValue;
}

}  // namespace m2
