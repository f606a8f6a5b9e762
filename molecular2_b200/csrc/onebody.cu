// Instantiations of the one-body integral and gradient kernels.
#include "onebody.cuh"

namespace m2 {

template <int LA, int LB>
static cudaError_t launch_onebody_class(const OneBodyParams& P, cudaStream_t s) {
  const size_t sm = sizeof(OneBodyShared<LA, LB>);
  return launch_smem(k_onebody<LA, LB>, P.pairs.npair, OB_THREADS, sm, sm, s, P);
}

cudaError_t launch_onebody(int pc, const OneBodyParams& P, cudaStream_t s) {
  if (pc == 0) return launch_onebody_class<0, 0>(P, s);
  if (pc == 1) return launch_onebody_class<1, 0>(P, s);
  if (pc == 2) return launch_onebody_class<1, 1>(P, s);
  if (pc == 3) return launch_onebody_class<2, 0>(P, s);
  if (pc == 4) return launch_onebody_class<2, 1>(P, s);
  if (pc == 5) return launch_onebody_class<2, 2>(P, s);
  return cudaErrorInvalidValue;
}

template <int LA, int LB>
static cudaError_t launch_grad1e_class(const Grad1eParams& P, cudaStream_t s) {
  constexpr size_t base = sizeof(Grad1eShared<LA, LB>) + 16, most = base + 24 * G1_ATOMS;
  static_assert(most <= SMEM_BLOCK_MAX, "shared memory of G1_ATOMS atoms");
  const size_t sm = base + (P.natom <= G1_ATOMS ? 24 * (size_t)P.natom : 0);
  // a few blocks per SM walk over the entries, so that the per-atom sums leave
  // a block once
  const int blocks = P.ent.nent < 8 * P.nsm ? P.ent.nent : 8 * P.nsm;
  return launch_smem(k_grad1e<LA, LB>, blocks, G1_THREADS, sm, most, s, P);
}

cudaError_t launch_grad1e(int pc, const Grad1eParams& P, cudaStream_t s) {
  if (pc == 0) return launch_grad1e_class<0, 0>(P, s);
  if (pc == 1) return launch_grad1e_class<1, 0>(P, s);
  if (pc == 2) return launch_grad1e_class<1, 1>(P, s);
  if (pc == 3) return launch_grad1e_class<2, 0>(P, s);
  if (pc == 4) return launch_grad1e_class<2, 1>(P, s);
  if (pc == 5) return launch_grad1e_class<2, 2>(P, s);
  return cudaErrorInvalidValue;
}

}  // namespace m2
