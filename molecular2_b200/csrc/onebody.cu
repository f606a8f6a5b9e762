// Instantiations of the one-body integral and gradient kernels.
#include "onebody.cuh"

namespace m2 {

template <int LA, int LB>
static void launch_onebody_class(const OneBodyParams& P, cudaStream_t s) {
  const size_t sm = sizeof(OneBodyShared<LA, LB>);
  cudaFuncSetAttribute(k_onebody<LA, LB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  k_onebody<LA, LB><<<P.ent.nent, OB_THREADS, sm, s>>>(P);
}

void launch_onebody(int pc, const OneBodyParams& P, cudaStream_t s) {
  if (pc == 0) launch_onebody_class<0, 0>(P, s);
  if (pc == 1) launch_onebody_class<1, 0>(P, s);
  if (pc == 2) launch_onebody_class<1, 1>(P, s);
  if (pc == 3) launch_onebody_class<2, 0>(P, s);
  if (pc == 4) launch_onebody_class<2, 1>(P, s);
  if (pc == 5) launch_onebody_class<2, 2>(P, s);
}

template <int LA, int LB>
static void launch_grad1e_class(const Grad1eParams& P, cudaStream_t s) {
  const size_t sm = sizeof(Grad1eShared<LA, LB>) + 16 + (P.natom <= G1_ATOMS ? 24 * (size_t)P.natom : 0);
  cudaFuncSetAttribute(k_grad1e<LA, LB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  // a few blocks per SM walk over the entries, so that the per-atom sums leave
  // a block once
  const int blocks = P.ent.nent < 8 * 148 ? P.ent.nent : 8 * 148;
  k_grad1e<LA, LB><<<blocks, OB_THREADS, sm, s>>>(P);
}

void launch_grad1e(int pc, const Grad1eParams& P, cudaStream_t s) {
  if (pc == 0) launch_grad1e_class<0, 0>(P, s);
  if (pc == 1) launch_grad1e_class<1, 0>(P, s);
  if (pc == 2) launch_grad1e_class<1, 1>(P, s);
  if (pc == 3) launch_grad1e_class<2, 0>(P, s);
  if (pc == 4) launch_grad1e_class<2, 1>(P, s);
  if (pc == 5) launch_grad1e_class<2, 2>(P, s);
}

}  // namespace m2
