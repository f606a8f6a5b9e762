// Device side of the density-fitted RHF gradient: derivative three-index
// (mn|P)^x and two-index (P|Q)^x integrals contracted at once with their
// weights, recomputed per shell pair / aux shell (nothing derivative is
// stored).  With c = V^-1 gamma, gamma_P = sum_mn (P|mn) D_mn, and
// d^P_ij = sum_Q (V^-1)_PQ (Q|ij) over the occupied orbitals, the two-electron
// energy of compute_2body_fock_df (molecular2 src/fockbuild.cpp:585-660),
//   E2 = 1/2 gamma^T V^-1 gamma - sum_ij sum_PQ (P|ij) (V^-1)_PQ (Q|ij),
// has the nuclear derivative
//   dE2 = sum_{P,mn} (mn|P)^x W3_{mn,P} + sum_{PQ} (P|Q)^x W2_{PQ},
//   W3_{mn,P} = c_P D_mn - 2 sum_ij C_mi C_nj d^P_ij,
//   W2_{PQ}   = -1/2 c_P c_Q + sum_ij d^P_ij d^Q_ij.
// The orbital centres' derivatives come from one Hermite table per primitive
// quartet as in grad_kernels.cuh; with the fitting function as the bra, d/dP is
// its shift and d/dn = -d/dP - d/dm.  For (P|Q) d/dQ = -d/dP.
#pragma once
#include "df_kernels.cuh"
#include "grad_kernels.cuh"

namespace m2 {

struct Grad3Params {
  int nsm;
  AuxView aux;            // fitting shells of one group
  const int* aux_atom;
  const int* atom;        // orbital shell -> atom
  EntryView ent;          // orbital pairs of one class
  PairView pairs;
  const double *ox, *oy, *oz;
  const int* coff;        // Cartesian function offsets of the orbital shells
  const double* sph;
  const double* boysp;
  int nc;
  const double* W3;       // [P - w3_f0][y][x] over Cartesian orbital functions: W3[((P - w3_f0) * nc + y) * nc + x]
  int w3_f0;              // first fitting function held in W3
  int natom;
  double* grad;           // 3 * natom
};

template <int LP>
struct Grad3Shared {
  double boys[boysp_size(LP + 5)];  // orbital pairs up to dd
  double sphP[(2 * LP + 1) * ncart(LP)];
  double red[GRAD_THREADS / 32][3];
};

// Block = (fitting shell, kets by blocks, ket component).  The weights of a ket
// entry are folded into the fitting shell's Hermite expansion G, of which a
// pure, s or p shell has only the top degree.  (H2O)8/cc-pVDZ: the whole
// gradient call 86 -> 8.8 ms, 3.7 without its allocations (44 ms of it four shifted evaluations a pair with
// their integral blocks in local memory).
template <int LP, bool PURE, int LC, int LD>
__global__ void __launch_bounds__(GRAD_THREADS, 2) k_grad3(const Grad3Params P) {
  constexpr int NP = ncart(LP), NF = e3_nfun(LP, PURE), ND = ncart(LD), LCD = LC + LD, L = LP + LCD;
  constexpr bool TOP = LP <= 1 || PURE;
  constexpr int NG = TOP ? NP : nherm(LP);
  static_assert(LCD <= 4, "the Boys table covers the ket");
  extern __shared__ __align__(16) unsigned char g3_sm[];
  Grad3Shared<LP>& S = *reinterpret_cast<Grad3Shared<LP>*>(g3_sm);
  double* s_g = reinterpret_cast<double*>(g3_sm + ((sizeof(Grad3Shared<LP>) + 15) & ~(size_t)15));
  const int tid = threadIdx.x, lane = tid & 31;
  const bool local = P.natom <= GRAD_ATOMS;
  double* g_atom = local ? s_g : P.grad;
  load_boys<L + 1>(S.boys, P.boysp);
  if constexpr (PURE && LP > 1)
    for (int i = tid; i < NF * NP; i += GRAD_THREADS) S.sphP[i] = P.sph[sph_off(LP) + i];
  if (local)
    for (int i = tid; i < 3 * P.natom; i += GRAD_THREADS) s_g[i] = 0.0;
  __syncthreads();
  const int sh = P.aux.shells[blockIdx.x];
  const int j0 = P.aux.prim_off[sh], nj = P.aux.nprim[sh];
  const double* W3 = P.W3 + (size_t)(P.aux.foff[sh] - P.w3_f0) * P.nc * P.nc;
  const int ic = blockIdx.z / ND, id = blockIdx.z % ND;
  int ce[3], de[3];
  ce[0] = LC > 0 ? c_herm.t[nherm(LC - 1) + ic] : 0;
  ce[1] = LC > 0 ? c_herm.u[nherm(LC - 1) + ic] : 0;
  ce[2] = LC > 0 ? c_herm.v[nherm(LC - 1) + ic] : 0;
  de[0] = LD > 0 ? c_herm.t[nherm(LD - 1) + id] : 0;
  de[1] = LD > 0 ? c_herm.u[nherm(LD - 1) + id] : 0;
  de[2] = LD > 0 ? c_herm.v[nherm(LD - 1) + id] : 0;
  const int tx = ce[0] + de[0], ty = ce[1] + de[1], tz = ce[2] + de[2];
  double sP[3] = {0, 0, 0};
  for (int e0 = blockIdx.y * GRAD_THREADS; e0 < P.ent.nent; e0 += gridDim.y * GRAD_THREADS) {
    const bool active = e0 + tid < P.ent.nent;
    const int e = active ? e0 + tid : P.ent.nent - 1;
    const int kl = P.ent.pair[e], c = P.pairs.sa[kl], d = P.pairs.sb[kl];
    const double* kp = entry_prims(P.ent, e);
    const int nk = P.ent.np[e];
    const int nkm = __reduce_max_sync(0xffffffffu, nk);
    // the sum over ordered (m, n) counts an off-diagonal canonical pair twice
    const double deg = !active ? 0.0 : (c == d ? 1.0 : 2.0);
    const double Cc[3] = {P.ox[c], P.oy[c], P.oz[c]}, Dd[3] = {P.ox[d], P.oy[d], P.oz[d]};
    double w[NP];  // weights of the Cartesian fitting components
    {
      const double* q = W3 + (size_t)(P.coff[d] + id) * P.nc + P.coff[c] + ic;
      double f[NF];
#pragma unroll
      for (int i = 0; i < NF; ++i) f[i] = deg * __ldg(q + (size_t)i * P.nc * P.nc);
      if constexpr (PURE && LP > 1) {
#pragma unroll
        for (int i = 0; i < NP; ++i) {
          w[i] = 0.0;
#pragma unroll
          for (int m = 0; m < NF; ++m) w[i] += S.sphP[m * NP + i] * f[m];
        }
      } else {
#pragma unroll
        for (int i = 0; i < NP; ++i) w[i] = f[i];
      }
    }
    double gP[3] = {0, 0, 0}, gC[3] = {0, 0, 0};
    for (int j = j0; j < j0 + nj; ++j) {
      const double p = __ldg(P.aux.p + j), Px = __ldg(P.aux.x + j), Py = __ldg(P.aux.y + j), Pz = __ldg(P.aux.z + j);
      const double Kb = __ldg(P.aux.Kp + j), h1 = __ldg(P.aux.h + j);
      double G[NG];
      if constexpr (TOP) {
        const double hl = LP == 0 ? 1.0 : (LP == 1 ? h1 : (LP == 2 ? h1 * h1 : h1 * h1 * h1));
#pragma unroll
        for (int i = 0; i < NP; ++i) G[i] = hl * w[i];
      } else {
        static_for<NG>([&](auto hh) {
          constexpr int h = decltype(hh)::value;
          double g = 0.0;
          static_for<NP>([&](auto ii) {
            constexpr int i = decltype(ii)::value;
            g += w[i] * centred_coef(cart_a(LP, i), herm_t(h), h1) * centred_coef(cart_b(LP, i), herm_u(h), h1) *
                 centred_coef(cart_c(LP, i), herm_v(h), h1);
          });
          G[h] = g;
        });
      }
      for (int k = 0; k < nkm; ++k) {
        const int kk = min(k, nk - 1);
        const double KK = k < nk ? Kb * entry_field(kp, kk, 4) : 0.0;
        const double q = entry_field(kp, kk, 0);
        const double Q[3] = {entry_field(kp, kk, 1), entry_field(kp, kk, 2), entry_field(kp, kk, 3)};
        const double h2 = entry_field(kp, kk, 5), ga = entry_field(kp, kk, 6);
        double R[nherm(L + 1)];
        quartet_R<L + 1>(p, q, KK, Px - Q[0], Py - Q[1], Pz - Q[2], S.boys, R);
        double ex[3][LCD + 1], er[3][LCD + 1];
        ket_expansions<LC, LD>(ex, er, Q, Cc, Dd, ga, h2, ce, de);
        double gp[3] = {0, 0, 0};
        ket_gradient<LP, LCD, TOP ? LP : 0>(G, R, ex, er, tx, ty, tz, gp, gC);
        const double fc = 2.0 * h2 * ga;
#pragma unroll
        for (int x = 0; x < 3; ++x) {
          gP[x] += gp[x];
          gC[x] -= fc * gp[x];
        }
      }
    }
    const int atc = 3 * P.atom[c], atd = 3 * P.atom[d];
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      sP[x] += gP[x];
      if (active) {
        atomicAdd(g_atom + atc + x, gC[x]);
        atomicAdd(g_atom + atd + x, -gP[x] - gC[x]);
      }
    }
  }
  // the fitting centre: one sum per block
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    for (int o = 16; o > 0; o >>= 1) sP[x] += __shfl_down_sync(0xffffffffu, sP[x], o);
    if (lane == 0) S.red[tid >> 5][x] = sP[x];
  }
  __syncthreads();
  if (tid < 3) {
    double v = 0.0;
    for (int k = 0; k < GRAD_THREADS / 32; ++k) v += S.red[k][tid];
    atomicAdd(P.grad + 3 * P.aux_atom[sh] + tid, v);
  }
  if (local)
    for (int i = tid; i < 3 * P.natom; i += GRAD_THREADS)
      if (s_g[i] != 0.0) atomicAdd(P.grad + i, s_g[i]);
}

template <int LP, bool PURE, int LC, int LD>
inline cudaError_t launch_grad3_class(const Grad3Params& P, cudaStream_t s) {
  constexpr size_t base = sizeof(Grad3Shared<LP>) + 16, most = base + 24 * GRAD_ATOMS;
  static_assert(most <= SMEM_BLOCK_MAX, "shared memory of GRAD_ATOMS atoms");
  const size_t sm = base + (P.natom <= GRAD_ATOMS ? 24 * (size_t)P.natom : 0);
  const int layers = ncart(LC) * ncart(LD), chunks = (P.ent.nent + GRAD_THREADS - 1) / GRAD_THREADS;
  // blocks walk over several ket chunks where there are enough of them to fill the GPU
  int y = 1;
  while (y < chunks && (long long)P.aux.count * layers * y < 16 * P.nsm) ++y;
  return launch_smem(k_grad3<LP, PURE, LC, LD>, dim3(P.aux.count, y, layers), GRAD_THREADS, sm, most, s, P);
}
template <int LP, bool PURE>
inline cudaError_t launch_grad3_l(int pc, const Grad3Params& P, cudaStream_t s) {
  if (pc == 0) return launch_grad3_class<LP, PURE, 0, 0>(P, s);
  if (pc == 1) return launch_grad3_class<LP, PURE, 1, 0>(P, s);
  if (pc == 2) return launch_grad3_class<LP, PURE, 1, 1>(P, s);
  if (pc == 3) return launch_grad3_class<LP, PURE, 2, 0>(P, s);
  if (pc == 4) return launch_grad3_class<LP, PURE, 2, 1>(P, s);
  if (pc == 5) return launch_grad3_class<LP, PURE, 2, 2>(P, s);
  return cudaErrorInvalidValue;
}

struct Grad2Params {
  AuxView P, Q;           // two groups of fitting shells
  const int* aux_atom;
  const double* sph;
  const double* boysp;
  int naux;
  const double* W2;       // naux x naux, symmetric
  double* grad;
};

// Hermite coefficients of one fitting shell's functions from weights of its
// final functions: the top degree only (TOP), or all degrees.
template <int LP, bool PURE>
__device__ __forceinline__ void aux_cart_weights(const double* f, const double* sph, double* w) {
  constexpr int NP = ncart(LP), NF = e3_nfun(LP, PURE);
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    if constexpr (PURE && LP > 1) {
      w[i] = 0.0;
#pragma unroll
      for (int m = 0; m < NF; ++m) w[i] += sph[m * NP + i] * f[m];
    } else {
      w[i] = f[i];
    }
  }
}

// W2 . d/dP (P|Q) over the pairs of two groups: block = shell P, lanes = shells
// Q; it goes to P's atom and its negative to Q's atom.
constexpr int G2_THREADS = 64;
template <int LP, bool PP, int LQ, bool PQ>
__global__ void __launch_bounds__(G2_THREADS) k_grad2(const Grad2Params P) {
  constexpr int NP = ncart(LP), NQ = ncart(LQ), FP = e3_nfun(LP, PP), FQ = e3_nfun(LQ, PQ), L = LP + LQ + 1;
  constexpr bool TOP = (LP <= 1 || PP) && (LQ <= 1 || PQ);
  __shared__ double boys[boysp_size(L)];
  __shared__ double sphP[FP * NP], sphQ[FQ * NQ];
  const int tid = threadIdx.x, lane = tid & 31;
  load_boys<L>(boys, P.boysp);
  if (PP && LP > 1)
    for (int i = tid; i < FP * NP; i += G2_THREADS) sphP[i] = P.sph[sph_off(LP) + i];
  if (PQ && LQ > 1)
    for (int i = tid; i < FQ * NQ; i += G2_THREADS) sphQ[i] = P.sph[sph_off(LQ) + i];
  __syncthreads();
  const int sP = P.P.shells[blockIdx.x], aP = P.aux_atom[sP];
  const int p0 = P.P.foff[sP];
  double tot[3] = {0, 0, 0};
  for (int s = blockIdx.y * G2_THREADS + tid; s < P.Q.count; s += gridDim.y * G2_THREADS) {
    const int sQ = P.Q.shells[s], aQ = P.aux_atom[sQ];
    if (aP == aQ) continue;  // one-centre: d/dP + d/dQ = 0 on the same atom
    const int q0 = P.Q.foff[sQ];
    double w[NQ][NP];  // [Cartesian Q][Cartesian P]
    {
      double t[FQ][NP];
#pragma unroll
      for (int b = 0; b < FQ; ++b) {
        double f[FP];
#pragma unroll
        for (int a = 0; a < FP; ++a) f[a] = P.W2[(size_t)(q0 + b) * P.naux + p0 + a];
        aux_cart_weights<LP, PP>(f, sphP, t[b]);
      }
#pragma unroll
      for (int i = 0; i < NP; ++i) {
        double f[FQ], o[NQ];
#pragma unroll
        for (int b = 0; b < FQ; ++b) f[b] = t[b][i];
        aux_cart_weights<LQ, PQ>(f, sphQ, o);
#pragma unroll
        for (int b = 0; b < NQ; ++b) w[b][i] = o[b];
      }
    }
    double g[3] = {0, 0, 0};
    for (int j = P.P.prim_off[sP]; j < P.P.prim_off[sP] + P.P.nprim[sP]; ++j)
      for (int k = P.Q.prim_off[sQ]; k < P.Q.prim_off[sQ] + P.Q.nprim[sQ]; ++k) {
        const double hp = __ldg(P.P.h + j), hq = -__ldg(P.Q.h + k);
        double R[nherm(L)];
        quartet_R<L>(__ldg(P.P.p + j), __ldg(P.Q.p + k), __ldg(P.P.Kp + j) * __ldg(P.Q.Kp + k),
                     __ldg(P.P.x + j) - __ldg(P.Q.x + k), __ldg(P.P.y + j) - __ldg(P.Q.y + k),
                     __ldg(P.P.z + j) - __ldg(P.Q.z + k), boys, R);
        if constexpr (TOP) {
          double hl = 1.0;
#pragma unroll
          for (int i = 0; i < LP; ++i) hl *= hp;
#pragma unroll
          for (int i = 0; i < LQ; ++i) hl *= hq;
          double v[3] = {0, 0, 0};
          static_for<NP * NQ>([&](auto ab) {
            constexpr int i = decltype(ab)::value % NP, b = decltype(ab)::value / NP;
            constexpr int t = cart_a(LP, i) + cart_a(LQ, b), u = cart_b(LP, i) + cart_b(LQ, b),
                          z = cart_c(LP, i) + cart_c(LQ, b);
            v[0] += w[b][i] * R[hidx(t + 1, u, z)];
            v[1] += w[b][i] * R[hidx(t, u + 1, z)];
            v[2] += w[b][i] * R[hidx(t, u, z + 1)];
          });
#pragma unroll
          for (int x = 0; x < 3; ++x) g[x] += hl * v[x];
        } else {  // every degree of a Cartesian d or f shell; the sign of Q's odd degrees is in -h
          for (int i = 0; i < NP; ++i)
            for (int b = 0; b < NQ; ++b) {
              int pe[3] = {0, 0, 0}, qe[3] = {0, 0, 0};
              if (LP > 0) pe[0] = c_herm.t[nherm(LP - 1) + i], pe[1] = c_herm.u[nherm(LP - 1) + i], pe[2] = c_herm.v[nherm(LP - 1) + i];
              if (LQ > 0) qe[0] = c_herm.t[nherm(LQ - 1) + b], qe[1] = c_herm.u[nherm(LQ - 1) + b], qe[2] = c_herm.v[nherm(LQ - 1) + b];
              for (int m = 0; m < nherm(LP); ++m) {
                const double cp = centred_coef(pe[0], c_herm.t[m], hp) * centred_coef(pe[1], c_herm.u[m], hp) *
                                  centred_coef(pe[2], c_herm.v[m], hp) * w[b][i];
                if (cp == 0.0) continue;
                for (int n = 0; n < nherm(LQ); ++n) {
                  const int t = c_herm.t[n], u = c_herm.u[n], z = c_herm.v[n];
                  const double c0 = cp * centred_coef(qe[0], t, -hq) * centred_coef(qe[1], u, -hq) * centred_coef(qe[2], z, -hq);
                  const double c = ((t + u + z) & 1) ? -c0 : c0;
                  if (c == 0.0) continue;
                  const int T = t + c_herm.t[m], U = u + c_herm.u[m], Z = z + c_herm.v[m];
                  g[0] += c * R[hidx(T + 1, U, Z)];
                  g[1] += c * R[hidx(T, U + 1, Z)];
                  g[2] += c * R[hidx(T, U, Z + 1)];
                }
              }
            }
        }
      }
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      tot[x] += g[x];
      atomicAdd(P.grad + 3 * aQ + x, -g[x]);
    }
  }
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    double v = tot[x];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0 && v != 0.0) atomicAdd(P.grad + 3 * aP + x, v);
  }
}

// launchers (df_grad_*.cu): orbital pair class id; fitting groups gP, gQ
cudaError_t launch_grad3_s(int pair_class_id, const Grad3Params& P, cudaStream_t s);
cudaError_t launch_grad3_p(int pair_class_id, const Grad3Params& P, cudaStream_t s);
cudaError_t launch_grad3_d_pure(int pair_class_id, const Grad3Params& P, cudaStream_t s);
cudaError_t launch_grad3_d_cart(int pair_class_id, const Grad3Params& P, cudaStream_t s);
cudaError_t launch_grad3_f_pure(int pair_class_id, const Grad3Params& P, cudaStream_t s);
cudaError_t launch_grad3_f_cart(int pair_class_id, const Grad3Params& P, cudaStream_t s);
cudaError_t launch_grad2(int gP, int gQ, const Grad2Params& P, cudaStream_t s);

}  // namespace m2
