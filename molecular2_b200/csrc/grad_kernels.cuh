// Device side of the RHF nuclear gradient (FP64): the adjoint of the direct
// J/K build and of the one-body matrices.  Derivative integrals are recomputed
// per shell quartet / pair and contracted at once with the density weights, so
// no derivative integral or derivative Fock matrix is ever stored
// (molecular2 builds 3N derivative Fock matrices, src/rhfgrad.cpp:419-598).
//
// The derivatives with respect to the four centres of a quartet come from one
// table of Hermite integrals of order L + 1 per primitive quartet (quartet.cuh):
// d/dP by index shifts, d/dA = (alpha/p) d/dP + d/dR_ab and
// d/dC = -(gamma/q) d/dP + d/dR_cd from differentiated expansion coefficients,
// d/dB = d/dP - d/dA, d/dD = -d/dP - d/dC.
#pragma once
#include "jk_kernels.cuh"

namespace m2 {

struct Grad2eParams {
  PairView bra, ket;
  EntryView bra_ent, ket_ent;
  int same_class;
  ShellView sh;
  const int* atom;     // shell -> atom
  const unsigned char* bra_sig;  // overlap significance of each pair (shell-pair list)
  const unsigned char* ket_sig;
  const double* Dnorm;
  int nshell;
  const double* Dmax;
  const double* Dc;    // Cartesian density, nc x nc
  int nc;
  double precision, eps;  // eps: prim_eps(precision)
  const double* boysp;
  double* grad;        // 3 * natom
  int natom;
  int kchunk;          // ket entries per block, at most GRAD_LIST
  int bra0, bra_step;        // this rank's bra pairs: bra0, bra0 + bra_step, ...
};

constexpr int GRAD_THREADS = 128;
constexpr int GRAD_LIST = 512;
constexpr int GRAD_ATOMS = 512;  // atoms whose gradient a block sums in shared memory

template <int LA, int LB>
struct GradShared {
  double boys[boysp_size(2 * (LA + LB) + 1)];
  BraGradShared<LA, LB> bra;
  double Dab[ncart(LA) * ncart(LB)];
  double red[GRAD_THREADS / 32][6];
  int list[GRAD_LIST];
  int n;
};

// Four-index gradient of one class pair: block (x, y, z) = bra entry, ket entry
// chunk, ket component.  Per entry pair a thread folds the density weights
// 1/2 D_ab D_cd - 1/8 (D_ac D_bd + D_ad D_bc) into the bra's Hermite expansion
// (G), so that a primitive quartet costs one R table of order L + 1 and the
// products of G with it; nothing of the size of the integral block exists.
// The bra's derivatives stay in registers over all kets of the thread, the
// kets' are summed per atom in shared memory (few atoms: global atomics on the
// same addresses would serialise).  Measured, the 21 class launches of
// (H2O)8/cc-pVDZ: 340 -> 14 ms against six shifted quartet evaluations per
// quartet with the integral block and its weights in local memory; the whole
// call 372 -> 18 ms, 13.5 ms with the Boys table and cached device blocks.  Two
// blocks per SM are asked for because ptxas otherwise
// gives the dd classes 32 registers and 50 to 120 KB of spills.
template <int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__(GRAD_THREADS, 2) k_grad2e(const Grad2eParams P) {
  constexpr int NA = ncart(LA), NB = ncart(LB), ND = ncart(LD), NAB = NA * NB;
  constexpr int LAB = LA + LB, LCD = LC + LD, L = LAB + LCD, HAB = nherm(LAB);
  static_assert(LCD <= LAB, "the bra's Boys table covers the ket");
  extern __shared__ __align__(16) unsigned char grad_sm[];
  GradShared<LA, LB>& S = *reinterpret_cast<GradShared<LA, LB>*>(grad_sm);
  double* s_g = reinterpret_cast<double*>(grad_sm + ((sizeof(GradShared<LA, LB>) + 15) & ~(size_t)15));

  const int eb = blockIdx.x;
  const int bra = P.bra_ent.pair[eb];
  if (bra % P.bra_step != P.bra0 || !P.bra_sig[bra]) return;
  const int a = P.bra.sa[bra], b = P.bra.sb[bra];
  const double Qab = P.bra.Q[bra];
  const double Dmax = *P.Dmax;
  if (!(Qab * Dmax > 0.0)) return;
  int npk = window_up(q_prefix(P.ket.Q, P.ket.npair, P.precision / (Qab * Dmax)), P.ket.npair);
  if (P.same_class) npk = min(npk, bra + 1);
  const int nent = P.ket_ent.first[npk];
  const int start = blockIdx.y * P.kchunk;
  if (start >= nent) return;
  const int end = min(start + P.kchunk, nent);
  const int tid = threadIdx.x, lane = tid & 31;
  const int ns = P.nshell;
  const double* Dn = P.Dnorm;
  const double dab = Dn[a * ns + b];
  const int n = pack_kets(start, end, 0, S.list, &S.n, [&](int e) {
    const int kl = P.ket_ent.pair[e];
    if (!P.ket_sig[kl]) return false;
    const int c = P.ket.sa[kl], d = P.ket.sb[kl];
    double dn = fmax(fmax(dab, Dn[c * ns + d]), fmax(Dn[a * ns + c], Dn[a * ns + d]));
    dn = fmax(dn, fmax(Dn[b * ns + c], Dn[b * ns + d]));
    return !(dn * Qab * P.ket.Q[kl] < P.precision);
  });
  if (n == 0) return;

  const int a0 = P.sh.coff[a], b0 = P.sh.coff[b], nc = P.nc;
  const int nb = P.bra_ent.np[eb];
  const double* __restrict__ Dc = P.Dc;
  const bool local = P.natom <= GRAD_ATOMS;
  load_boys<L + 1>(S.boys, P.boysp);
  for (int i = tid; i < NAB; i += GRAD_THREADS) S.Dab[i] = Dc[(size_t)(a0 + i / NB) * nc + b0 + i % NB];
  if (local)
    for (int i = tid; i < 3 * P.natom; i += GRAD_THREADS) s_g[i] = 0.0;
  load_bra_grad<LA, LB>(S.bra, entry_prims(P.bra_ent, eb), nb, P.sh.x[a], P.sh.y[a], P.sh.z[a], P.sh.x[b],
                        P.sh.y[b], P.sh.z[b]);
  double* g_atom = local ? s_g : P.grad;

  // this block's ket component
  const int ic = blockIdx.z / ND, id = blockIdx.z % ND;
  int ce[3] = {0, 0, 0}, de[3] = {0, 0, 0};
  if constexpr (LC > 0) {
    ce[0] = c_herm.t[nherm(LC - 1) + ic];
    ce[1] = c_herm.u[nherm(LC - 1) + ic];
    ce[2] = c_herm.v[nherm(LC - 1) + ic];
  }
  if constexpr (LD > 0) {
    de[0] = c_herm.t[nherm(LD - 1) + id];
    de[1] = c_herm.u[nherm(LD - 1) + id];
    de[2] = c_herm.v[nherm(LD - 1) + id];
  }
  const int tx = ce[0] + de[0], ty = ce[1] + de[1], tz = ce[2] + de[2];

  double sA[3] = {0, 0, 0}, sP[3] = {0, 0, 0};  // bra: d/dA and d/dP over this thread's kets
  for (int t0 = (tid >> 5) * 32; t0 < n; t0 += GRAD_THREADS) {
    const bool active = t0 + lane < n;
    const int e = S.list[active ? t0 + lane : n - 1];
    const int kl = P.ket_ent.pair[e];
    const int c = P.ket.sa[kl], d = P.ket.sb[kl];
    const double* kp = entry_prims(P.ket_ent, e);
    const int nk = P.ket_ent.np[e];
    const int nkm = __reduce_max_sync(0xffffffffu, nk);
    const double deg = !active ? 0.0
                               : ((a == b) ? 1.0 : 2.0) * ((c == d) ? 1.0 : 2.0) *
                                     ((P.same_class && kl == bra) ? 1.0 : 2.0);
    const double Cc[3] = {P.sh.x[c], P.sh.y[c], P.sh.z[c]}, Dd[3] = {P.sh.x[d], P.sh.y[d], P.sh.z[d]};
    double w[NAB];  // density weights of the 2e energy
    {
      const int c0 = P.sh.coff[c] + ic, d0 = P.sh.coff[d] + id;
      const double h = 0.5 * deg * Dc[(size_t)c0 * nc + d0], q = -0.125 * deg;
      double bc[NB], bd[NB];
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        bc[j] = q * Dc[(size_t)(b0 + j) * nc + c0];
        bd[j] = q * Dc[(size_t)(b0 + j) * nc + d0];
      }
#pragma unroll
      for (int i = 0; i < NA; ++i) {
        const double ac = Dc[(size_t)(a0 + i) * nc + c0], ad = Dc[(size_t)(a0 + i) * nc + d0];
#pragma unroll
        for (int j = 0; j < NB; ++j) w[i * NB + j] = h * S.Dab[i * NB + j] + ac * bd[j] + ad * bc[j];
      }
    }
    double gP[3] = {0, 0, 0}, gC[3] = {0, 0, 0};
    for (int ib = 0; ib < nb; ++ib) {
      const double p = S.bra.prim[ib][0], Px = S.bra.prim[ib][1], Py = S.bra.prim[ib][2], Pz = S.bra.prim[ib][3];
      const double Kb = S.bra.prim[ib][4];
      double G[HAB], W[HAB], gb[3] = {0, 0, 0};
#pragma unroll
      for (int h = 0; h < HAB; ++h) G[h] = W[h] = 0.0;
      const double* M = S.bra.M[ib][0];
      for_terms<LA, LB>([&](auto ab, auto k, auto h) {
        G[decltype(h)::value] += w[decltype(ab)::value] * M[decltype(k)::value];
      });
      KetPrim next = load_ket<true>(kp, 0);
      for (int k = 0; k < nkm; ++k) {
        const KetPrim kq = next;  // the next primitive's loads run behind this one's arithmetic
        const double ga = entry_field(kp, min(k, nk - 1), 6);
        next = load_ket<true>(kp, min(k + 1, nk - 1));
        const double KK = k < nk && active ? Kb * kq.K : 0.0;
        if (!__any_sync(0xffffffffu, fabs(KK) > P.eps)) break;  // largest first: the rest is smaller
        const double q = kq.q, h2 = kq.h;
        const double Q[3] = {kq.x, kq.y, kq.z};
        double R[nherm(L + 1)];
        quartet_R<L + 1>(p, q, KK, Px - Q[0], Py - Q[1], Pz - Q[2], S.boys, R);
        double ex[3][LCD + 1], er[3][LCD + 1];
        ket_expansions<LC, LD>(ex, er, Q, Cc, Dd, ga, h2, ce, de);
        ket_accumulate<LAB, LCD>(W, R, ex[0], ex[1], ex[2], tx, ty, tz);
        double gp[3] = {0, 0, 0};
        ket_gradient<LAB, LCD>(G, R, ex, er, tx, ty, tz, gp, gC);
        const double fc = 2.0 * h2 * ga;
#pragma unroll
        for (int x = 0; x < 3; ++x) {
          gb[x] += gp[x];
          gC[x] -= fc * gp[x];
        }
      }
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        gP[x] += gb[x];
        sA[x] += S.bra.prim[ib][5] * gb[x];
      }
      for_terms<LA, LB>([&](auto ab, auto k, auto h) {
        const double v = w[decltype(ab)::value] * W[decltype(h)::value];
        constexpr int NT = nterms(LA, LB), kk = decltype(k)::value;
        sA[0] += M[NT + kk] * v;
        sA[1] += M[2 * NT + kk] * v;
        sA[2] += M[3 * NT + kk] * v;
      });
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
  // the bra's atoms are the same for the whole block: one sum, one atomic
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    double v = sA[x], u = sP[x] - sA[x];
    for (int o = 16; o > 0; o >>= 1) {
      v += __shfl_down_sync(0xffffffffu, v, o);
      u += __shfl_down_sync(0xffffffffu, u, o);
    }
    if (lane == 0) {
      S.red[tid >> 5][x] = v;
      S.red[tid >> 5][3 + x] = u;
    }
  }
  __syncthreads();
  if (tid < 6) {
    double v = 0.0;
    for (int k = 0; k < GRAD_THREADS / 32; ++k) v += S.red[k][tid];
    atomicAdd(P.grad + 3 * P.atom[tid < 3 ? a : b] + tid % 3, v);
  }
  if (local)
    for (int i = tid; i < 3 * P.natom; i += GRAD_THREADS)
      if (s_g[i] != 0.0) atomicAdd(P.grad + i, s_g[i]);
}

template <int LA, int LB, int LC, int LD>
inline cudaError_t launch_grad2e_class(const Grad2eParams& P, dim3 grid, cudaStream_t s) {
  constexpr size_t base = sizeof(GradShared<LA, LB>) + 16, most = base + 24 * GRAD_ATOMS;
  static_assert(most <= SMEM_BLOCK_MAX, "shared memory of GRAD_ATOMS atoms");
  const size_t sm = base + (P.natom <= GRAD_ATOMS ? 24 * (size_t)P.natom : 0);
  return launch_smem(k_grad2e<LA, LB, LC, LD>, grid, GRAD_THREADS, sm, most, s, P);
}

// launchers (grad_cls_*.cu)
cudaError_t launch_grad2e_bra_s(int A, int B, const Grad2eParams& P, dim3 grid, cudaStream_t s);
cudaError_t launch_grad2e_bra_ds(int B, const Grad2eParams& P, dim3 grid, cudaStream_t s);
cudaError_t launch_grad2e_bra_dp(int B, const Grad2eParams& P, dim3 grid, cudaStream_t s);
cudaError_t launch_grad2e_bra_dd(int B, const Grad2eParams& P, dim3 grid, cudaStream_t s);
cudaError_t launch_grad2e_bra_dd_hi(int B, const Grad2eParams& P, dim3 grid, cudaStream_t s);

}  // namespace m2
