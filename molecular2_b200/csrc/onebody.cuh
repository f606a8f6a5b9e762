// Device side of the one-body integrals and of the one-body part of the RHF
// gradient: overlap, kinetic and nuclear attraction (IntegralEngine
// constructor, molecular2 src/integrals.cpp:70-72, 394-449; derivatives
// inc/integrals.hpp:169-349, contracted in src/rhfgrad.cpp:23-45).
// A nucleus is a ket of infinite exponent: sum over h of E_ab[h] R_h(p, P - C).
#pragma once
#include "jk_kernels.cuh"

namespace m2 {

constexpr int OB_THREADS = 128;  // of k_onebody
constexpr int G1_THREADS = 64;   // of k_grad1e

struct OneBodyParams {
  PairView pairs;
  EntryView ent;
  const double *ox, *oy, *oz;
  const int* foff;
  const int* pure;
  const double* sph;
  const double* boysp;
  int natom;
  const double* Z;
  const double* cxyz;  // 3*natom
  int n;
  double *S, *T, *V;   // n x n final basis, pairs that are not listed set to zero by the caller; T and V may both be NULL
};

// E^{ij}_0 of one direction for i <= LI, j <= LJ (all that overlap and kinetic
// energy need), at out[i * (LJ + 1) + j].
template <int LI, int LJ>
__device__ __forceinline__ void e0_table(double PA, double PB, double h, double* out) {
  constexpr int N = LI + LJ;
  double ea[N + 1];
#pragma unroll
  for (int t = 0; t <= N; ++t) ea[t] = 0.0;
  ea[0] = 1.0;
#pragma unroll
  for (int i = 0; i <= LI; ++i) {
    if (i > 0) e1_raise<N>(ea, PA, h);
    double eb[N + 1];
#pragma unroll
    for (int t = 0; t <= N; ++t) eb[t] = ea[t];
#pragma unroll
    for (int j = 0; j <= LJ; ++j) {
      if (j > 0) e1_raise<N>(eb, PB, h);
      out[i * (LJ + 1) + j] = eb[0];
    }
  }
}
// <i| -1/2 d2/dx2 |j> of one direction from a table of row length ld
__device__ __forceinline__ double kin1(const double* e, int ld, int i, int j, double be) {
  const double* r = e + i * ld;
  double v = -2.0 * be * be * r[j + 2] + be * (2 * j + 1) * r[j];
  if (j > 1) v -= 0.5 * j * (j - 1) * r[j - 2];
  return v;
}
template <int L>
__device__ __forceinline__ void cart_exps(int i, int* e) {
  if constexpr (L == 0) {
    e[0] = e[1] = e[2] = 0;
  } else {
    e[0] = c_herm.t[nherm(L - 1) + i];
    e[1] = c_herm.u[nherm(L - 1) + i];
    e[2] = c_herm.v[nherm(L - 1) + i];
  }
}

template <int LA, int LB>
struct OneBodyShared {
  double boys[boysp_size(LA + LB)];
  BraShared<LA, LB> bra;
  double E0[ENTRY_PRIMS][3][(LA + 1) * (LB + 3)];
  double Rs[ENTRY_PRIMS][nherm(LA + LB)];  // sum over nuclei of -Z R
  double blk[3][ncart(LA) * ncart(LB)];
};

// One block per pair, entry by entry.  A warp sums the Hermite integrals of one
// primitive over the nuclei (lanes), a thread then adds to its Cartesian element
// of S, T and V.  Every element is summed by one thread in a fixed order and
// written to both triangles, so that the matrices are the same in every run and
// exactly symmetric.  Bound by the chain of a contracted pair's entries (11 of a
// 9 x 9 contraction, 50 us for (H2O)8's ss class), which the classes' side streams
// overlap: jk_one_body of (H2O)8/cc-pVDZ 0.34 ms, of H2O 0.14 (a block per entry
// with atomics, the classes one after another: 0.39 and 0.17).
template <int LA, int LB>
__global__ void __launch_bounds__(OB_THREADS) k_onebody(const OneBodyParams P) {
  constexpr int NA = ncart(LA), NB = ncart(LB), NAB = NA * NB, L = LA + LB, H = nherm(L);
  static_assert(NAB <= OB_THREADS, "a thread per Cartesian element");
  extern __shared__ __align__(16) unsigned char ob_sm[];
  OneBodyShared<LA, LB>& S = *reinterpret_cast<OneBodyShared<LA, LB>*>(ob_sm);
  const int ip = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
  const int a = P.pairs.sa[ip], b = P.pairs.sb[ip];
  const double A[3] = {P.ox[a], P.oy[a], P.oz[a]}, B[3] = {P.ox[b], P.oy[b], P.oz[b]};
  const bool with_v = P.V != nullptr;
  if (with_v) load_boys<L>(S.boys, P.boysp);
  int ea[3] = {0, 0, 0}, eb[3] = {0, 0, 0};
  if (tid < NAB) {
    cart_exps<LA>(tid / NB, ea);
    cart_exps<LB>(tid % NB, eb);
  }
  double s = 0.0, t = 0.0, v = 0.0;
  for (int e = P.ent.first[ip]; e < P.ent.first[ip + 1]; ++e) {
    const int nb = P.ent.np[e];
    const double* base = entry_prims(P.ent, e);
    __syncthreads();  // the entry before is done with
    for (int i = tid; i < nb * 3; i += OB_THREADS) {
      const int x = i % 3;
      const double X = entry_field(base, i / 3, 1 + x);
      e0_table<LA, LB + 2>(X - A[x], X - B[x], entry_field(base, i / 3, 5), S.E0[i / 3][x]);
    }
    load_bra<LA, LB>(S.bra, base, nb, A[0], A[1], A[2], B[0], B[1], B[2]);
    if (with_v) {
      for (int ib = tid >> 5; ib < nb; ib += OB_THREADS / 32) {
        const double* q = S.bra.prim[ib];
        double acc[H];
#pragma unroll
        for (int h = 0; h < H; ++h) acc[h] = 0.0;
        for (int c = lane; c < P.natom; c += 32) {
          double R[H];
          hermite_R<L>(q[0], -P.Z[c], q[1] - P.cxyz[3 * c], q[2] - P.cxyz[3 * c + 1], q[3] - P.cxyz[3 * c + 2],
                       S.boys, R);
#pragma unroll
          for (int h = 0; h < H; ++h) acc[h] += R[h];
        }
#pragma unroll
        for (int h = 0; h < H; ++h) {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) acc[h] += __shfl_down_sync(0xffffffffu, acc[h], o);
          if (lane == 0) S.Rs[ib][h] = acc[h];
        }
      }
      __syncthreads();
    }
    if (tid < NAB) {
      for (int ib = 0; ib < nb; ++ib) {
        const double p = S.bra.prim[ib][0], K = S.bra.prim[ib][4] * p / SQRT_PI25X2();
        const double be = p - entry_field(base, ib, 6), pip = M_PI / p, ov = K * pip * sqrt(pip);
        double o[3], k[3];
        for (int x = 0; x < 3; ++x) {
          o[x] = S.E0[ib][x][ea[x] * (LB + 3) + eb[x]];
          k[x] = kin1(S.E0[ib][x], LB + 3, ea[x], eb[x], be);
        }
        s += ov * o[0] * o[1] * o[2];
        t += ov * (k[0] * o[1] * o[2] + o[0] * k[1] * o[2] + o[0] * o[1] * k[2]);
        if (with_v) v += 2.0 * M_PI / p * K * bra_component<LA, LB>(S.bra.M[L > 0 ? ib : 0], S.Rs[ib], tid);
      }
    }
  }
  if (tid < NAB) {
    S.blk[0][tid] = s;
    S.blk[1][tid] = t;
    S.blk[2][tid] = v;
  }
  __syncthreads();
  // final basis, both triangles
  const int pa = P.pure[a], pb = P.pure[b];
  const int fa = pa ? 2 * LA + 1 : NA, fb = pb ? 2 * LB + 1 : NB;
  const int a0 = P.foff[a], b0 = P.foff[b];
  double* outs[3] = {P.S, P.T, P.V};
  for (int i = tid; i < (with_v ? 3 : 1) * fa * fb; i += OB_THREADS) {
    const int k = i / (fa * fb), m = (i / fb) % fa, q = i % fb;
    if (a == b && m < q) continue;  // (q, m) writes it
    double val = 0.0;
    for (int i1 = pa ? 0 : m; i1 < (pa ? NA : m + 1); ++i1) {
      const double ta = pa ? P.sph[sph_off(LA) + m * NA + i1] : 1.0;
      for (int j1 = pb ? 0 : q; j1 < (pb ? NB : q + 1); ++j1)
        val += ta * (pb ? P.sph[sph_off(LB) + q * NB + j1] : 1.0) * S.blk[k][i1 * NB + j1];
    }
    outs[k][(size_t)(b0 + q) * P.n + a0 + m] = val;
    outs[k][(size_t)(a0 + m) * P.n + b0 + q] = val;
  }
}

struct Grad1eParams {
  int nsm;
  PairView pairs;
  EntryView ent;
  const double *ox, *oy, *oz;
  const int* coff;
  const int* atom;
  const unsigned char* sig;
  const double* Dc;  // Cartesian D, nc x nc
  const double* Wc;  // Cartesian W
  int nc;
  const double* boysp;
  int natom;
  const double* Z;
  const double* cxyz;
  double* grad;
};
constexpr int G1_ATOMS = 2048;  // atoms whose gradient a block sums in shared memory

template <int LA, int LB>
struct Grad1eShared {
  double boys[boysp_size(LA + LB + 1)];
  BraGradShared<LA, LB> bra;
  double E0[ENTRY_PRIMS][3][(LA + 2) * (LB + 3)];
  double G[ENTRY_PRIMS][4][nherm(LA + LB)];  // sum over ab of D_ab M, and of the d/dR tables
  double red[G1_THREADS / 32][6];
};

// T'.D - 2 S'.W + V'.D.  Blocks walk over the pair entries; the density is
// folded into the Hermite expansions once per primitive (G), a thread then
// takes one (primitive, nucleus): R of order LAB + 1 gives the bra's shift, the
// coefficient derivatives and the nucleus's own force.  One thread per pair
// with a Hermite sum per component and nucleus took 29 ms for (H2O)8, the six
// launches now take under 1 ms.
template <int LA, int LB>
__global__ void __launch_bounds__(G1_THREADS) k_grad1e(const Grad1eParams P) {
  constexpr int NA = ncart(LA), NB = ncart(LB), NAB = NA * NB, L = LA + LB, H = nherm(L), LD = LB + 3;
  extern __shared__ __align__(16) unsigned char g1_sm[];
  Grad1eShared<LA, LB>& S = *reinterpret_cast<Grad1eShared<LA, LB>*>(g1_sm);
  double* s_g = reinterpret_cast<double*>(g1_sm + ((sizeof(Grad1eShared<LA, LB>) + 15) & ~(size_t)15));
  const int tid = threadIdx.x, lane = tid & 31;
  const bool local = P.natom <= G1_ATOMS;
  double* g_atom = local ? s_g : P.grad;
  load_boys<L + 1>(S.boys, P.boysp);
  if (local)
    for (int i = tid; i < 3 * P.natom; i += G1_THREADS) s_g[i] = 0.0;
  for (int e = blockIdx.x; e < P.ent.nent; e += gridDim.x) {
    const int ip = P.ent.pair[e];
    if (!P.sig[ip]) continue;
    __syncthreads();  // the previous entry's tables
    const int a = P.pairs.sa[ip], b = P.pairs.sb[ip], nb = P.ent.np[e];
    const double sym = (a == b) ? 1.0 : 2.0;
    const double A[3] = {P.ox[a], P.oy[a], P.oz[a]}, B[3] = {P.ox[b], P.oy[b], P.oz[b]};
    const double* base = entry_prims(P.ent, e);
    const int a0 = P.coff[a], b0 = P.coff[b];
    for (int i = tid; i < nb * 3; i += G1_THREADS) {
      const int x = i % 3;
      const double X = entry_field(base, i / 3, 1 + x);
      e0_table<LA + 1, LB + 2>(X - A[x], X - B[x], entry_field(base, i / 3, 5), S.E0[i / 3][x]);
    }
    load_bra_grad<LA, LB>(S.bra, base, nb, A[0], A[1], A[2], B[0], B[1], B[2]);
    for (int i = tid; i < nb * 4; i += G1_THREADS) {
      const double* M = S.bra.M[i / 4][i % 4];
      double g[H];
#pragma unroll
      for (int h = 0; h < H; ++h) g[h] = 0.0;
      double d[NAB];
#pragma unroll
      for (int j = 0; j < NAB; ++j) d[j] = sym * P.Dc[(size_t)(a0 + j / NB) * P.nc + b0 + j % NB];
      for_terms<LA, LB>([&](auto ab, auto k, auto h) {
        g[decltype(h)::value] += d[decltype(ab)::value] * M[decltype(k)::value];
      });
#pragma unroll
      for (int h = 0; h < H; ++h) S.G[i / 4][i % 4][h] = g[h];
    }
    __syncthreads();
    double gA[3] = {0, 0, 0}, gB[3] = {0, 0, 0};
    // nuclear attraction
    for (int i = tid; i < nb * P.natom; i += G1_THREADS) {
      const int c = i % P.natom, ib = i / P.natom;
      const double* q = S.bra.prim[ib];
      double R[nherm(L + 1)];
      hermite_R<L + 1>(q[0], -P.Z[c] * 2.0 * M_PI / SQRT_PI25X2() * q[4], q[1] - P.cxyz[3 * c],
                       q[2] - P.cxyz[3 * c + 1], q[3] - P.cxyz[3 * c + 2], S.boys, R);
      double gp[3] = {0, 0, 0}, gr[3] = {0, 0, 0};
      static_for<H>([&](auto hh) {
        constexpr int h = decltype(hh)::value, t = herm_t(h), u = herm_u(h), v = herm_v(h);
        const double g0 = S.G[ib][0][h];
        gp[0] += g0 * R[hidx(t + 1, u, v)];
        gp[1] += g0 * R[hidx(t, u + 1, v)];
        gp[2] += g0 * R[hidx(t, u, v + 1)];
        gr[0] += S.G[ib][1][h] * R[h];
        gr[1] += S.G[ib][2][h] * R[h];
        gr[2] += S.G[ib][3][h] * R[h];
      });
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        const double dA = q[5] * gp[x] + gr[x];
        gA[x] += dA;
        gB[x] += gp[x] - dA;
        atomicAdd(g_atom + 3 * c + x, -gp[x]);
      }
    }
    // overlap and kinetic: d/dB = -d/dA
    for (int i = tid; i < nb * NAB; i += G1_THREADS) {
      const int ib = i / NAB, ia = (i % NAB) / NB, jb = i % NB;
      int ea[3], eb[3];
      cart_exps<LA>(ia, ea);
      cart_exps<LB>(jb, eb);
      const double p = S.bra.prim[ib][0], al = entry_field(base, ib, 6), be = p - al;
      const double K = S.bra.prim[ib][4] * p / SQRT_PI25X2(), pip = M_PI / p, ov = K * pip * sqrt(pip);
      const double dab = sym * ov * P.Dc[(size_t)(a0 + ia) * P.nc + b0 + jb];
      const double wab = -2.0 * sym * ov * P.Wc[(size_t)(a0 + ia) * P.nc + b0 + jb];
      double o[3], k[3], od[3], kd[3];  // overlap and kinetic factors and their derivatives
      for (int x = 0; x < 3; ++x) {
        const double* E = S.E0[ib][x];
        o[x] = E[ea[x] * LD + eb[x]];
        k[x] = kin1(E, LD, ea[x], eb[x], be);
        od[x] = 2.0 * al * E[(ea[x] + 1) * LD + eb[x]];
        kd[x] = 2.0 * al * kin1(E, LD, ea[x] + 1, eb[x], be);
        if (ea[x] > 0) {
          od[x] -= ea[x] * E[(ea[x] - 1) * LD + eb[x]];
          kd[x] -= ea[x] * kin1(E, LD, ea[x] - 1, eb[x], be);
        }
      }
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        const int y = (x + 1) % 3, z = (x + 2) % 3;
        const double v = dab * (kd[x] * o[y] * o[z] + od[x] * (k[y] * o[z] + o[y] * k[z])) + wab * od[x] * o[y] * o[z];
        gA[x] += v;
        gB[x] -= v;
      }
    }
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      for (int o = 16; o > 0; o >>= 1) {
        gA[x] += __shfl_down_sync(0xffffffffu, gA[x], o);
        gB[x] += __shfl_down_sync(0xffffffffu, gB[x], o);
      }
      if (lane == 0) {
        S.red[tid >> 5][x] = gA[x];
        S.red[tid >> 5][3 + x] = gB[x];
      }
    }
    __syncthreads();
    if (tid < 6) {
      double v = 0.0;
      for (int w = 0; w < G1_THREADS / 32; ++w) v += S.red[w][tid];
      atomicAdd(g_atom + 3 * P.atom[tid < 3 ? a : b] + tid % 3, v);
    }
  }
  __syncthreads();
  if (local)
    for (int i = tid; i < 3 * P.natom; i += G1_THREADS)
      if (s_g[i] != 0.0) atomicAdd(P.grad + i, s_g[i]);
}

cudaError_t launch_onebody(int pc, const OneBodyParams& P, cudaStream_t s);  // onebody.cu
cudaError_t launch_grad1e(int pc, const Grad1eParams& P, cudaStream_t s);

}  // namespace m2
