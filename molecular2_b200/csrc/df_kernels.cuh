// Device side of the density-fitting integrals: three-index (P|mn) and
// two-index (P|Q) Coulomb integrals over the fitting basis, McMurchie-Davidson
// with a unit s function as the partner of each fitting function (libint2 BraKet::xs_xx
// and xs_xs in molecular2, src/eris.cpp:89-156, 304-356).
#pragma once
#include "jk_kernels.cuh"

struct jk_engine;

namespace m2 {

// Fitting shells of one angular momentum, all pure or all Cartesian.
struct AuxView {
  const int* shells;
  int count;
  const int* prim_off;
  const int* nprim;
  const double *p, *x, *y, *z;  // primitives
  const double* Kp;             // coefficient sqrt(2 pi^(5/2)) / p
  const double* h;              // 1 / (2p)
  const int* foff;              // final function offsets
};

AuxView aux_group_view(const jk_engine* e, const int* shells, int count);  // df.cu

struct Eri3Params {
  int nsm;
  AuxView aux;
  EntryView ent;          // orbital pairs of one class
  PairView pairs;
  const double *ox, *oy, *oz;
  const int* obs_foff;
  const int* obs_pure;
  const double* sph;
  const double* boysp;
  const int* plist;       // the pairs to do (indices into the class list), or NULL for all
  int nlist;
  // T[(r ncol + c) naux + P] = (P | x y) for x = x0 + r < x0 + nrow and
  // y = y0 + c < y0 + ncol, both orientations of a pair
  int x0, y0, nrow, ncol;
  int naux;
  double* T;
  // k_eri3_J: J[x][y] (x >= y) += sum over this view's P of cc_P (P | x y)
  const double* cc;       // coefficients of the Cartesian fitting components
  const int* aux_coff;    // Cartesian function offsets of the fitting shells
  int n;
  double* J;              // n x n column-major
};

constexpr int DF_TILE = 128;
constexpr int E3_THREADS = 128;  // most threads of a block

// Whether a thread keeps all functions of its fitting shell at once (their
// Hermite sums and Cartesian blocks beside R in registers), or the block does
// one function per layer.
__host__ __device__ constexpr int e3_nfun(int lp, bool pure) { return pure ? 2 * lp + 1 : ncart(lp); }
__host__ __device__ constexpr bool e3_full(int la, int lb, int lp, bool pure) {
  return e3_nfun(lp, pure) * (ncart(la) * ncart(lb) + nherm(la + lb)) + nherm(la + lb + lp) <= 90 &&
         (lp <= 1 || pure);
}

template <int LA, int LB, int LP>
struct Eri3Shared {
  double boys[boysp_size(LA + LB + LP)];
  BraShared<LA, LB> bra;
  double sphP[(2 * LP + 1) * ncart(LP)];
  double red[E3_THREADS / 32][nherm(LA + LB)];
};

// W[h] += f R[h + a] for the Hermite index a of degree LP
template <int HL, int LP, int A>
__device__ __forceinline__ void shift_accumulate(double* W, const double* R, double f) {
  constexpr int a = LP > 0 ? nherm(LP - 1) + A : 0;
  static_for<nherm(HL)>([&](auto hh) {
    constexpr int h = decltype(hh)::value;
    W[h] += f * R[hidx(herm_t(h) + herm_t(a), herm_u(h) + herm_u(a), herm_v(h) + herm_v(a))];
  });
}

// d index of a Cartesian block [6][REST] or [REST][6] (STRIDE) to the pure d
// functions, in place of the first five: xy, yz, z^2, xz, x^2 - y^2.
template <int N, int STRIDE>
__device__ __forceinline__ void pure_d(const double* in, double* out, const double* T) {
  // rows of the solid-harmonic block and their non-zero components
  out[0 * STRIDE] = __ldg(T + 0 * 6 + 1) * in[1 * STRIDE];
  out[1 * STRIDE] = __ldg(T + 1 * 6 + 4) * in[4 * STRIDE];
  out[2 * STRIDE] = __ldg(T + 2 * 6 + 0) * in[0 * STRIDE] + __ldg(T + 2 * 6 + 3) * in[3 * STRIDE] +
                    __ldg(T + 2 * 6 + 5) * in[5 * STRIDE];
  out[3 * STRIDE] = __ldg(T + 3 * 6 + 2) * in[2 * STRIDE];
  out[4 * STRIDE] = __ldg(T + 4 * 6 + 0) * in[0 * STRIDE] + __ldg(T + 4 * 6 + 3) * in[3 * STRIDE];
}

// (P|mn).  Block = (orbital pair, function layer, slice of the fitting
// shells); the lanes hold fitting shells and T keeps P fastest, so a warp
// writes neighbouring words (a lane per orbital pair scattered 8-byte words
// over rows naux apart).  A pure or s, p fitting function centred on its own
// primitive has only Hermite terms of its top degree (solid harmonics are
// harmonic), (1/2q)^l of its Cartesian coefficients.  Measured through the FP64
// build on tiled storage, (H2O)16/aug-cc-pVDZ (n 656, naux 2400), which takes
// one pass of T and one of J: 340 -> 79 ms, 43 ms with the later GEMM (a thread per contracted (pair,
// shell) before, T re-made for J).
template <int LA, int LB, int LP, bool PURE>
__global__ void __launch_bounds__(E3_THREADS, 2) k_eri3(const Eri3Params P) {
  constexpr int NA = ncart(LA), NB = ncart(LB), NAB = NA * NB, LAB = LA + LB, H = nherm(LAB), L = LAB + LP;
  constexpr int NP = ncart(LP), NF = e3_nfun(LP, PURE);
  constexpr bool FULL = e3_full(LA, LB, LP, PURE), TOP = LP <= 1 || PURE;
  constexpr int G = FULL ? NF : 1;
  extern __shared__ __align__(16) unsigned char e3_sm[];
  Eri3Shared<LA, LB, LP>& S = *reinterpret_cast<Eri3Shared<LA, LB, LP>*>(e3_sm);
  const int tid = threadIdx.x;
  const int ip = P.plist ? P.plist[blockIdx.x] : (int)blockIdx.x;
  const int a = P.pairs.sa[ip], b = P.pairs.sb[ip];
  const int e0 = P.ent.first[ip], e1 = P.ent.first[ip + 1];
  const int f0 = blockIdx.y;  // the layer's function
  load_boys<L, BOYSP_COEF_DF>(S.boys, P.boysp);
  if constexpr (PURE && LP > 1)
    for (int i = tid; i < NF * NP; i += blockDim.x) S.sphP[i] = P.sph[sph_off(LP) + i];
  const double A[3] = {P.ox[a], P.oy[a], P.oz[a]}, B[3] = {P.ox[b], P.oy[b], P.oz[b]};
  if (e1 - e0 == 1) load_bra<LA, LB>(S.bra, entry_prims(P.ent, e0), P.ent.np[e0], A[0], A[1], A[2], B[0], B[1], B[2]);

  for (int s0 = blockIdx.z * blockDim.x; s0 < P.aux.count; s0 += gridDim.z * blockDim.x) {
    const bool active = s0 + tid < P.aux.count;
    const int sh = P.aux.shells[active ? s0 + tid : P.aux.count - 1];
    const int j0 = P.aux.prim_off[sh], nj = P.aux.nprim[sh];
    const int njm = __reduce_max_sync(0xffffffffu, nj);
    double out[G][NAB];
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
      for (int i = 0; i < NAB; ++i) out[g][i] = 0.0;
    for (int e = e0; e < e1; ++e) {
      const int nb = P.ent.np[e];
      if (e1 - e0 > 1) {
        __syncthreads();
        load_bra<LA, LB>(S.bra, entry_prims(P.ent, e), nb, A[0], A[1], A[2], B[0], B[1], B[2]);
      }
      for (int ib = 0; ib < nb; ++ib) {
        const double* q = S.bra.prim[ib];
        double W[G][H];
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
          for (int h = 0; h < H; ++h) W[g][h] = 0.0;
        for (int j = 0; j < njm; ++j) {
          const int k = j0 + min(j, nj - 1);
          const double KK = j < nj ? q[4] * __ldg(P.aux.Kp + k) : 0.0;
          double R[nherm(L)];
          quartet_R<L, BOYSP_COEF_DF>(q[0], __ldg(P.aux.p + k), KK, q[1] - __ldg(P.aux.x + k), q[2] - __ldg(P.aux.y + k),
                       q[3] - __ldg(P.aux.z + k), S.boys, R);
          if constexpr (LP == 0) {
#pragma unroll
            for (int h = 0; h < H; ++h) W[0][h] += R[h];
          } else if constexpr (TOP) {
            const double h1 = -__ldg(P.aux.h + k);
            const double hl = LP == 1 ? h1 : (LP == 2 ? h1 * h1 : h1 * h1 * h1);
            static_for<G>([&](auto gg) {
              constexpr int g = decltype(gg)::value;
              static_for<NP>([&](auto aa) {
                constexpr int ca = decltype(aa)::value;
                if constexpr (LP == 1) {
                  if (FULL ? g == ca : f0 == ca) shift_accumulate<LAB, LP, ca>(W[g], R, hl);
                } else {
                  const double c = S.sphP[(FULL ? g : f0) * NP + ca];
                  if (c != 0.0) shift_accumulate<LAB, LP, ca>(W[g], R, hl * c);
                }
              });
            });
          } else {
            const double h1 = __ldg(P.aux.h + k);
            const int ce[3] = {c_herm.t[nherm(LP - 1) + f0], c_herm.u[nherm(LP - 1) + f0], c_herm.v[nherm(LP - 1) + f0]};
            double ex[3][LP + 1];
#pragma unroll
            for (int x = 0; x < 3; ++x) {
#pragma unroll
              for (int t = 0; t <= LP; ++t) ex[x][t] = t == 0 ? 1.0 : 0.0;
#pragma unroll
              for (int t = 0; t < LP; ++t)
                if (t < ce[x]) e1_raise<LP>(ex[x], 0.0, h1);
            }
            ket_accumulate<LAB, LP>(W[0], R, ex[0], ex[1], ex[2], ce[0], ce[1], ce[2]);
          }
        }
#pragma unroll
        for (int g = 0; g < G; ++g) bra_transform<LA, LB, 1>(S.bra.M[LAB > 0 ? ib : 0], W[g], out[g]);
      }
    }
    if (!active) continue;
    // final orbital functions, both orientations
    const bool pa = LA == 2 && P.obs_pure[a], pb = LB == 2 && P.obs_pure[b];
    const int fa = pa ? 5 : NA, fb = pb ? 5 : NB;
    const int m0 = P.obs_foff[a], n0 = P.obs_foff[b];
    double* T = P.T + P.aux.foff[sh] + (FULL ? 0 : f0);
#pragma unroll
    for (int g = 0; g < G; ++g) {
      if constexpr (LA == 2) {
        if (pa) {
          double t[5 * NB];
#pragma unroll
          for (int j = 0; j < NB; ++j) pure_d<NB, NB>(out[g] + j, t + j, P.sph + sph_off(2));
#pragma unroll
          for (int i = 0; i < 5 * NB; ++i) out[g][i] = t[i];
        }
      }
      if constexpr (LB == 2) {
        if (pb) {
#pragma unroll
          for (int i = 0; i < NA; ++i) {
            double t[5];
            pure_d<1, 1>(out[g] + i * 6, t, P.sph + sph_off(2));
#pragma unroll
            for (int j = 0; j < 5; ++j) out[g][i * 6 + j] = t[j];
          }
        }
      }
#pragma unroll
      for (int i = 0; i < NA; ++i)
#pragma unroll
        for (int j = 0; j < NB; ++j)
          if (i < fa && j < fb) {
            const int X = m0 + i, Y = n0 + j;
            const unsigned r1 = (unsigned)(X - P.x0), c1 = (unsigned)(Y - P.y0);
            if (r1 < (unsigned)P.nrow && c1 < (unsigned)P.ncol) T[((size_t)r1 * P.ncol + c1) * P.naux + g] = out[g][i * NB + j];
            const unsigned r2 = (unsigned)(Y - P.x0), c2 = (unsigned)(X - P.y0);
            if (r2 < (unsigned)P.nrow && c2 < (unsigned)P.ncol) T[((size_t)r2 * P.ncol + c2) * P.naux + g] = out[g][i * NB + j];
          }
    }
  }
}

// J_mn = sum_P c_P (P|mn) without storing an integral: the coefficients are
// folded into the fitting functions' Hermite expansions, the block sums the
// bra's Hermite potential W over its lanes' shells and transforms it once.
template <int LA, int LB, int LP, bool PURE>
__global__ void __launch_bounds__(E3_THREADS, 2) k_eri3_J(const Eri3Params P) {
  constexpr int NA = ncart(LA), NB = ncart(LB), NAB = NA * NB, LAB = LA + LB, H = nherm(LAB), L = LAB + LP;
  constexpr int NP = ncart(LP);
  constexpr bool TOP = LP <= 1 || PURE;
  extern __shared__ __align__(16) unsigned char e3_sm[];
  Eri3Shared<LA, LB, LP>& S = *reinterpret_cast<Eri3Shared<LA, LB, LP>*>(e3_sm);
  const int tid = threadIdx.x, lane = tid & 31;
  const int ip = blockIdx.x;
  const int a = P.pairs.sa[ip], b = P.pairs.sb[ip];
  load_boys<L>(S.boys, P.boysp);
  const double A[3] = {P.ox[a], P.oy[a], P.oz[a]}, B[3] = {P.ox[b], P.oy[b], P.oz[b]};
  __shared__ double cart[NAB];
  for (int i = tid; i < NAB; i += blockDim.x) cart[i] = 0.0;
  for (int e = P.ent.first[ip]; e < P.ent.first[ip + 1]; ++e) {
    const int nb = P.ent.np[e];
    __syncthreads();
    load_bra<LA, LB>(S.bra, entry_prims(P.ent, e), nb, A[0], A[1], A[2], B[0], B[1], B[2]);
    for (int ib = 0; ib < nb; ++ib) {
      const double* q = S.bra.prim[ib];
      double W[H];
#pragma unroll
      for (int h = 0; h < H; ++h) W[h] = 0.0;
      for (int s = tid; s < P.aux.count; s += blockDim.x) {
        const int sh = P.aux.shells[s];
        const int j0 = P.aux.prim_off[sh], nj = P.aux.nprim[sh];
        const double* cc = P.cc + P.aux_coff[sh];
        for (int k = j0; k < j0 + nj; ++k) {
          double R[nherm(L)];
          quartet_R<L>(q[0], __ldg(P.aux.p + k), q[4] * __ldg(P.aux.Kp + k), q[1] - __ldg(P.aux.x + k),
                       q[2] - __ldg(P.aux.y + k), q[3] - __ldg(P.aux.z + k), S.boys, R);
          const double h1 = -__ldg(P.aux.h + k);
          if constexpr (TOP) {
            const double hl = LP == 0 ? 1.0 : (LP == 1 ? h1 : (LP == 2 ? h1 * h1 : h1 * h1 * h1));
            static_for<NP>([&](auto aa) { shift_accumulate<LAB, LP, decltype(aa)::value>(W, R, hl * cc[decltype(aa)::value]); });
          } else {
#pragma unroll 1
            for (int c = 0; c < NP; ++c) {
              const int ce[3] = {c_herm.t[nherm(LP - 1) + c], c_herm.u[nherm(LP - 1) + c], c_herm.v[nherm(LP - 1) + c]};
              double ex[3][LP + 1];
#pragma unroll
              for (int x = 0; x < 3; ++x) {
#pragma unroll
                for (int t = 0; t <= LP; ++t) ex[x][t] = t == 0 ? (x == 0 ? cc[c] : 1.0) : 0.0;
#pragma unroll
                for (int t = 0; t < LP; ++t)
                  if (t < ce[x]) e1_raise<LP>(ex[x], 0.0, -h1);
              }
              ket_accumulate<LAB, LP>(W, R, ex[0], ex[1], ex[2], ce[0], ce[1], ce[2]);
            }
          }
        }
      }
#pragma unroll
      for (int h = 0; h < H; ++h) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) W[h] += __shfl_down_sync(0xffffffffu, W[h], o);
        if (lane == 0) S.red[tid >> 5][h] = W[h];
      }
      __syncthreads();
      for (int h = tid; h < H; h += blockDim.x) {
        double v = 0.0;
        for (int w = 0; w < (int)blockDim.x / 32; ++w) v += S.red[w][h];
        S.red[0][h] = v;
      }
      __syncthreads();
      for (int i = tid; i < NAB; i += blockDim.x)
        cart[i] += bra_component<LA, LB>(S.bra.M[LAB > 0 ? ib : 0], S.red[0], i);
      __syncthreads();
    }
  }
  // final functions, lower triangle
  const bool pa = LA >= 2 && P.obs_pure[a], pb = LB >= 2 && P.obs_pure[b];
  const int fa = pa ? 2 * LA + 1 : NA, fb = pb ? 2 * LB + 1 : NB;
  const int m0 = P.obs_foff[a], n0 = P.obs_foff[b];
  for (int i = tid; i < fa * fb; i += blockDim.x) {
    const int m = i / fb, q = i % fb;
    double v = 0.0;
    for (int i1 = pa ? 0 : m; i1 < (pa ? NA : m + 1); ++i1) {
      const double ta = pa ? P.sph[sph_off(LA) + m * NA + i1] : 1.0;
      for (int j1 = pb ? 0 : q; j1 < (pb ? NB : q + 1); ++j1)
        v += ta * (pb ? P.sph[sph_off(LB) + q * NB + j1] : 1.0) * cart[i1 * NB + j1];
    }
    const int X = m0 + m, Y = n0 + q;
    if (a == b && X < Y) continue;  // the same block holds its mirror image
    atomicAdd(P.J + (size_t)(X < Y ? X : Y) * P.n + (X < Y ? Y : X), v);
  }
}

template <int LA, int LB, int LP, bool PURE>
inline cudaError_t launch_eri3_class(const Eri3Params& P, bool j, cudaStream_t s) {
  const size_t sm = sizeof(Eri3Shared<LA, LB, LP>);
  const int iters = (P.aux.count + E3_THREADS - 1) / E3_THREADS;
  const int threads = ((P.aux.count + iters - 1) / iters + 31) / 32 * 32;
  if (j) return launch_smem(k_eri3_J<LA, LB, LP, PURE>, P.pairs.npair, threads, sm, sm, s, P);
  const int layers = e3_full(LA, LB, LP, PURE) ? 1 : e3_nfun(LP, PURE);
  // one block walks over all fitting shells of a pair unless that leaves the GPU short of blocks
  int z = 1;
  while (z < iters && (long long)P.nlist * layers * z < 8 * P.nsm) ++z;
  return launch_smem(k_eri3<LA, LB, LP, PURE>, dim3(P.nlist, layers, z), threads, sm, sm, s, P);
}
template <int LP, bool PURE>
inline cudaError_t launch_eri3_l(int pc, const Eri3Params& P, bool j, cudaStream_t s) {
  if (pc == 0) return launch_eri3_class<0, 0, LP, PURE>(P, j, s);
  if (pc == 1) return launch_eri3_class<1, 0, LP, PURE>(P, j, s);
  if (pc == 2) return launch_eri3_class<1, 1, LP, PURE>(P, j, s);
  if (pc == 3) return launch_eri3_class<2, 0, LP, PURE>(P, j, s);
  if (pc == 4) return launch_eri3_class<2, 1, LP, PURE>(P, j, s);
  if (pc == 5) return launch_eri3_class<2, 2, LP, PURE>(P, j, s);
  return cudaErrorInvalidValue;
}

// Group number of a fitting shell: s, p, pure d, Cartesian d, pure f, Cartesian f.
inline int aux_group_of(int l, int pure) { return l <= 1 ? l : 2 * l - (pure ? 2 : 1); }

// Coefficient of Hermite order t in x^i exp(-q x^2), h = 1/(2q), i <= 3.
__device__ __forceinline__ double centred_coef(int i, int t, double h) {
  if (t > i || ((i - t) & 1)) return 0.0;
  double v = (i == 3 && t == 1) ? 3.0 * h * h : (i == 2 && t == 0) ? h : 1.0;
  if (t == i)
    for (int k = 0; k < i; ++k) v *= h;
  return v;
}

struct Eri2Params {
  AuxView P, Q;     // two groups of fitting shells
  const double* sph;
  const double* boysp;
  int naux;
  int same;         // P and Q are one group: each unordered pair once
  double* V;        // naux x naux
};

// (P|Q) of two groups: block = shell P, lanes = shells Q.  A pair of pure, s or
// p shells needs only the Hermite integrals of the two top degrees.
constexpr int E2_THREADS = 64;
template <int LP, bool PP, int LQ, bool PQ>
__global__ void __launch_bounds__(E2_THREADS) k_eri2(const Eri2Params P) {
  constexpr int NP = ncart(LP), NQ = ncart(LQ), FP = e3_nfun(LP, PP), FQ = e3_nfun(LQ, PQ), L = LP + LQ;
  constexpr bool TOP = (LP <= 1 || PP) && (LQ <= 1 || PQ);
  __shared__ double boys[boysp_size(L)];
  __shared__ double sphP[FP * NP], sphQ[FQ * NQ];
  const int tid = threadIdx.x;
  load_boys<L, BOYSP_COEF_DF>(boys, P.boysp);
  for (int i = tid; i < FP * NP; i += E2_THREADS)
    sphP[i] = PP && LP > 1 ? P.sph[sph_off(LP) + i] : (i / NP == i % NP ? 1.0 : 0.0);
  for (int i = tid; i < FQ * NQ; i += E2_THREADS)
    sphQ[i] = PQ && LQ > 1 ? P.sph[sph_off(LQ) + i] : (i / NQ == i % NQ ? 1.0 : 0.0);
  __syncthreads();
  const int s = blockIdx.y * E2_THREADS + tid;
  if (s >= P.Q.count || (P.same && s > (int)blockIdx.x)) return;
  const int sP = P.P.shells[blockIdx.x], sQ = P.Q.shells[s];
  double A[NP][NQ];  // Cartesian block (its top-degree part)
#pragma unroll
  for (int i = 0; i < NP; ++i)
#pragma unroll
    for (int j = 0; j < NQ; ++j) A[i][j] = 0.0;
  for (int j = P.P.prim_off[sP]; j < P.P.prim_off[sP] + P.P.nprim[sP]; ++j)
    for (int k = P.Q.prim_off[sQ]; k < P.Q.prim_off[sQ] + P.Q.nprim[sQ]; ++k) {
      const double hp = __ldg(P.P.h + j), hq = __ldg(P.Q.h + k);
      double R[nherm(L)];
      quartet_R<L, BOYSP_COEF_DF>(__ldg(P.P.p + j), __ldg(P.Q.p + k), __ldg(P.P.Kp + j) * __ldg(P.Q.Kp + k),
                   __ldg(P.P.x + j) - __ldg(P.Q.x + k), __ldg(P.P.y + j) - __ldg(P.Q.y + k),
                   __ldg(P.P.z + j) - __ldg(P.Q.z + k), boys, R);
      if constexpr (TOP) {
        double hl = (LQ & 1) ? -1.0 : 1.0;
#pragma unroll
        for (int i = 0; i < LP; ++i) hl *= hp;
#pragma unroll
        for (int i = 0; i < LQ; ++i) hl *= hq;
        static_for<NP * NQ>([&](auto ab) {
          constexpr int i = decltype(ab)::value / NQ, b = decltype(ab)::value % NQ;
          A[i][b] += hl * R[hidx(cart_a(LP, i) + cart_a(LQ, b), cart_b(LP, i) + cart_b(LQ, b),
                                 cart_c(LP, i) + cart_c(LQ, b))];
        });
      } else {
        for (int m = 0; m < nherm(LP); ++m)
          for (int n = 0; n < nherm(LQ); ++n) {
            const int t = c_herm.t[n], u = c_herm.u[n], z = c_herm.v[n];
            const double r0 = R[hidx(t + c_herm.t[m], u + c_herm.u[m], z + c_herm.v[m])];
            const double r = ((t + u + z) & 1) ? -r0 : r0;
            for (int i = 0; i < NP; ++i) {
              int e[3] = {0, 0, 0};
              if (LP > 0) e[0] = c_herm.t[nherm(LP - 1) + i], e[1] = c_herm.u[nherm(LP - 1) + i], e[2] = c_herm.v[nherm(LP - 1) + i];
              const double cp = r * centred_coef(e[0], c_herm.t[m], hp) * centred_coef(e[1], c_herm.u[m], hp) *
                                centred_coef(e[2], c_herm.v[m], hp);
              if (cp == 0.0) continue;
              for (int b = 0; b < NQ; ++b) {
                int f[3] = {0, 0, 0};
                if (LQ > 0) f[0] = c_herm.t[nherm(LQ - 1) + b], f[1] = c_herm.u[nherm(LQ - 1) + b], f[2] = c_herm.v[nherm(LQ - 1) + b];
                A[i][b] += cp * centred_coef(f[0], t, hq) * centred_coef(f[1], u, hq) * centred_coef(f[2], z, hq);
              }
            }
          }
      }
    }
  const int p0 = P.P.foff[sP], q0 = P.Q.foff[sQ];
  double t[FP][NQ];
#pragma unroll
  for (int m = 0; m < FP; ++m)
#pragma unroll
    for (int b = 0; b < NQ; ++b) {
      t[m][b] = 0.0;
#pragma unroll
      for (int i = 0; i < NP; ++i) t[m][b] += sphP[m * NP + i] * A[i][b];
    }
#pragma unroll
  for (int m = 0; m < FP; ++m)
#pragma unroll
    for (int f = 0; f < FQ; ++f) {
      double v = 0.0;
#pragma unroll
      for (int b = 0; b < NQ; ++b) v += sphQ[f * NQ + b] * t[m][b];
      P.V[(size_t)(q0 + f) * P.naux + p0 + m] = v;
      P.V[(size_t)(p0 + m) * P.naux + q0 + f] = v;
    }
}

// launchers in df_cls_*.cu: pair class id, T (j false) or J (j true)
cudaError_t launch_eri3_s(int pair_class_id, const Eri3Params& P, bool j, cudaStream_t s);
cudaError_t launch_eri3_p(int pair_class_id, const Eri3Params& P, bool j, cudaStream_t s);
cudaError_t launch_eri3_d_pure(int pair_class_id, const Eri3Params& P, bool j, cudaStream_t s);
cudaError_t launch_eri3_d_cart(int pair_class_id, const Eri3Params& P, bool j, cudaStream_t s);
cudaError_t launch_eri3_f_pure(int pair_class_id, const Eri3Params& P, bool j, cudaStream_t s);
cudaError_t launch_eri3_f_cart(int pair_class_id, const Eri3Params& P, bool j, cudaStream_t s);
cudaError_t launch_eri2(int gP, int gQ, const Eri2Params& P, cudaStream_t s);  // groups gP >= gQ

}  // namespace m2
