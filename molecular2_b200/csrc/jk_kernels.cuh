// Device side of the integral-direct J/K build and the Schwarz bounds (FP64).
// Included by the per-class translation units jk_cls_*.cu and jk_direct.cu.
#pragma once
#include "launch.cuh"
#include "md.cuh"
#include "quartet.cuh"

namespace m2 {

struct PairView {
  const int* sa;
  const int* sb;
  const int* prim_off;
  const int* nprim;
  const double* Q;
  int npair;
};
struct PrimView {
  const double *p, *x, *y, *z, *K;
};
struct ShellView {
  const double *x, *y, *z;
  const int* coff;  // Cartesian function offset
};

// Hermite triples and Cartesian exponents by index, for run-time indices
// (tables cover totals up to 9).
struct HermTab {
  unsigned char t[nherm(9)], u[nherm(9)], v[nherm(9)];
};
__host__ __device__ constexpr HermTab make_herm_tab() {
  HermTab h{};
  int i = 0;
  for (int k = 0; k <= 9; ++k)
    for (int j = 0; j < ncart(k); ++j, ++i) {
      h.t[i] = (unsigned char)cart_a(k, j);
      h.u[i] = (unsigned char)cart_b(k, j);
      h.v[i] = (unsigned char)cart_c(k, j);
    }
  return h;
}
__constant__ constexpr HermTab c_herm = make_herm_tab();

struct JKParams {
  PairView bra, ket;
  EntryView bra_ent, ket_ent;
  int same_class;
  ShellView sh;
  const double* Dnorm;  // nshell x nshell (final-basis shell-block max norms)
  int nshell;
  const double* Dmax;   // device scalar
  int nden;             // densities digested per quartet: 1 (RHF), or the two spins of UHF (1 or 2)
  const double* Dc;     // Cartesian density, nc x nc (nden of them, dstride apart)
  int nc;
  double* Jc;           // raw accumulators (nden of each, dstride apart)
  double* Kc;
  size_t dstride;       // elements between consecutive densities / accumulators
  double precision, eps;  // eps: prim_eps(precision)
  const double* boysp;  // polynomial Boys tables, BOYSP_SIZE doubles per order
  unsigned long long* counter;
  unsigned long long* work;  // NULL or this class pair's [quartets, sum bra primitive pairs, sum primitive quartets]
  int kchunk;                // ket entries per block
  int bra0, bra_step;        // this rank's bra pairs: bra0, bra0 + bra_step, ...
};

// Pairs of a class are sorted by Schwarz bound Q descending and then, inside
// consecutive windows of PAIR_WINDOW pairs, by contraction length, so that
// the 32 kets of a warp have similar primitive counts.  The Q prefix of a
// threshold is therefore rounded up to a whole window; the per-ket screen
// drops the extra kets.  Every Q of a window is >= every Q of the next one,
// so a binary search lands inside the window holding the cut; window_up
// returns the end of the window containing index k (k itself included).
constexpr int PAIR_WINDOW = 256;
__device__ __forceinline__ int window_up(int k, int n) {
  return min(n, (k / PAIR_WINDOW + 1) * PAIR_WINDOW);
}

// number of kets in [0, n) whose Q >= thr (Q sorted descending)
__device__ __forceinline__ int q_prefix(const double* Q, int n, double thr) {
  int lo = 0, hi = n;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (__ldg(Q + mid) >= thr)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

__device__ __forceinline__ void atomic_add_f64(double* a, double v) {
  if (v != 0.0) atomicAdd(a, v);
}

// How a thread works on its quartet.  JK_FULL: all ket components at once, the
// ket s or p shell with an s shell.  JK_PP: one first-shell component of a pp
// ket per block layer (blockIdx.z), its three partners together.  JK_ONE: one
// ket component per layer.  The layers recompute the Hermite integrals R
// (nherm(L) of them, ~2 flops each) but leave the Hermite-space sums W and R in
// registers; a thread that holds a whole p or d quartet spills them.
enum { JK_FULL = 0, JK_PP = 1, JK_ONE = 2 };
__host__ __device__ constexpr int jk_mode(int la, int lb, int lc, int ld) {
  if (lc == 0) return JK_FULL;
  if (lc == 1 && ld == 0) return ncart(la) * ncart(lb) <= 9 ? JK_FULL : JK_ONE;
  if (lc == 1 && ld == 1 && ncart(la) * ncart(lb) <= 9) return JK_PP;
  return JK_ONE;
}
__host__ __device__ constexpr int jk_layers(int la, int lb, int lc, int ld) {
  return jk_mode(la, lb, lc, ld) == JK_FULL ? 1
         : jk_mode(la, lb, lc, ld) == JK_PP ? ncart(lc)
                                            : ncart(lc) * ncart(ld);
}
constexpr int JK_THREADS = 128;
constexpr int JK_LIST = 1024;      // ket entries screened and packed at a time
// Primitive quartets whose prefactor is below this in every lane of a warp are
// skipped.  The line follows the caller's threshold: an integral is its prefactor
// times the density and the expansions' |P - A|, 1/(2p), ... (up to four factors a
// side, above 1e3 in all for diffuse distant pairs), and nine decades below the
// threshold leave room for both.  precision = 0 skips nothing but exact zeros.
inline double prim_eps(double precision) { return precision < 1e-12 ? 1e-9 * precision : 1e-21; }

template <int LA, int LB>
struct JKShared {
  double boys[boysp_size(2 * (LA + LB))];  // no ket class is above the bra's
  BraShared<LA, LB> bra;
  double Dab[2][ncart(LA) * ncart(LB)];
  int list[JK_LIST + JK_THREADS];
  int n;
};
template <int LA, int LB>
__host__ __device__ constexpr size_t jk_smem(int nden) {
  return sizeof(JKShared<LA, LB>) + sizeof(double) * (size_t)nden * ncart(LA) * ncart(LB) * JK_THREADS + 16;
}

// Direct J/K of one class pair.  Block (x, y, z): bra entry x, ket entries
// [y kchunk, (y + 1) kchunk), component layer z.  The block first screens its
// kets and packs the survivors (density screening leaves 60 % of the lanes of
// a fixed ket-to-lane map busy on C20H42), then a thread takes one survivor at
// a time: Hermite sums W over the ket primitives for each bra primitive, bra
// transform from the tables in shared memory, digestion with FP64 atomics.
// J_ab is kept per thread in shared memory and reduced once per block.
// Two densities (UHF, UnrestrictedFock::formJKdirect,
// src/fockbuild.cpp:266-362) are digested from the same integrals; the screen
// uses the norms of their sum.
// Measured (one thread per contracted quartet with its 6 to 81 integrals in
// local memory -> this kernel): H2O/cc-pVDZ 18.0 -> 0.25 ms, (H2O)8/cc-pVDZ
// 44.3 -> 4.6 ms, C20H42/6-311G** 262 -> 45 ms.  Of that, 52 -> 44 ms came from
// fewer instructions per primitive (Boys function, reciprocal square root), the
// next primitive's loads issued ahead, and rounds of whole warps over the packed
// list.  Tried and slower on C20H42: entries of 16 primitives (56 for 52 ms),
// the bra's K rows summed in shared memory instead of by global atomics (54 for
// 44 ms), one block per bra over all kets (55 for 50 ms).
template <int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__(JK_THREADS) k_jk_direct(const JKParams P) {
  constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD), NAB = NA * NB;
  constexpr int LAB = LA + LB, LCD = LC + LD, L = LAB + LCD, HAB = nherm(LAB);
  constexpr int MODE = jk_mode(LA, LB, LC, LD);
  static_assert(LCD <= LAB, "the bra's Boys table covers the ket");
  constexpr int GC = MODE == JK_FULL ? NC : 1, GD = MODE == JK_ONE ? 1 : ND, G = GC * GD;
  extern __shared__ __align__(16) unsigned char jk_sm[];
  JKShared<LA, LB>& S = *reinterpret_cast<JKShared<LA, LB>*>(jk_sm);
  double* s_jab = reinterpret_cast<double*>(jk_sm + ((sizeof(JKShared<LA, LB>) + 15) & ~(size_t)15));

  const int eb = blockIdx.x;
  const int bra = P.bra_ent.pair[eb];
  if (bra % P.bra_step != P.bra0) return;
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

  unsigned long long cnt = 0, wb = 0, wq = 0;
  const int ns = P.nshell;
  const double* Dn = P.Dnorm;
  const double dab = Dn[a * ns + b];
  const bool count = blockIdx.z == 0 && P.bra_ent.first[bra] == eb;
  const int a0 = P.sh.coff[a], b0 = P.sh.coff[b], nc = P.nc;
  const int nb = P.bra_ent.np[eb];
  bool ready = false;

  // this layer's ket component (block-uniform)
  int ic0 = 0, id0 = 0, cx = 0, cy = 0, cz = 0, dx = 0, dy = 0, dz = 0;
  if constexpr (MODE == JK_PP) ic0 = blockIdx.z;
  if constexpr (MODE == JK_ONE) {
    ic0 = blockIdx.z / ND;
    id0 = blockIdx.z % ND;
    if constexpr (LD > 0) {
      dx = c_herm.t[nherm(LD - 1) + id0];
      dy = c_herm.u[nherm(LD - 1) + id0];
      dz = c_herm.v[nherm(LD - 1) + id0];
    }
  }
  if constexpr (MODE != JK_FULL && LC > 0) {
    cx = c_herm.t[nherm(LC - 1) + ic0];
    cy = c_herm.u[nherm(LC - 1) + ic0];
    cz = c_herm.v[nherm(LC - 1) + ic0];
  }

  int have = 0;  // survivors left over from the stretch before
  for (int l0 = start; l0 < end; l0 += JK_LIST) {
    // screen: max6(|D| blocks) Q_ab Q_cd >= precision
    const int got = pack_kets(l0, min(l0 + JK_LIST, end), have, S.list, &S.n, [&](int e) {
      const int kl = P.ket_ent.pair[e];
      const int c = P.ket.sa[kl], d = P.ket.sb[kl];
      double dn = fmax(fmax(dab, Dn[c * ns + d]), fmax(Dn[a * ns + c], Dn[a * ns + d]));
      dn = fmax(dn, fmax(Dn[b * ns + c], Dn[b * ns + d]));
      const bool pass = !(dn * Qab * P.ket.Q[kl] < P.precision);
      if (pass && count && P.ket_ent.first[kl] == e) {
        const int bnp = P.bra.nprim[bra];
        ++cnt;
        wb += bnp;
        wq += (unsigned long long)bnp * P.ket.nprim[kl];
      }
      return pass;
    });
    // whole rounds of the block's threads; the rest waits for the next stretch
    const int n = l0 + JK_LIST < end ? got / JK_THREADS * JK_THREADS : got;
    if (n == 0) {
      have = got;
      __syncthreads();
      continue;
    }
    if (!ready) {  // the bra's tables, once there are kets
      ready = true;
      load_boys<L>(S.boys, P.boysp);
      for (int i = tid; i < P.nden * NAB; i += JK_THREADS)
        S.Dab[i / NAB][i % NAB] =
            P.Dc[(i / NAB) * P.dstride + (size_t)(a0 + (i % NAB) / NB) * nc + b0 + (i % NAB) % NB];
      for (int i = 0; i < P.nden * NAB; ++i) s_jab[i * JK_THREADS + tid] = 0.0;
      load_bra<LA, LB>(S.bra, entry_prims(P.bra_ent, eb), nb, P.sh.x[a], P.sh.y[a], P.sh.z[a], P.sh.x[b],
                       P.sh.y[b], P.sh.z[b]);
    }
  for (int t0 = (tid >> 5) * 32; t0 < n; t0 += JK_THREADS) {
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
    double Cx = 0, Cy = 0, Cz = 0, Ex = 0, Ey = 0, Ez = 0;
    if constexpr (LC > 0) {
      Cx = P.sh.x[c];
      Cy = P.sh.y[c];
      Cz = P.sh.z[c];
    }
    if constexpr (LD > 0) {
      Ex = P.sh.x[d];
      Ey = P.sh.y[d];
      Ez = P.sh.z[d];
    }
    double v[NAB * G];  // [ab][c][d]
#pragma unroll
    for (int i = 0; i < NAB * G; ++i) v[i] = 0.0;
    for (int ib = 0; ib < nb; ++ib) {
      const double p = S.bra.prim[ib][0], Px = S.bra.prim[ib][1], Py = S.bra.prim[ib][2], Pz = S.bra.prim[ib][3];
      const double Kb = S.bra.prim[ib][4] * deg;
      double W[G][HAB];
#pragma unroll
      for (int g = 0; g < G; ++g)
#pragma unroll
        for (int h = 0; h < HAB; ++h) W[g][h] = 0.0;
      KetPrim next = load_ket<(LCD > 0)>(kp, 0);
      for (int k = 0; k < nkm; ++k) {
        const KetPrim kq = next;  // the next primitive's loads run behind this one's arithmetic
        next = load_ket<(LCD > 0)>(kp, min(k + 1, nk - 1));
        const double KK = k < nk ? Kb * kq.K : 0.0;
        if (!__any_sync(0xffffffffu, fabs(KK) > P.eps)) break;  // largest first: the rest is smaller
        const double Qx = kq.x, Qy = kq.y, Qz = kq.z;
        double R[nherm(L)];
        quartet_R<L>(p, kq.q, KK, Px - Qx, Py - Qy, Pz - Qz, S.boys, R);
        if constexpr (LCD == 0) {
#pragma unroll
          for (int h = 0; h < HAB; ++h) W[0][h] += R[h];
        } else if constexpr (MODE == JK_FULL) {  // ps
          const double h2 = kq.h;
          const double QC[3] = {Qx - Cx, Qy - Cy, Qz - Cz};
          static_for<3 * HAB>([&](auto gh) {
            constexpr int g = decltype(gh)::value / HAB, h = decltype(gh)::value % HAB;
            W[g][h] += QC[g] * R[h] - h2 * R[hidx(herm_t(h) + (g == 0), herm_u(h) + (g == 1), herm_v(h) + (g == 2))];
          });
        } else {
          const double h2 = kq.h;
          double e1[3][LCD + 1];
          const double QC[3] = {Qx - Cx, Qy - Cy, Qz - Cz}, QD[3] = {Qx - Ex, Qy - Ey, Qz - Ez};
          const int ce[3] = {cx, cy, cz}, de[3] = {dx, dy, dz};
#pragma unroll
          for (int x = 0; x < 3; ++x) {
            e1[x][0] = 1.0;
#pragma unroll
            for (int t = 1; t <= LCD; ++t) e1[x][t] = 0.0;
#pragma unroll
            for (int s = 0; s < LC; ++s)
              if (s < ce[x]) e1_raise<LCD>(e1[x], QC[x], h2);
            if constexpr (MODE == JK_ONE)
#pragma unroll
              for (int s = 0; s < LD; ++s)
                if (s < de[x]) e1_raise<LCD>(e1[x], QD[x], h2);
          }
          if constexpr (MODE == JK_ONE) {
            ket_accumulate<LAB, LCD>(W[0], R, e1[0], e1[1], e1[2], cx + dx, cy + dy, cz + dz);
          } else {
#pragma unroll
            for (int g = 0; g < GD; ++g) {
              double r[LCD + 1];
#pragma unroll
              for (int t = 0; t <= LCD; ++t) r[t] = e1[g][t];
              e1_raise<LCD>(r, QD[g], h2);
              ket_accumulate<LAB, LCD>(W[g], R, g == 0 ? r : e1[0], g == 1 ? r : e1[1], g == 2 ? r : e1[2],
                                       cx + (g == 0), cy + (g == 1), cz + (g == 2));
            }
          }
        }
      }
#pragma unroll
      for (int g = 0; g < G; ++g) bra_transform<LA, LB, G>(S.bra.M[LAB > 0 ? ib : 0], W[g], v + g);
    }
    // digestion: 6 updates per integral (src/fockbuild.cpp:121-153)
    if (active) {
      const int c0 = P.sh.coff[c] + ic0, d0 = P.sh.coff[d] + id0;
#pragma unroll 1
      for (int dd = 0; dd < P.nden; ++dd) {
        const double* __restrict__ Dc = P.Dc + dd * P.dstride;
        const double* __restrict__ Dra = Dc + (size_t)a0 * nc;  // the bra's rows
        const double* __restrict__ Drb = Dc + (size_t)b0 * nc;
        double* __restrict__ Jd = P.Jc + dd * P.dstride;
        double* __restrict__ Kra = P.Kc + dd * P.dstride + (size_t)a0 * nc;
        double* __restrict__ Krb = P.Kc + dd * P.dstride + (size_t)b0 * nc;
        double* jab = s_jab + (size_t)dd * NAB * JK_THREADS + tid;
        const double* Dab = S.Dab[dd];
        double Dcd[G];
#pragma unroll
        for (int g = 0; g < G; ++g) Dcd[g] = __ldg(Dc + (size_t)(c0 + g / GD) * nc + d0 + g % GD);
#pragma unroll
        for (int i = 0; i < NAB; ++i) {
          double s = 0.0;
#pragma unroll
          for (int g = 0; g < G; ++g) s += Dcd[g] * v[i * G + g];
          jab[i * JK_THREADS] += s;
        }
#pragma unroll
        for (int g = 0; g < G; ++g) {
          double s = 0.0;
#pragma unroll
          for (int i = 0; i < NAB; ++i) s += Dab[i] * v[i * G + g];
          atomicAdd(Jd + (size_t)(c0 + g / GD) * nc + d0 + g % GD, s);
        }
        // K_ac, K_bc from D_bd, D_ad; K_ad, K_bd from D_bc, D_ac
#pragma unroll
        for (int side = 0; side < 2; ++side) {
          const int r0 = side ? d0 : c0, q0 = side ? c0 : d0;
          constexpr int GX[2] = {GC, GD};
          const int nr = GX[side], nq = GX[1 - side];
#pragma unroll
          for (int r = 0; r < nr; ++r) {
            double ka[NA], kb[NB];
#pragma unroll
            for (int i = 0; i < NA; ++i) ka[i] = 0.0;
#pragma unroll
            for (int j = 0; j < NB; ++j) kb[j] = 0.0;
#pragma unroll
            for (int q = 0; q < nq; ++q) {
              const int g = side ? q * GD + r : r * GD + q;
              double Da[NA], Db[NB];
#pragma unroll
              for (int i = 0; i < NA; ++i) Da[i] = __ldg(Dra + i * nc + q0 + q);
#pragma unroll
              for (int j = 0; j < NB; ++j) Db[j] = __ldg(Drb + j * nc + q0 + q);
#pragma unroll
              for (int i = 0; i < NA; ++i)
#pragma unroll
                for (int j = 0; j < NB; ++j) {
                  ka[i] += Db[j] * v[(i * NB + j) * G + g];
                  kb[j] += Da[i] * v[(i * NB + j) * G + g];
                }
            }
#pragma unroll
            for (int i = 0; i < NA; ++i) atomicAdd(Kra + i * nc + r0 + r, ka[i]);
#pragma unroll
            for (int j = 0; j < NB; ++j) atomicAdd(Krb + j * nc + r0 + r, kb[j]);
          }
        }
      }
    }
    }
    __syncthreads();  // every warp is through with the list
    have = got - n;
    const int keep = tid < have ? S.list[n + tid] : 0;
    __syncthreads();
    if (tid < have) S.list[tid] = keep;
  }
  if (!ready) return;
  __syncthreads();
  // J_ab: one warp per component
  for (int i = tid >> 5; i < P.nden * NAB; i += JK_THREADS / 32) {
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < JK_THREADS / 32; ++w) s += s_jab[i * JK_THREADS + w * 32 + lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0)
      atomic_add_f64(P.Jc + (i / NAB) * P.dstride + (size_t)(a0 + (i % NAB) / NB) * nc + b0 + (i % NAB) % NB, s);
  }
  if (blockIdx.z != 0) return;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    cnt += __shfl_down_sync(0xffffffffu, cnt, o);
    wb += __shfl_down_sync(0xffffffffu, wb, o);
    wq += __shfl_down_sync(0xffffffffu, wq, o);
  }
  if (lane == 0 && cnt) {
    atomicAdd(P.counter, cnt);
    if (P.work) {
      atomicAdd(P.work, cnt);
      atomicAdd(P.work + 1, wb);
      atomicAdd(P.work + 2, wq);
    }
  }
}

template <int LA, int LB, int LC, int LD>
inline cudaError_t launch_jk_class(const JKParams& P, dim3 grid, cudaStream_t s) {
  static_assert(jk_smem<LA, LB>(2) <= SMEM_BLOCK_MAX, "shared memory of two densities");
  grid.z = jk_layers(LA, LB, LC, LD);
  return launch_smem(k_jk_direct<LA, LB, LC, LD>, grid, JK_THREADS, jk_smem<LA, LB>(P.nden), jk_smem<LA, LB>(2), s, P);
}

// Schwarz bound of each pair of one class: sqrt(max diag (ab|ab)) over the
// final (pure or Cartesian) functions (compute_schwarz_ints, src/integrals.cpp:472-513).
struct SchwarzParams {
  PairView pairs;
  PrimView pp;
  ShellView sh;
  const int* l;
  const int* pure;
  const double* sph;
  const double* boysp;
  double* Qout;
};

// One block per pair.  The Hermite expansions of the final functions' products
// are formed for SCHWARZ_PRIMS primitives at a time, a thread takes primitive
// quartets of one function pair: one thread per pair walked up to 6,561 of them
// and the whole (ab|ab) block (creating the engine of (H2O)8: 32 ms, now 3.5 ms).
// A thread keeps its function pair over the whole block and the partial sums are
// added in a fixed order, so that the bounds are the same to the last bit in
// every run: the ranks of a partitioned build (jk_direct_set_partition) each sort
// their class lists by them and must get the same order, also where pairs have
// equal bounds by symmetry.
constexpr int SCHWARZ_THREADS = 128;
constexpr int SCHWARZ_PRIMS = 8;

template <int LA, int LB>
struct SchwarzShared {
  static constexpr int NF = ncart(LA) * ncart(LB), H = nherm(LA + LB);
  double boys[boysp_size(2 * (LA + LB))];
  double prim[2][SCHWARZ_PRIMS][5];      // p, P, K'
  double E[SCHWARZ_PRIMS][3][e1_size(LA, LB)];
  double M[2][SCHWARZ_PRIMS][NF * H];    // [function pair][h]
  double part[SCHWARZ_THREADS];
};

template <int LA, int LB>
__global__ void __launch_bounds__(SCHWARZ_THREADS, 2) k_schwarz(const SchwarzParams P) {
  constexpr int NA = ncart(LA), NB = ncart(LB), H = nherm(LA + LB), L2 = 2 * (LA + LB);
  extern __shared__ __align__(16) unsigned char sch_sm[];
  SchwarzShared<LA, LB>& S = *reinterpret_cast<SchwarzShared<LA, LB>*>(sch_sm);
  const int ip = blockIdx.x, tid = threadIdx.x;
  const int a = P.pairs.sa[ip], b = P.pairs.sb[ip];
  const int p0 = P.pairs.prim_off[ip], np = P.pairs.nprim[ip];
  const double A[3] = {P.sh.x[a], P.sh.y[a], P.sh.z[a]}, B[3] = {P.sh.x[b], P.sh.y[b], P.sh.z[b]};
  const int pa = P.pure[a], pb = P.pure[b];
  const int ma = pa ? 2 * LA + 1 : NA, mb = pb ? 2 * LB + 1 : NB, nf = ma * mb;
  load_boys<L2>(S.boys, P.boysp);
  // threads of a function pair, and this thread's
  const int ng = SCHWARZ_THREADS / nf, f = tid % nf, group = tid / nf;
  double diag = 0.0;

  auto load = [&](int side, int k0, int n) {
    __syncthreads();
    for (int i = tid; i < n * 5; i += SCHWARZ_THREADS) {
      const int k = p0 + k0 + i / 5, f = i % 5;
      S.prim[side][i / 5][f] = f == 0   ? P.pp.p[k]
                               : f == 1 ? P.pp.x[k]
                               : f == 2 ? P.pp.y[k]
                               : f == 3 ? P.pp.z[k]
                                        : P.pp.K[k] * SQRT_PI25X2() / P.pp.p[k];
    }
    for (int i = tid; i < n * 3; i += SCHWARZ_THREADS) {
      const int k = p0 + k0 + i / 3, x = i % 3;
      const double X = x == 0 ? P.pp.x[k] : (x == 1 ? P.pp.y[k] : P.pp.z[k]);
      E1<LA, LB> e;
      md_E1<LA, LB>(X - A[x], X - B[x], 0.5 / P.pp.p[k], e);
#pragma unroll
      for (int u = 0; u <= LA; ++u)
#pragma unroll
        for (int v = 0; v <= LB; ++v)
#pragma unroll
          for (int t = 0; t <= LA + LB; ++t) S.E[i / 3][x][e1_pos(LA, LB, u, v, t)] = e.e[u][v][t];
    }
    __syncthreads();
    for (int i = tid; i < n * nf * H; i += SCHWARZ_THREADS) {
      const int k = i / (nf * H), f = (i / H) % nf, h = i % H, mu = f / mb, nu = f % mb;
      const int t = c_herm.t[h], u = c_herm.u[h], v = c_herm.v[h];
      double s = 0.0;
      for (int i1 = pa ? 0 : mu; i1 < (pa ? NA : mu + 1); ++i1) {
        const double ta = pa ? P.sph[sph_off(LA) + mu * NA + i1] : 1.0;
        const int ha = LA > 0 ? nherm(LA - 1) + i1 : 0;
        for (int j1 = pb ? 0 : nu; j1 < (pb ? NB : nu + 1); ++j1) {
          const double tb = pb ? P.sph[sph_off(LB) + nu * NB + j1] : 1.0;
          if (ta == 0.0 || tb == 0.0) continue;
          const int hb = LB > 0 ? nherm(LB - 1) + j1 : 0;
          s += ta * tb * S.E[k][0][e1_pos(LA, LB, c_herm.t[ha], c_herm.t[hb], t)] *
               S.E[k][1][e1_pos(LA, LB, c_herm.u[ha], c_herm.u[hb], u)] *
               S.E[k][2][e1_pos(LA, LB, c_herm.v[ha], c_herm.v[hb], v)];
        }
      }
      S.M[side][k][f * H + h] = s;
    }
    __syncthreads();
  };

  for (int k0 = 0; k0 < np; k0 += SCHWARZ_PRIMS) {
    const int nb = min(SCHWARZ_PRIMS, np - k0);
    load(0, k0, nb);
    for (int k1 = k0; k1 < np; k1 += SCHWARZ_PRIMS) {
      const int nk = min(SCHWARZ_PRIMS, np - k1);
      if (k1 != k0) load(1, k1, nk);
      const int ks = k1 != k0 ? 1 : 0;
      const double w = k1 != k0 ? 2.0 : 1.0;  // both orders of two primitive ranges
      for (int it = group < ng ? group : nb * nk; it < nb * nk; it += ng) {
        const int ib = it % nb, ik = it / nb;
        const double* pb_ = S.prim[0][ib];
        const double* pk_ = S.prim[ks][ik];
        double R[nherm(L2)];
        quartet_R<L2>(pb_[0], pk_[0], w * pb_[4] * pk_[4], pb_[1] - pk_[1], pb_[2] - pk_[2], pb_[3] - pk_[3], S.boys,
                      R);
        const double* Mb = S.M[0][ib] + f * H;
        const double* Mk = S.M[ks][ik] + f * H;
        double acc = 0.0;
        static_for<H>([&](auto gg) {
          constexpr int g = decltype(gg)::value;
          double s = 0.0;
          static_for<H>([&](auto hh) {
            constexpr int h = decltype(hh)::value;
            s += Mb[h] * R[hidx(herm_t(h) + herm_t(g), herm_u(h) + herm_u(g), herm_v(h) + herm_v(g))];
          });
          acc += ((herm_t(g) + herm_u(g) + herm_v(g)) & 1) ? -Mk[g] * s : Mk[g] * s;
        });
        diag += acc;
      }
    }
  }
  S.part[tid] = diag;
  __syncthreads();
  if (tid == 0) {
    double m = 0.0;
    for (int k = 0; k < nf; ++k) {
      double d = 0.0;
      for (int g = 0; g < ng; ++g) d += S.part[g * nf + k];
      m = fmax(m, fabs(d));
    }
    P.Qout[ip] = sqrt(m);
  }
}

template <int LA, int LB>
inline cudaError_t launch_schwarz_class(const SchwarzParams& P, cudaStream_t s) {
  const size_t sm = sizeof(SchwarzShared<LA, LB>);
  return launch_smem(k_schwarz<LA, LB>, P.pairs.npair, SCHWARZ_THREADS, sm, sm, s, P);
}

struct PairClassDev;
PairView view(const PairClassDev& c);

EntryView entry_view(const PairClassDev& c);

// per-translation-unit launchers (jk_cls_*.cu); A, B are pair-class ids
cudaError_t launch_jk_bra_s(int A, int B, const JKParams& P, dim3 grid, cudaStream_t s);   // A in {0,1,2}
cudaError_t launch_jk_bra_ds(int B, const JKParams& P, dim3 grid, cudaStream_t s);         // A = 3
cudaError_t launch_jk_bra_dp(int B, const JKParams& P, dim3 grid, cudaStream_t s);         // A = 4
cudaError_t launch_jk_bra_dd_lo(int B, const JKParams& P, dim3 grid, cudaStream_t s);      // A = 5, B < 4
cudaError_t launch_jk_bra_dd_hi(int B, const JKParams& P, dim3 grid, cudaStream_t s);      // A = 5, B >= 4
cudaError_t launch_schwarz(int la, int lb, const SchwarzParams& P, cudaStream_t s);  // schwarz.cu

}  // namespace m2
