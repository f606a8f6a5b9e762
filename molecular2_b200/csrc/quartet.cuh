// Device building blocks of the quartet kernels: pair entries, Boys function,
// Hermite integrals in registers and the bra tables a block shares.
//
// A shell pair is kept as one or more ENTRIES of at most ENTRY_PRIMS primitive
// pairs (largest prefactor first), and a kernel works on pairs of entries.  The
// integrals of a quartet are sums over its entry pairs and every consumer is
// linear in them, so no entry pair waits for another: a 9 x 9 contraction no
// longer makes one thread walk 6,561 primitive quartets, and the lanes of a
// warp, which hold different kets, run loops of nearly equal length.  The
// primitives of 32 consecutive entries are stored field by field with the
// entry index fastest, so that a warp reads a field of its 32 kets in two
// 128-byte lines (a gather of 8-byte words costs ten L1 cycles instead).
#pragma once
#include <type_traits>
#include <utility>

#include "md.cuh"

namespace m2 {

// f(integral_constant 0), ..., f(integral_constant N - 1): every index is a
// constant expression, so arrays indexed with it stay in registers (with plain
// unrolled loops the compiler left R in local memory).
template <class F, int... I>
__device__ __forceinline__ void static_for_impl(F&& f, std::integer_sequence<int, I...>) {
  (f(std::integral_constant<int, I>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void static_for(F&& f) {
  static_for_impl(f, std::make_integer_sequence<int, N>{});
}
// exponents of Hermite index h
__host__ __device__ constexpr int herm_k(int h) {
  int k = 0;
  while (nherm(k) <= h) ++k;
  return k;
}
__host__ __device__ constexpr int herm_t(int h) { return cart_a(herm_k(h), h - nherm(herm_k(h) - 1)); }
__host__ __device__ constexpr int herm_u(int h) { return cart_b(herm_k(h), h - nherm(herm_k(h) - 1)); }
__host__ __device__ constexpr int herm_v(int h) { return cart_c(herm_k(h), h - nherm(herm_k(h) - 1)); }

constexpr int ENTRY_PRIMS = 8;   // primitive pairs per entry
constexpr int ENTRY_FIELDS = 7;  // p, Px, Py, Pz, K sqrt(2 pi^(5/2)) / p, 1/(2p), exponent of the first shell
__host__ __device__ constexpr double PI25X2() { return 34.986836655249725; }          // 2 pi^(5/2)
__host__ __device__ constexpr double SQRT_PI25X2() { return 5.914967172795612; }      // its square root

struct EntryView {
  const int* pair;        // pair index in the class list (Schwarz-sorted)
  const int* np;          // primitive pairs of the entry
  const int* first;       // [npair + 1] first entry of each pair
  const long long* goff;  // offset of each group of 32 entries in prim
  const double* prim;
  int nent;
};
__device__ __forceinline__ const double* entry_prims(const EntryView& v, int e) {
  return v.prim + __ldg(v.goff + (e >> 5)) + (e & 31);
}
__device__ __forceinline__ double entry_field(const double* base, int k, int f) {
  return __ldg(base + (k * ENTRY_FIELDS + f) * 32);
}

// One primitive of a ket entry.
struct KetPrim {
  double q, x, y, z, K, h;
};
template <bool H>
__device__ __forceinline__ KetPrim load_ket(const double* base, int k) {
  const double* b = base + k * (ENTRY_FIELDS * 32);
  KetPrim r;
  r.K = __ldg(b + 4 * 32);
  r.q = __ldg(b);
  r.x = __ldg(b + 32);
  r.y = __ldg(b + 2 * 32);
  r.z = __ldg(b + 3 * 32);
  r.h = H ? __ldg(b + 5 * 32) : 0.0;
  return r;
}

// Appends the ket entries e in [start, end) with pass(e) to the `have` entries of
// list; returns the new number.  All threads of the block call this (n_shared: a
// shared counter); a barrier must lie between the last use of list or n_shared
// and the call.
template <class Pass>
__device__ __forceinline__ int pack_kets(int start, int end, int have, int* list, int* n_shared, Pass&& pass) {
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) *n_shared = have;
  __syncthreads();
  for (int e0 = start; e0 < end; e0 += blockDim.x) {
    const int e = e0 + threadIdx.x;
    const bool ok = e < end && pass(e);
    const unsigned m = __ballot_sync(0xffffffffu, ok);
    int pos = 0;
    if (lane == 0 && m) pos = atomicAdd(n_shared, __popc(m));
    pos = __shfl_sync(0xffffffffu, pos, 0) + __popc(m & ((1u << lane) - 1));
    if (ok) list[pos] = e;
  }
  __syncthreads();
  return *n_shared;
}

// ---------------------------------------------------------------- Boys
// F_M by a degree-9 polynomial in T - centre on intervals of width 3/8 centred
// on its multiples, up to T = 36 + 3M; e^{-T} from a table at the centres times
// a degree-9 polynomial; then downward recursion
// F_m = (2T F_{m+1} + e^{-T})/(2m+1).  From 36 + 3M on, F_m is its leading
// asymptotic term (what that drops is below 3e-17 of F_m).
// The table of one order (a row: 10 coefficients, e^{-centre}; 11 words, so that
// rows start in different banks) is staged in shared memory: eleven 8-byte reads,
// against seven L1 gathers and a call of exp for a Taylor table.  A kernel with
// exp() in both branches of the asymptotic test and the library's rsqrt ran 280
// instructions per (ps|ss) primitive quartet, 85 of them FP64.  Both polynomials
// interpolate at Chebyshev nodes; what they leave is below 2e-17 of F_M and 4e-17
// of e^{-T}.  Largest relative error in double arithmetic, of F_M below 36 + 3M:
// 2.2e-16 for every M (a Taylor table of 7 terms and step 1/20: 2.4e-16 at M = 0,
// 7.7e-16 at 4, 1.6e-15 at 9; nine coefficients: 6e-16 at 1, 2e-15 at 9); of all
// F_m from there: 3.8e-16 at M = 1, 8.5e-16 at 4, 1.6e-15 at 9.  There the orders
// are products of their own: downward recursion for both ranges gave 1.0e-15 at
// M = 4 (direct builds of C20H42 and H2O 44.6 and 0.250 ms with it, 44.9 and 0.252
// so, 44.4 and 0.247 with nine coefficients).  Even and odd coefficients side by side,
// a shorter chain of more operations, took 45.3 ms and 14.05 for the (H2O)8 gradient's
// 13.5.
//
// The three- and two-index integrals (k_eri3, k_eri2) keep nine coefficients and
// the asymptotic value of F_M carried down: the fitted tensor made of them is split
// into BF16, and a last bit of B that rounds the other way is a step of 2^-17 of
// its element there.  With ten coefficients J and K of a split-BF16 build move by
// 1e-9 to 3e-9, at the same error against 64 bits (4.1e-6), and stored results of
// such builds would no longer be met; FP64 results of the fitted builds carry the
// metric's condition number times eps, some 1e-12, either way.
constexpr double BOYSP_WIDTH = 0.375;
constexpr int BOYSP_COEF = 10, BOYSP_COEF_DF = 9;
constexpr int BOYSP_ROW = BOYSP_COEF + 1;
constexpr int BOYSP_MMAX = 9;   // orders 0..9
constexpr double boysp_tmax(int m) { return 36.0 + 3.0 * m; }
constexpr int boysp_rows(int m) { return (int)(boysp_tmax(m) / BOYSP_WIDTH + 0.5) + 1; }
constexpr int boysp_size(int m) { return boysp_rows(m) * BOYSP_ROW; }  // table of order m
constexpr int BOYSP_ROWS = boysp_rows(BOYSP_MMAX);
constexpr int BOYSP_SIZE = boysp_size(BOYSP_MMAX);                     // distance of the orders' tables
constexpr int BOYSP_SET = (BOYSP_MMAX + 1) * BOYSP_SIZE;               // ten coefficients, then nine
// Gamma(m + 1/2) / 2
__host__ __device__ constexpr double boys_gamma(int m) {
  constexpr double g[BOYSP_MMAX + 1] = {0.886226925452758,  0.443113462726379,  0.6646701940895685, 1.6616754852239213,
                                        5.815864198283724,  26.17138889227676,  143.94263890752217, 935.6271528988942,
                                        7017.2036467417065, 59646.230997304505};
  return g[m];
}

// The table of order M to shared memory; a barrier must follow.
template <int M, int NC = BOYSP_COEF>
__device__ __forceinline__ void load_boys(double* dst, const double* __restrict__ all) {
  const double* src = all + (NC == BOYSP_COEF ? 0 : BOYSP_SET) + (size_t)M * BOYSP_SIZE;
  for (int i = threadIdx.x; i < boysp_size(M); i += blockDim.x) dst[i] = __ldg(src + i);
}

// x^{-1/2} for x well inside the range of float: the single-precision estimate y
// times the binomial series of (1 - h)^{-1/2}, h = 1 - x y^2, to its second order
// (relative error e -> 5/2 e^3, e < 2^-21).
__device__ __forceinline__ double rsqrt_pos(double x) {
  const double y = (double)rsqrtf((float)x);
  const double h = 1.0 - x * y * y;
  return y + y * h * (0.5 + 0.375 * h);
}

// Row of the interval that holds T and T's distance d from its centre.
__device__ __forceinline__ const double* boys_row(double T, const double* tab, double& d) {
  // nearest multiple of the width, by the rounding of an addition to 1.5 2^52
  const double u = T * (1.0 / BOYSP_WIDTH) + 6755399441055744.0;
  d = T - (u - 6755399441055744.0) * BOYSP_WIDTH;
  return tab + __double2loint(u) * BOYSP_ROW;
}
template <int NC>
__device__ __forceinline__ double boys_horner(const double* c, double d) {
  double acc = c[NC - 1];
#pragma unroll
  for (int j = NC - 2; j >= 0; --j) acc = acc * d + c[j];
  return acc;
}
__device__ __forceinline__ double exp_minus(double d) {  // e^{-d}, |d| <= 3/16
  double x = -2.7579345743837904673e-6;
  x = x * d + 2.4825818086831339934e-5;
  x = x * d - 1.9841263064743021626e-4;
  x = x * d + 1.3888881434054876645e-3;
  x = x * d - 8.3333333341842252384e-3;
  x = x * d + 4.1666666676027388464e-2;
  x = x * d - 1.6666666666666292731e-1;
  x = x * d + 0.49999999999995886287;
  x = x * d - 1.0;
  return x * d + 1.0;
}
template <int M>
__device__ __forceinline__ void boys_down(double T, double e, double* F) {
  const double T2 = 2.0 * T;
#pragma unroll
  for (int m = M - 1; m >= 0; --m) F[m] = (T2 * F[m + 1] + e) * (1.0 / (2 * m + 1));
}

template <int M, int NC = BOYSP_COEF>
__device__ __forceinline__ void boys_poly(double T, const double* tab, double* F) {
  static_assert(M <= BOYSP_MMAX, "Boys order too high");
  static_assert(NC == BOYSP_COEF || NC == BOYSP_COEF_DF, "no such table");
  double d;
  if constexpr (NC == BOYSP_COEF) {
    if (T < boysp_tmax(M)) {
      const double* c = boys_row(T, tab, d);
      F[M] = boys_horner<NC>(c, d);
      if constexpr (M > 0) boys_down<M>(T, exp_minus(d) * c[NC], F);
    } else {  // Gamma(m + 1/2)/2 T^{-m-1/2}
      const double r = rsqrt_pos(T);
      double f = r, r2 = r * r;
      r2 = r2 + r2 * (1.0 - T * r2);  // r's rounding would be in every factor
#pragma unroll
      for (int m = 0; m <= M; ++m) {
        F[m] = boys_gamma(m) * f;
        f *= r2;
      }
    }
  } else {
    double e = 0.0;
    if (T < boysp_tmax(M)) {
      const double* c = boys_row(T, tab, d);
      F[M] = boys_horner<NC>(c, d);
      if constexpr (M > 0) e = exp_minus(d) * c[NC];
    } else {
      const double r = rsqrt_pos(T), r2 = r * r;
      double f = 0.886226925452758014 * r;
#pragma unroll
      for (int m = 0; m < M; ++m) f *= (m + 0.5) * r2;
      F[M] = f;
    }
    if constexpr (M > 0) boys_down<M>(T, e, F);
  }
}

// scale R_tuv (t + u + v <= L) for the reduced exponent a and distance (X, Y, Z).
template <int L, int NC = BOYSP_COEF>
__device__ __forceinline__ void hermite_R(double a, double scale, double X, double Y, double Z, const double* tab,
                                          double* R) {
  double F[L + 1];
  boys_poly<L, NC>(a * (X * X + Y * Y + Z * Z), tab, F);
  const double m2a = -2.0 * a;
  double pw = scale;
#pragma unroll
  for (int n = 0; n <= L; ++n) {
    F[n] *= pw;
    pw *= m2a;
  }
  R[0] = F[L];
  static_for<L>([&](auto step) {
    constexpr int n = L - 1 - decltype(step)::value;
    static_for<nherm(L - n) - 1>([&](auto rev) {  // highest total first: in place
      constexpr int h = nherm(L - n) - 1 - decltype(rev)::value;
      constexpr int t = herm_t(h), u = herm_u(h), v = herm_v(h);
      double val;
      if constexpr (t > 0) {
        val = X * R[hidx(t - 1, u, v)];
        if constexpr (t > 1) val += (t - 1) * R[hidx(t - 2, u, v)];
      } else if constexpr (u > 0) {
        val = Y * R[hidx(t, u - 1, v)];
        if constexpr (u > 1) val += (u - 1) * R[hidx(t, u - 2, v)];
      } else {
        val = Z * R[hidx(t, u, v - 1)];
        if constexpr (v > 1) val += (v - 1) * R[hidx(t, u, v - 2)];
      }
      R[h] = val;
    });
    R[0] = F[n];
  });
}
// The same for a primitive quartet with exponents p, q and prefactors KK =
// K'_ab K'_cd: prefactor and reduced exponent from one reciprocal square root.
template <int L, int NC = BOYSP_COEF>
__device__ __forceinline__ void quartet_R(double p, double q, double KK, double X, double Y, double Z,
                                          const double* tab, double* R) {
  const double r = rsqrt_pos(p + q);
  hermite_R<L, NC>(p * q * r * r, KK * r, X, Y, Z, tab, R);
}

// ---------------------------------------------------------------- bra tables
// Hermite expansion of the Cartesian products of one primitive pair as a list
// of its non-zero terms, component by component, (t, u, v) in loop order.
__host__ __device__ constexpr int nterms(int la, int lb) {
  int n = 0;
  for (int i = 0; i < ncart(la); ++i)
    for (int j = 0; j < ncart(lb); ++j)
      n += (cart_a(la, i) + cart_a(lb, j) + 1) * (cart_b(la, i) + cart_b(lb, j) + 1) *
           (cart_c(la, i) + cart_c(lb, j) + 1);
  return n;
}
// position of E^{ij}_t in the one-direction table of (la, lb)
__host__ __device__ constexpr int e1_pos(int la, int lb, int i, int j, int t) {
  return (i * (lb + 1) + j) * (la + lb + 1) + t;
}
__host__ __device__ constexpr int e1_size(int la, int lb) { return (la + 1) * (lb + 1) * (la + lb + 1); }

template <int LA, int LB>
struct TermTab {
  unsigned char x[nterms(LA, LB)], y[nterms(LA, LB)], z[nterms(LA, LB)];  // e1_pos of the three factors
  short first[ncart(LA) * ncart(LB) + 1];                                 // first term of each component
};
template <int LA, int LB>
__host__ __device__ constexpr TermTab<LA, LB> make_terms() {
  TermTab<LA, LB> T{};
  int n = 0;
  for (int i = 0; i < ncart(LA); ++i)
    for (int j = 0; j < ncart(LB); ++j) {
      const int ax = cart_a(LA, i), ay = cart_b(LA, i), az = cart_c(LA, i);
      const int bx = cart_a(LB, j), by = cart_b(LB, j), bz = cart_c(LB, j);
      T.first[i * ncart(LB) + j] = (short)n;
      for (int t = 0; t <= ax + bx; ++t)
        for (int u = 0; u <= ay + by; ++u)
          for (int v = 0; v <= az + bz; ++v, ++n) {
            T.x[n] = (unsigned char)e1_pos(LA, LB, ax, bx, t);
            T.y[n] = (unsigned char)e1_pos(LA, LB, ay, by, u);
            T.z[n] = (unsigned char)e1_pos(LA, LB, az, bz, v);
          }
    }
  T.first[ncart(LA) * ncart(LB)] = (short)n;
  return T;
}
__constant__ constexpr TermTab<0, 0> c_terms00 = make_terms<0, 0>();
__constant__ constexpr TermTab<1, 0> c_terms10 = make_terms<1, 0>();
__constant__ constexpr TermTab<1, 1> c_terms11 = make_terms<1, 1>();
__constant__ constexpr TermTab<2, 0> c_terms20 = make_terms<2, 0>();
__constant__ constexpr TermTab<2, 1> c_terms21 = make_terms<2, 1>();
__constant__ constexpr TermTab<2, 2> c_terms22 = make_terms<2, 2>();
template <int LA, int LB>
__device__ __forceinline__ const TermTab<LA, LB>& term_tab() {
  if constexpr (LA == 0) return c_terms00;
  else if constexpr (LA == 1 && LB == 0) return c_terms10;
  else if constexpr (LA == 1) return c_terms11;
  else if constexpr (LB == 0) return c_terms20;
  else if constexpr (LB == 1) return c_terms21;
  else return c_terms22;
}

// What a block keeps of its bra entry: primitive data and the term products.
template <int LA, int LB>
struct BraShared {
  double prim[ENTRY_PRIMS][5];                             // p, Px, Py, Pz, K'
  double E[LA + LB > 0 ? ENTRY_PRIMS : 1][3][e1_size(LA, LB)];
  double M[LA + LB > 0 ? ENTRY_PRIMS : 1][nterms(LA, LB)];
};
// All threads of the block call this; ends with a barrier.
template <int LA, int LB>
__device__ __forceinline__ void load_bra(BraShared<LA, LB>& S, const double* base, int nb, double Ax, double Ay,
                                         double Az, double Bx, double By, double Bz) {
  const int tid = threadIdx.x;
  for (int i = tid; i < nb * 5; i += blockDim.x) S.prim[i / 5][i % 5] = entry_field(base, i / 5, i % 5);
  if constexpr (LA + LB > 0) {
    for (int i = tid; i < nb * 3; i += blockDim.x) {
      const int ib = i / 3, dir = i % 3;
      const double A = dir == 0 ? Ax : (dir == 1 ? Ay : Az), B = dir == 0 ? Bx : (dir == 1 ? By : Bz);
      const double P = entry_field(base, ib, 1 + dir);
      E1<LA, LB> e;
      md_E1<LA, LB>(P - A, P - B, entry_field(base, ib, 5), e);
#pragma unroll
      for (int a = 0; a <= LA; ++a)
#pragma unroll
        for (int b = 0; b <= LB; ++b)
#pragma unroll
          for (int t = 0; t <= LA + LB; ++t) S.E[ib][dir][e1_pos(LA, LB, a, b, t)] = e.e[a][b][t];
    }
    __syncthreads();
    constexpr int NT = nterms(LA, LB);
    const TermTab<LA, LB>& T = term_tab<LA, LB>();
    for (int i = tid; i < nb * NT; i += blockDim.x) {
      const int ib = i / NT, k = i % NT;
      S.M[ib][k] = S.E[ib][0][T.x[k]] * S.E[ib][1][T.y[k]] * S.E[ib][2][T.z[k]];
    }
  }
  __syncthreads();
}
// first term of component (i, j) in the list
__host__ __device__ constexpr int term_off(int la, int lb, int ij) {
  int n = 0;
  for (int k = 0; k < ij; ++k) {
    const int i = k / ncart(lb), j = k % ncart(lb);
    n += (cart_a(la, i) + cart_a(lb, j) + 1) * (cart_b(la, i) + cart_b(lb, j) + 1) *
         (cart_c(la, i) + cart_c(lb, j) + 1);
  }
  return n;
}
// out[ab * STRIDE] += sum of M W over the terms of each component
template <int LA, int LB, int STRIDE>
__device__ __forceinline__ void bra_transform(const double* M, const double* W, double* out) {
  if constexpr (LA + LB == 0) {
    out[0] += W[0];
  } else {
    static_for<ncart(LA) * ncart(LB)>([&](auto ij) {
      constexpr int i = decltype(ij)::value / ncart(LB), j = decltype(ij)::value % ncart(LB);
      constexpr int nu = cart_b(LA, i) + cart_b(LB, j) + 1, nv = cart_c(LA, i) + cart_c(LB, j) + 1;
      constexpr int nt = (cart_a(LA, i) + cart_a(LB, j) + 1) * nu * nv;
      constexpr int k0 = term_off(LA, LB, decltype(ij)::value);
      double acc = out[decltype(ij)::value * STRIDE];
      static_for<nt>([&](auto q) {
        constexpr int k = decltype(q)::value;
        acc += M[k0 + k] * W[hidx(k / (nu * nv), (k / nv) % nu, k % nv)];
      });
      out[decltype(ij)::value * STRIDE] = acc;
    });
  }
}

// One component of the bra transform, by a run-time index: sum of M W.
template <int LA, int LB>
__device__ __forceinline__ double bra_component(const double* M, const double* W, int ij) {
  if constexpr (LA + LB == 0) {
    return W[0];
  } else {
    const TermTab<LA, LB>& T = term_tab<LA, LB>();
    constexpr int N = LA + LB + 1;
    int k = T.first[ij];
    const int k1 = T.first[ij + 1];
    double acc = 0.0;
    for (; k < k1; ++k) acc += M[k] * W[hidx(T.x[k] % N, T.y[k] % N, T.z[k] % N)];
    return acc;
  }
}

// ---------------------------------------------------------------- ket expansion
// One application of (x - centre) to a one-direction Hermite expansion.
template <int N>
__device__ __forceinline__ void e1_raise(double* e, double X, double h) {
  double n[N + 1];
#pragma unroll
  for (int t = 0; t <= N; ++t) {
    n[t] = X * e[t];
    if (t > 0) n[t] += h * e[t - 1];
    if (t < N) n[t] += (t + 1) * e[t + 1];
  }
#pragma unroll
  for (int t = 0; t <= N; ++t) e[t] = n[t];
}
// W[h] += sum over the ket's Hermite terms (t', u', v') <= (tx, ty, tz) of
// (-1)^(t'+u'+v') ex ey ez R[h + (t', u', v')].  The bounds are the same for the
// whole block (one ket component at a time), so the loops stay unrolled with R
// in registers and a uniform branch skips the terms that vanish.
template <int HL, int LK>
__device__ __forceinline__ void ket_accumulate(double* W, const double* R, const double* ex, const double* ey,
                                               const double* ez, int tx, int ty, int tz) {
  static_for<nherm(LK)>([&](auto g) {
    constexpr int a = herm_t(decltype(g)::value), b = herm_u(decltype(g)::value), c = herm_v(decltype(g)::value);
    if (a <= tx && b <= ty && c <= tz) {
      const double e0 = ex[a] * ey[b] * ez[c];
      const double e = ((a + b + c) & 1) ? -e0 : e0;
      static_for<nherm(HL)>([&](auto hh) {
        constexpr int h = decltype(hh)::value;
        W[h] += e * R[hidx(herm_t(h) + a, herm_u(h) + b, herm_v(h) + c)];
      });
    }
  });
}

// ---------------------------------------------------------------- derivatives
// With P = (alpha A + beta B)/p and R = A - B, d/dA = (alpha/p) d/dP + d/dR: the
// first part shifts a Hermite index, the second differentiates the expansion
// coefficients (and the prefactor exp(-mu R^2), whose factor belongs to them),
// which leaves their order unchanged.  One table of R integrals of order L + 1
// therefore gives the derivatives with respect to all centres.

// (x - centre) applied to an expansion e and to its R derivative r; Xr = d(X)/dR.
template <int N>
__device__ __forceinline__ void e1_raise_dual(double* e, double* r, double X, double Xr, double h) {
  double n[N + 1];
#pragma unroll
  for (int t = 0; t <= N; ++t) n[t] = Xr * e[t];
  e1_raise<N>(e, X, h);
  e1_raise<N>(r, X, h);
#pragma unroll
  for (int t = 0; t <= N; ++t) r[t] += n[t];
}

// Term products of the bra entry and their derivatives d/dR_x, x = 0, 1, 2.
template <int LA, int LB>
struct BraGradShared {
  double prim[ENTRY_PRIMS][6];  // p, Px, Py, Pz, K', alpha/p
  double E[ENTRY_PRIMS][2][3][e1_size(LA, LB)];
  double M[ENTRY_PRIMS][4][nterms(LA, LB)];
};
template <int LA, int LB>
__device__ __forceinline__ void load_bra_grad(BraGradShared<LA, LB>& S, const double* base, int nb, double Ax,
                                              double Ay, double Az, double Bx, double By, double Bz) {
  const int tid = threadIdx.x;
  for (int i = tid; i < nb * 6; i += blockDim.x) {
    const int ib = i / 6, f = i % 6;
    S.prim[ib][f] = f < 5 ? entry_field(base, ib, f) : entry_field(base, ib, 6) * 2.0 * entry_field(base, ib, 5);
  }
  for (int i = tid; i < nb * 3; i += blockDim.x) {
    const int ib = i / 3, dir = i % 3;
    const double A = dir == 0 ? Ax : (dir == 1 ? Ay : Az), B = dir == 0 ? Bx : (dir == 1 ? By : Bz);
    const double P = entry_field(base, ib, 1 + dir), h = entry_field(base, ib, 5);
    const double al = entry_field(base, ib, 6), fa = 2.0 * h * al, fb = 1.0 - fa;  // alpha/p, beta/p
    constexpr int N = LA + LB;
    double ea[N + 1], ra[N + 1];
#pragma unroll
    for (int t = 0; t <= N; ++t) ea[t] = ra[t] = 0.0;
    ea[0] = 1.0;
    ra[0] = -2.0 * al * fb * (A - B);
#pragma unroll
    for (int a = 0; a <= LA; ++a) {
      if (a > 0) e1_raise_dual<N>(ea, ra, P - A, -fb, h);
      double eb[N + 1], rb[N + 1];
#pragma unroll
      for (int t = 0; t <= N; ++t) {
        eb[t] = ea[t];
        rb[t] = ra[t];
      }
#pragma unroll
      for (int b = 0; b <= LB; ++b) {
        if (b > 0) e1_raise_dual<N>(eb, rb, P - B, fa, h);
#pragma unroll
        for (int t = 0; t <= N; ++t) {
          S.E[ib][0][dir][e1_pos(LA, LB, a, b, t)] = eb[t];
          S.E[ib][1][dir][e1_pos(LA, LB, a, b, t)] = rb[t];
        }
      }
    }
  }
  __syncthreads();
  constexpr int NT = nterms(LA, LB);
  const TermTab<LA, LB>& T = term_tab<LA, LB>();
  for (int i = tid; i < nb * 4 * NT; i += blockDim.x) {
    const int ib = i / (4 * NT), w = (i / NT) % 4, k = i % NT;  // w = 0: value, 1 + x: d/dR_x
    S.M[ib][w][k] = S.E[ib][w == 1][0][T.x[k]] * S.E[ib][w == 2][1][T.y[k]] * S.E[ib][w == 3][2][T.z[k]];
  }
  __syncthreads();
}

// f(component, term, Hermite index), all constants, over the terms of (LA, LB)
template <int LA, int LB, class F>
__device__ __forceinline__ void for_terms(F&& f) {
  static_for<ncart(LA) * ncart(LB)>([&](auto ij) {
    constexpr int c = decltype(ij)::value, i = c / ncart(LB), j = c % ncart(LB);
    constexpr int nu = cart_b(LA, i) + cart_b(LB, j) + 1, nv = cart_c(LA, i) + cart_c(LB, j) + 1;
    constexpr int nt = (cart_a(LA, i) + cart_a(LB, j) + 1) * nu * nv;
    constexpr int k0 = term_off(LA, LB, c);
    static_for<nt>([&](auto q) {
      constexpr int k = decltype(q)::value;
      f(std::integral_constant<int, c>{}, std::integral_constant<int, k0 + k>{},
        std::integral_constant<int, hidx(k / (nu * nv), (k / nv) % nu, k % nv)>{});
    });
  });
}

// One primitive quartet's derivatives for bra weights G (Hermite orders <= HL)
// and one ket component with expansions e, their R derivatives r and bounds
// (tx, ty, tz): gP[x] += d/dP_x, gR[x] += the ket's d/dR_x part.  R holds orders
// up to HL + LK + 1.  V is the bra's potential at one ket Hermite index.  G holds
// the bra's degrees LO .. HL only.
template <int HL, int LK, int LO = 0>
__device__ __forceinline__ void ket_gradient(const double* G, const double* R, const double (*e)[LK + 1],
                                             const double (*r)[LK + 1], int tx, int ty, int tz, double* gP,
                                             double* gR) {
  static_for<nherm(LK + 1)>([&](auto gg) {
    constexpr int a = herm_t(decltype(gg)::value), b = herm_u(decltype(gg)::value), c = herm_v(decltype(gg)::value);
    const bool box = a <= tx && b <= ty && c <= tz;
    const bool sx = a > 0 && a - 1 <= tx && b <= ty && c <= tz;
    const bool sy = b > 0 && a <= tx && b - 1 <= ty && c <= tz;
    const bool sz = c > 0 && a <= tx && b <= ty && c - 1 <= tz;
    if (box || sx || sy || sz) {
      double v0 = 0.0, v1 = 0.0;
      constexpr int h0 = LO > 0 ? nherm(LO - 1) : 0;
      static_for<nherm(HL) - h0>([&](auto hh) {
        constexpr int i = decltype(hh)::value, h = h0 + i;
        if constexpr (h & 1)
          v1 += G[i] * R[hidx(herm_t(h) + a, herm_u(h) + b, herm_v(h) + c)];
        else
          v0 += G[i] * R[hidx(herm_t(h) + a, herm_u(h) + b, herm_v(h) + c)];
      });
      const double V = ((a + b + c) & 1) ? -(v0 + v1) : v0 + v1;
      if constexpr (a + b + c <= LK) {
        if (box) {
          gR[0] += r[0][a] * e[1][b] * e[2][c] * V;
          gR[1] += e[0][a] * r[1][b] * e[2][c] * V;
          gR[2] += e[0][a] * e[1][b] * r[2][c] * V;
        }
      }
      if constexpr (a > 0)
        if (sx) gP[0] -= e[0][a - 1] * e[1][b] * e[2][c] * V;
      if constexpr (b > 0)
        if (sy) gP[1] -= e[0][a] * e[1][b - 1] * e[2][c] * V;
      if constexpr (c > 0)
        if (sz) gP[2] -= e[0][a] * e[1][b] * e[2][c - 1] * V;
    }
  });
}
// One-direction expansions of the ket component (i, j) in each direction and
// their R derivatives.
template <int LC, int LD>
__device__ __forceinline__ void ket_expansions(double (*e)[LC + LD + 1], double (*r)[LC + LD + 1], const double* Q,
                                               const double* C, const double* D, double ga, double h, const int* ce,
                                               const int* de) {
  constexpr int N = LC + LD;
  const double fc = 2.0 * h * ga, fd = 1.0 - fc;  // gamma/q, delta/q
#pragma unroll
  for (int x = 0; x < 3; ++x) {
#pragma unroll
    for (int t = 0; t <= N; ++t) e[x][t] = r[x][t] = 0.0;
    e[x][0] = 1.0;
    r[x][0] = -2.0 * ga * fd * (C[x] - D[x]);
#pragma unroll
    for (int s = 0; s < LC; ++s)
      if (s < ce[x]) e1_raise_dual<N>(e[x], r[x], Q[x] - C[x], -fd, h);
#pragma unroll
    for (int s = 0; s < LD; ++s)
      if (s < de[x]) e1_raise_dual<N>(e[x], r[x], Q[x] - D[x], fc, h);
  }
}

}  // namespace m2
