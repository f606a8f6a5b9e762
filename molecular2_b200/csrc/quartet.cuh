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

// ---------------------------------------------------------------- Boys
// F_M by a degree-8 polynomial on BOYSP_ROWS intervals of [0, 36), table of
// one order (BOYSP_ROWS x BOYSP_COEF, ascending powers of T - centre) in shared
// memory: nine conflict-light 8-byte reads against the seven L1 gathers over a
// 121 KB table of the Taylor form, and small enough (6.9 KB) to stage per
// block.  Interpolation at Chebyshev nodes: error below 2e-16 of F_M.
constexpr int BOYSP_ROWS = 96;
constexpr int BOYSP_COEF = 9;
constexpr int BOYSP_MMAX = 9;   // orders 0..9
constexpr int BOYSP_SIZE = BOYSP_ROWS * BOYSP_COEF;

template <int M>
__device__ __forceinline__ void boys_poly(double T, const double* tab, double* F) {
  static_assert(M <= BOYSP_MMAX, "Boys order too high");
  if (T < BOYS_TMAX) {
    const int row = (int)(T * (BOYSP_ROWS / BOYS_TMAX));
    const double d = T - (row + 0.5) * (BOYS_TMAX / BOYSP_ROWS);
    const double* c = tab + row * BOYSP_COEF;
    double acc = c[BOYSP_COEF - 1];
#pragma unroll
    for (int j = BOYSP_COEF - 2; j >= 0; --j) acc = acc * d + c[j];
    F[M] = acc;
    if constexpr (M > 0) {
      const double e = exp(-T), T2 = 2.0 * T;
#pragma unroll
      for (int m = M - 1; m >= 0; --m) F[m] = (T2 * F[m + 1] + e) * (1.0 / (2 * m + 1));
    }
  } else {
    const double r = rsqrt(T);
    F[0] = 0.886226925452758014 * r;  // sqrt(pi)/2 / sqrt(T)
    if constexpr (M > 0) {
      const double e = exp(-T), it = 0.5 * r * r;
#pragma unroll
      for (int m = 0; m < M; ++m) F[m + 1] = ((2 * m + 1) * F[m] - e) * it;
    }
  }
}

// R_tuv (t + u + v <= L) times `scale` of a primitive quartet with exponents
// p, q and distance (X, Y, Z): prefactor and reduced exponent from one
// reciprocal square root.
template <int L>
__device__ __forceinline__ void quartet_R(double p, double q, double KK, double X, double Y, double Z,
                                          const double* tab, double* R) {
  const double r = rsqrt(p + q);
  const double a = p * q * r * r;
  double F[L + 1];
  boys_poly<L>(a * (X * X + Y * Y + Z * Z), tab, F);
  const double m2a = -2.0 * a;
  double pw = KK * r;
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
  unsigned char x[nterms(LA, LB)], y[nterms(LA, LB)], z[nterms(LA, LB)];
};
template <int LA, int LB>
__host__ __device__ constexpr TermTab<LA, LB> make_terms() {
  TermTab<LA, LB> T{};
  int n = 0;
  for (int i = 0; i < ncart(LA); ++i)
    for (int j = 0; j < ncart(LB); ++j) {
      const int ax = cart_a(LA, i), ay = cart_b(LA, i), az = cart_c(LA, i);
      const int bx = cart_a(LB, j), by = cart_b(LB, j), bz = cart_c(LB, j);
      for (int t = 0; t <= ax + bx; ++t)
        for (int u = 0; u <= ay + by; ++u)
          for (int v = 0; v <= az + bz; ++v, ++n) {
            T.x[n] = (unsigned char)e1_pos(LA, LB, ax, bx, t);
            T.y[n] = (unsigned char)e1_pos(LA, LB, ay, by, u);
            T.z[n] = (unsigned char)e1_pos(LA, LB, az, bz, v);
          }
    }
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

}  // namespace m2
