// Symmetric eigenproblem of a small, nearly diagonal matrix, for the SCF driver:
// from the second iteration on, the Fock matrix in the previous eigenvectors.
// Cyclic Jacobi with the round-robin pair order (n / 2 disjoint rotations at a
// time), after Golub & Van Loan, "Matrix Computations" ch. 8.5, with the update
// formulas of Rutishauser, Numer. Math. 9 (1966) 1.
//
// k_jacobi keeps A in the shared memory of one block and writes the rotations
// down; k_jacobi_vectors applies them to the identity, a warp per row of V.  One
// block, because a round is short (0.9 us at n = 96: two barriers, the angles'
// two rsqrt and a divide, 72 bytes of shared memory per 2 x 2 block) and rounds
// depend on each other: 95 rounds a sweep, 6 sweeps in the second iteration down
// to 1 at convergence.  cuSOLVER's syevd, the only way up to now, is some hundred
// dependent launches whatever the matrix holds.  Per SCF iteration, diagonalisation
// with its transforms, mean of a run to 1e-9 (ms, before -> now): n = 7 0.108 ->
// 0.066, 24 0.25 -> 0.10, 48 0.77 -> 0.18, 96 1.75 -> 0.50, 120 2.14 -> 0.71,
// 150 1.37 -> 1.03.  Solved from nothing (8 or 9 sweeps) it gives 2.0 ms at n = 96
// and 5.6 at 150, so the overlap and the first Fock matrix stay with syevd.
//
// Error against extended precision (n = 7..160, |off-diagonal| 1e-6..0.1, norms
// of the matrix): eigenvalues <= 3e-16 through k_rayleigh (7e-16 as Jacobi has
// them, most of it from the transform into the previous vectors; syevd 3.5e-16),
// residuals 1.1 to 2.7e-16 (syevd 1.1 to 4.4e-16).
#include <cmath>

#include "engine.h"
#include "launch.cuh"

namespace m2 {
namespace {

constexpr int JAC_THREADS = 1024;  // n = 144: 0.93 ms an iteration, 512 threads 0.99; the same up to n = 96
constexpr int JAC_BLOCKS = ((SMALL_EIG_MAX / 2) * (SMALL_EIG_MAX / 2 + 1) / 2 + JAC_THREADS - 1) / JAC_THREADS;
constexpr int JAC_SWEEPS = 30;   // bound; 1 to 9 are needed
constexpr int VEC_WARPS = 8;     // rows per block of k_jacobi_vectors
constexpr int VEC_ROUNDS = 8;    // rounds staged at a time

__device__ __forceinline__ void pair_of(int round, int i, int np, int& p, int& q) {
  const int m = np - 1;
  if (i == 0) {
    p = round;
    q = m;
  } else {
    p = round + i;
    if (p >= m) p -= m;
    q = round - i;
    if (q < 0) q += m;
  }
  if (p > q) {
    const int t = p;
    p = q;
    q = t;
  }
}

// (a, b) <- (c a - s b, s a + c b) with c = 1 - s tau: r = (s, tau = s / (1 + c)).
// A small rotation then rounds only its small change.
__device__ __forceinline__ void rotate(double2 r, double& a, double& b) {
  const double a0 = a;
  a = fma(-r.x, fma(r.y, a, b), a);
  b = fma(r.x, fma(-r.y, b, a0), b);
}

__device__ double block_sum(double v, double* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
  for (int w = 0; w < JAC_THREADS / 32; ++w) s += red[w];
  return s;
}

// Ain: n x n symmetric.  rot: (s, tau) of every rotation, rounds in order; meta[0]:
// rounds done; meta[1 + k]: ascending rank of column k; vals: sorted eigenvalues.
// A is padded to an even size np by a zero row and column, which no rotation
// touches, and only its upper triangle is kept.
__global__ void __launch_bounds__(JAC_THREADS) k_jacobi(int n, const double* __restrict__ Ain, double* __restrict__ vals,
                                                        double2* __restrict__ rot, int* __restrict__ meta) {
  extern __shared__ double sm[];
  __shared__ double red[JAC_THREADS / 32];
  const int np = (n + 1) & ~1, h = np / 2, ld = np + 1, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* A = sm;                                       // np x ld, both even x odd: 16-byte aligned end
  double2* cs = reinterpret_cast<double2*>(sm + np * ld);  // h
  double* sh = reinterpret_cast<double*>(cs + h);       // h: t a_pq
  int2* pq = reinterpret_cast<int2*>(sh + h);           // h
  // this thread's 2 x 2 blocks (pair i <= pair j), the same in every round
  int ij[JAC_BLOCKS];
  const int nb = h * (h + 1) / 2;
#pragma unroll
  for (int k = 0; k < JAC_BLOCKS; ++k) {
    const int b = tid + k * JAC_THREADS;
    ij[k] = -1;
    if (b < nb) {
      int j = (int)((sqrtf(8.0f * b + 1.0f) - 1.0f) * 0.5f);
      while (j * (j + 1) / 2 > b) --j;
      while ((j + 1) * (j + 2) / 2 <= b) ++j;
      ij[k] = (b - j * (j + 1) / 2) | j << 16;
    }
  }
  double norm = 0.0;
  for (int r = warp; r < np; r += JAC_THREADS / 32)
    for (int c = r + lane; c < np; c += 32) {
      const double a = c < n ? Ain[r * n + c] : 0.0;
      A[r * ld + c] = a;
      norm += (r == c ? 1.0 : 2.0) * a * a;
    }
  norm = block_sum(norm, red);
  if (!(norm <= 1e300)) {  // an infinity or NaN: nothing to find
    for (int k = tid; k < n; k += JAC_THREADS) {
      meta[1 + k] = k;
      vals[k] = nan("");
    }
    if (tid == 0) meta[0] = -1;
    return;
  }
  const double tol2 = 0.5e-30 * n * norm;
  int rounds = 0;
  for (int sweep = 0; sweep < JAC_SWEEPS; ++sweep) {
    double off = 0.0;
    for (int r = warp; r < np; r += JAC_THREADS / 32)
      for (int c = r + 1 + lane; c < np; c += 32) off += A[r * ld + c] * A[r * ld + c];
    off = block_sum(off, red);
    if (!(off > tol2)) break;
    for (int round = 0; round < np - 1; ++round, ++rounds) {
      if (tid < h) {
        int p, q;
        pair_of(round, tid, np, p, q);
        // the smaller of the two angles that clear a_pq: with the double angle's
        // hypotenuse 1/w, c^2 = (1 + |d| w) / 2 and s = a2 w / (2 c)
        const double a2 = 2.0 * A[p * ld + q], d = A[q * ld + q] - A[p * ld + p];
        double2 r = make_double2(0.0, 0.0);
        double shift = 0.0;
        if (fabs(a2) > 1e-140) {
          const double w = rsqrt(fma(d, d, a2 * a2));
          const double c2 = fma(0.5 * fabs(d), w, 0.5);
          const double rc = rsqrt(c2);
          r.x = 0.5 * copysign(a2, a2 * d) * w * rc;
          r.y = r.x / fma(c2, rc, 1.0);
          shift = 0.5 * a2 * r.x * rc;
        }
        pq[tid] = make_int2(p, q);
        cs[tid] = r;
        sh[tid] = shift;
        rot[(size_t)rounds * h + tid] = r;
      }
      __syncthreads();
      // block <- R_i^T block R_j; the blocks are disjoint
#pragma unroll
      for (int k = 0; k < JAC_BLOCKS; ++k) {
        if (ij[k] < 0) break;
        const int i = ij[k] & 0xffff, j = ij[k] >> 16;
        const int2 rs = pq[i], uv = pq[j];
        const double2 ri = cs[i], rj = cs[j];
        double* e00 = A + (rs.x <= uv.x ? rs.x * ld + uv.x : uv.x * ld + rs.x);
        double* e01 = A + (rs.x <= uv.y ? rs.x * ld + uv.y : uv.y * ld + rs.x);
        double* e10 = A + (rs.y <= uv.x ? rs.y * ld + uv.x : uv.x * ld + rs.y);
        double* e11 = A + (rs.y <= uv.y ? rs.y * ld + uv.y : uv.y * ld + rs.y);
        const double a00 = *e00, a01 = *e01, a10 = *e10, a11 = *e11;
        if (i == j) {
          *e00 = a00 - sh[i];
          *e11 = a11 + sh[i];
          *e01 = 0.0;  // e10 is the same element
        } else {
          double b00 = a00, b01 = a01, b10 = a10, b11 = a11;
          rotate(ri, b00, b10);
          rotate(ri, b01, b11);
          rotate(rj, b00, b01);
          rotate(rj, b10, b11);
          *e00 = b00;
          *e01 = b01;
          *e10 = b10;
          *e11 = b11;
        }
      }
      __syncthreads();
    }
  }
  if (tid == 0) meta[0] = rounds;
  for (int k = tid; k < n; k += JAC_THREADS) {
    const double d = A[k * ld + k];
    int r = 0;
    for (int j = 0; j < n; ++j) {
      const double e = A[j * ld + j];
      r += e < d || (e == d && j < k);
    }
    meta[1 + k] = r;
    vals[r] = d;
  }
}

// vecs (column-major): column rank(k) = the k-th column of the rotations' product.
__global__ void __launch_bounds__(32 * VEC_WARPS) k_jacobi_vectors(int n, const double2* __restrict__ rot,
                                                                   const int* __restrict__ meta,
                                                                   double* __restrict__ vecs) {
  extern __shared__ double sm[];
  const int np = (n + 1) & ~1, h = np / 2, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = blockIdx.x * VEC_WARPS + warp;
  double2* stage = reinterpret_cast<double2*>(sm);  // VEC_ROUNDS x h
  double* v = sm + 2 * (size_t)VEC_ROUNDS * h + (size_t)warp * np;
  for (int k = lane; k < np; k += 32) v[k] = k == row ? 1.0 : 0.0;
  const int rounds = meta[0];
  if (rounds < 0)
    for (int k = lane; k < np; k += 32) v[k] = nan("");
  int round = 0;
  for (int r0 = 0; r0 < rounds; r0 += VEC_ROUNDS) {
    const int nr = min(VEC_ROUNDS, rounds - r0);
    __syncthreads();
    for (int i = threadIdx.x; i < nr * h; i += blockDim.x) stage[i] = rot[(size_t)r0 * h + i];
    __syncthreads();
    for (int r = 0; r < nr; ++r) {
      for (int i = lane; i < h; i += 32) {
        int p, q;
        pair_of(round, i, np, p, q);
        double a = v[p], b = v[q];
        rotate(stage[r * h + i], a, b);
        v[p] = a;
        v[q] = b;
      }
      if (++round == np - 1) round = 0;
      __syncwarp();
    }
  }
  if (row < n)
    for (int k = lane; k < n; k += 32) vecs[(size_t)meta[1 + k] * n + row] = v[k];
}

constexpr size_t jacobi_smem(int n) {
  const size_t np = (n + 1) & ~1;
  return sizeof(double) * np * (np + 1) + np / 2 * (sizeof(double2) + sizeof(double) + sizeof(int2));
}

// vals[k] = v_k^T A v_k, block k.  A is read from L2 by every block; n^2 FMAs each.
__global__ void k_rayleigh(int n, const double* __restrict__ A, const double* __restrict__ vecs,
                           double* __restrict__ vals) {
  __shared__ double v[SMALL_EIG_MAX];
  __shared__ double red[(SMALL_EIG_MAX + 31) / 32];
  const int i = threadIdx.x;
  if (i < n) v[i] = vecs[(size_t)blockIdx.x * n + i];
  __syncthreads();
  double a = 0.0;
  if (i < n) {
#pragma unroll 8
    for (int j = 0; j < n; ++j) a = fma(A[(size_t)j * n + i], v[j], a);
    a *= v[i];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  if ((i & 31) == 0) red[i >> 5] = a;
  __syncthreads();
  if (i == 0) {
    for (int w = 1; w < (int)(blockDim.x + 31) / 32; ++w) a += red[w];
    vals[blockIdx.x] = a;
  }
}

}  // namespace

size_t small_eig_scratch(int n) {
  const int np = (n + 1) & ~1;
  return sizeof(double2) * (size_t)JAC_SWEEPS * (np - 1) * (np / 2) + sizeof(int) * (size_t)(n + 1);
}

cudaError_t small_eig(const double* A, double* vecs, double* vals, int n, void* scratch, cudaStream_t s) {
  const int np = (n + 1) & ~1;
  double2* rot = static_cast<double2*>(scratch);
  int* meta = reinterpret_cast<int*>(rot + (size_t)JAC_SWEEPS * (np - 1) * (np / 2));
  static_assert(jacobi_smem(SMALL_EIG_MAX) <= SMEM_BLOCK_MAX, "one block holds the matrix");
  const cudaError_t st =
      launch_smem(k_jacobi, 1, JAC_THREADS, jacobi_smem(n), jacobi_smem(SMALL_EIG_MAX), s, n, A, vals, rot, meta);
  if (st != cudaSuccess) return st;
  const size_t vs = sizeof(double2) * (size_t)VEC_ROUNDS * (np / 2) + sizeof(double) * (size_t)VEC_WARPS * np;
  k_jacobi_vectors<<<(n + VEC_WARPS - 1) / VEC_WARPS, 32 * VEC_WARPS, vs, s>>>(n, rot, meta, vecs);
  return cudaGetLastError();
}

cudaError_t rayleigh(const double* A, const double* vecs, double* vals, int n, cudaStream_t s) {
  k_rayleigh<<<n, (n + 31) / 32 * 32, 0, s>>>(n, A, vecs, vals);
  return cudaGetLastError();
}

}  // namespace m2
