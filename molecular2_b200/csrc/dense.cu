// FP64 GEMM, blocked Cholesky and triangular inverse (dense.cuh).
//
// GEMM: 128 x BN output tiles, 256 threads = 8 warps of FP64 tensor-core tiles
// (mma.sync m8n8k4, the DMMA path, measured 37.1 TFLOP/s on its own, the same as
// every larger DMMA shape), k tiles of 16 in a three-stage shared-memory ring
// filled by cp.async (out-of-range elements are copied as zeros).  The copies
// are 16 bytes wide along an operand's contiguous dimension when its base and
// strides allow it, 8 bytes otherwise.  The shared-memory pitches (4 modulo 16
// doubles) spread the 4 x 8 elements of a fragment over the banks evenly.
// BN follows N: with the one 128-wide tile that was here before, N = 80 spent
// 37 % of its work on padding (see pick_bn).
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <string>
#include <type_traits>

#include "dense.cuh"

namespace m2 {
namespace {

constexpr int GBM = 128, GBK = 16, GT = 256, GST = 3;
constexpr int LDK = GBK + 4;                                    // pitch of [m][k] and [n][k] tiles
constexpr int lds(int n) { return n + (20 - n % 16) % 16; }     // pitch of [k][m] and [k][n] tiles: 4 modulo 16
constexpr int oper(int n) { return GBK * lds(n) > n * LDK ? GBK * lds(n) : n * LDK; }  // doubles per operand stage
constexpr int gsmem(int bn) { return GST * (oper(GBM) + oper(bn)) * (int)sizeof(double); }
// warps along N: as square a warp tile as BN allows in multiples of 8
constexpr int warps_n(int bn) { return bn >= 96 ? 4 : (bn % 16 == 0 ? 2 : 1); }

__device__ __forceinline__ void cp16(double* dst, const double* src, int bytes) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp8(double* dst, const double* src, bool ok) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(ok ? 8 : 0) : "memory");
}
// D = A B + D for one 8 x 8 x 4 FP64 tile: a = A(lane/4, lane%4),
// b = B(lane%4, lane/4), d = D(lane/4, 2*(lane%4) + {0, 1}).
__device__ __forceinline__ void dmma(double* d, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

__device__ __forceinline__ void tri_tile(int t, int& tm, int& tn) {
  int m = (int)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
  while (m * (m + 1) / 2 > t) --m;
  while ((m + 1) * (m + 2) / 2 <= t) ++m;
  tm = m;
  tn = t - m * (m + 1) / 2;
}

// One stage of an operand: ROWS rows (m or n) by 16 k.  K1: k contiguous in
// global memory, kept as [row][k]; otherwise [k][row].  Elements beyond nrow or
// k_end are zero.
template <int ROWS, bool K1>
__device__ __forceinline__ void load_stage(double* sm, const double* g, long long sr, long long sk, int r0, int nrow,
                                           int k0, int k_end, bool vec) {
  const int t = threadIdx.x;
  if (vec) {
    constexpr int NV = ROWS * GBK / 2;
#pragma unroll
    for (int i0 = 0; i0 < NV; i0 += GT) {
      const int i = i0 + t;
      if (NV % GT != 0 && i >= NV) break;
      int r, k, left;
      if (K1) {
        k = 2 * (i % (GBK / 2));
        r = i / (GBK / 2);
        left = r0 + r < nrow ? k_end - k0 - k : 0;
      } else {
        r = 2 * (i % (ROWS / 2));
        k = i / (ROWS / 2);
        left = k0 + k < k_end ? nrow - r0 - r : 0;
      }
      const int bytes = left >= 2 ? 16 : (left == 1 ? 8 : 0);
      const double* src = g + (long long)(r0 + r) * sr + (long long)(k0 + k) * sk;
      cp16(sm + (K1 ? r * LDK + k : k * lds(ROWS) + r), bytes ? src : g, bytes);
    }
  } else {
    constexpr int NE = ROWS * GBK;
#pragma unroll 4
    for (int i = t; i < NE; i += GT) {
      const int r = K1 ? i / GBK : i % ROWS, k = K1 ? i % GBK : i / ROWS;
      const bool ok = r0 + r < nrow && k0 + k < k_end;
      cp8(sm + (K1 ? r * LDK + k : k * lds(ROWS) + r),
          ok ? g + (long long)(r0 + r) * sr + (long long)(k0 + k) * sk : g, ok);
    }
  }
}

template <bool AK1, bool BN1, int BN>
__global__ void __launch_bounds__(GT) k_dgemm(const DGemm g, int tiles_n, bool vec_a, bool vec_b) {
  constexpr int WNW = warps_n(BN), WMW = 8 / WNW, WM = GBM / WMW, WN = BN / WNW, TM = WM / 8, TN = WN / 8;
  static_assert(TM * 8 * WMW == GBM && TN * 8 * WNW == BN, "warp tiles must cover the block tile");
  extern __shared__ __align__(16) double gsm[];
  double* As = gsm;
  double* Bs = gsm + GST * oper(GBM);
  auto aidx = [](int k, int m) { return AK1 ? m * LDK + k : k * lds(GBM) + m; };
  auto bidx = [](int k, int n) { return BN1 ? k * lds(BN) + n : n * LDK + k; };
  int tm, tn;
  if (g.c_lower)
    tri_tile(blockIdx.x, tm, tn);
  else {
    tm = blockIdx.x / tiles_n;
    tn = blockIdx.x % tiles_n;
    if (g.a_lower) tm = (gridDim.x / tiles_n) - 1 - tm;  // longest k ranges first
  }
  const int m0 = tm * GBM, n0 = tn * BN;
  const long long bz = blockIdx.z;
  const double* A = g.A + bz * g.bsa;
  const double* B = g.B + bz * g.bsb;
  double* C = g.C + bz * g.bsc;
  int kb = 0, ke = g.K;
  if (g.a_lower) ke = min(ke, m0 + GBM);
  if (g.b_lower) kb = min(ke, n0);
  kb = (kb / GBK) * GBK;
  if (g.ksplit > 1) {
    const int len = max(0, ke - kb);
    const int chunk = ((len + g.ksplit - 1) / g.ksplit + GBK - 1) / GBK * GBK;
    const int s0 = kb + (int)blockIdx.y * chunk;
    const int s1 = min(ke, s0 + chunk);
    if (s0 >= s1) return;
    kb = s0;
    ke = s1;
  }
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, wm = warp / WNW, wn = warp % WNW;
  auto load = [&](int it) {
    const int st = it % GST, k0 = kb + it * GBK;
    load_stage<GBM, AK1>(As + st * oper(GBM), A, g.sam, g.sak, m0, g.M, k0, ke, vec_a);
    load_stage<BN, !BN1>(Bs + st * oper(BN), B, g.sbn, g.sbk, n0, g.N, k0, ke, vec_b);
  };

  const int nk = ke > kb ? (ke - kb + GBK - 1) / GBK : 0;
#pragma unroll
  for (int it = 0; it < GST - 1; ++it) {
    if (it < nk) load(it);
    cp_commit();
  }
  const int fk = lane & 3, fr = lane >> 2;
  // the sums start from beta / alpha C, read while the first stages arrive (read
  // at the end, every element would wait for its own round trip behind the
  // stores before it)
  double acc[TM][TN][2];
  const double c_in = g.ksplit > 1 ? 0.0 : g.beta / g.alpha;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + wm * WM + i * 8 + fr;
#pragma unroll
    for (int j = 0; j < TN; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int gn = n0 + wn * WN + j * 8 + 2 * fk + h;
        acc[i][j][h] = 0.0;
        if (c_in != 0.0 && gm < g.M && gn < g.N)
          acc[i][j][h] = c_in * C[(long long)gm * g.scm + (long long)gn * g.scn];
      }
  }
  // a warp above the diagonal of a lower-triangle tile only helps to load
  const bool above = g.c_lower && tm == tn && wm * WM + WM <= wn * WN;
  for (int it = 0; it < nk; ++it) {
    cp_wait<GST - 2>();
    __syncthreads();
    if (it + GST - 1 < nk) load(it + GST - 1);
    cp_commit();
    if (above) continue;
    const double* a_s = As + (it % GST) * oper(GBM);
    const double* b_s = Bs + (it % GST) * oper(BN);
#pragma unroll
    for (int k4 = 0; k4 < GBK; k4 += 4) {
      double a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = a_s[aidx(k4 + fk, wm * WM + i * 8 + fr)];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = b_s[bidx(k4 + fk, wn * WN + j * 8 + fr)];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) dmma(acc[i][j], a[i], b[j]);
    }
  }
  if (above) return;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + wm * WM + i * 8 + fr;
    if (gm >= g.M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int gn = n0 + wn * WN + j * 8 + 2 * fk + h;
        if (gn >= g.N) continue;
        double* c = C + (long long)gm * g.scm + (long long)gn * g.scn;
        if (g.ksplit > 1)
          atomicAdd(c, g.alpha * acc[i][j][h]);
        else
          *c = g.alpha * acc[i][j][h];
      }
  }
}

__global__ void k_scale(double* C, int M, int N, long long scm, long long scn, long long bsc, double beta) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)M * N) return;
  const int m = (int)(idx % M), n = (int)(idx / M);
  double* c = C + (long long)blockIdx.y * bsc + (long long)m * scm + (long long)n * scn;
  *c = beta == 0.0 ? 0.0 : beta * *c;
}

// ---------------------------------------------------------------- Cholesky
constexpr int CNB = 64;  // panel width

// Factor the b x b diagonal block at (j, j) in place (lower triangle; the
// strict upper part of the block is zeroed) and write its inverse to Dinv
// (CNB x CNB, column-major, ld CNB).  A non-positive pivot sets *info to 1 +
// its index (first one wins) and the block continues with a unit pivot so
// that every later value stays finite.
//
// A chain of 64 steps on one SM, so what counts is a step's latency.  Thread (r, q)
// keeps row r, columns q, q + 4, .. of the block and of the inverse in registers;
// step c publishes column c of the block and row c of the inverse, both still
// unscaled, and every later row subtracts (a_rc / a_cc) times them: one barrier and
// one division a step.  The square roots are taken once, at the end.  41 us a
// block; 98 us with the block in shared memory, three barriers a step and the
// inverse by columns after it.
__global__ void __launch_bounds__(4 * CNB) k_potrf_diag(double* A, int n, int j, double* Dinv, int* info) {
  __shared__ double col[2][CNB], row[2][CNB], piv[CNB];
  const int b = min(CNB, n - j), t = threadIdx.x, r = t % CNB, q = t / CNB;
  double a[CNB / 4], x[CNB / 4];
#pragma unroll
  for (int k = 0; k < CNB / 4; ++k) {
    const int c = 4 * k + q;
    // rows past b: the unit matrix
    a[k] = r < b && c < b ? (r >= c ? A[(size_t)(j + c) * n + j + r] : 0.0) : (r == c ? 1.0 : 0.0);
    x[k] = r == c ? 1.0 : 0.0;
  }
#pragma unroll
  for (int k = 0; k < CNB / 4; ++k) {
    for (int cq = 0; cq < 4; ++cq) {
      const int c = 4 * k + cq, s = c & 1;
      if (q == cq) col[s][r] = a[k];
      if (r == c) {
#pragma unroll
        for (int l = 0; l <= k; ++l) row[s][4 * l + q] = x[l];
      }
      __syncthreads();
      double d = col[s][c];
      if (!(d > 0.0)) {
        if (t == 0) atomicCAS(info, 0, 1 + j + c);
        d = 1.0;
      }
      if (t == 0) piv[c] = d;
      if (r > c) {
        const double f = -col[s][r] / d;
#pragma unroll
        for (int l = k; l < CNB / 4; ++l) {
          // a column up to c has its final value; the rest of the upper triangle is not used
          if (4 * l + q > c) a[l] = fma(f, col[s][4 * l + q], a[l]);
        }
#pragma unroll
        for (int l = 0; l <= k; ++l)
          if (4 * l + q <= c) x[l] = fma(f, row[s][4 * l + q], x[l]);
      }
    }
  }
  __syncthreads();
  const double dr = sqrt(piv[r]);
#pragma unroll
  for (int k = 0; k < CNB / 4; ++k) {
    const int c = 4 * k + q;
    if (r < b && c < b) {
      const double dc = sqrt(piv[c]);
      A[(size_t)(j + c) * n + j + r] = r > c ? a[k] / dc : (r == c ? dc : 0.0);
      Dinv[(size_t)c * CNB + r] = r >= c ? x[k] / dr : 0.0;
    }
  }
}

__global__ void k_zero_upper(double* A, int n) {
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (size_t)n * n) return;
  if ((int)(idx % n) < (int)(idx / n)) A[idx] = 0.0;
}

__global__ void k_mirror(double* C, int n) {
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (size_t)n * n) return;
  const int i = (int)(idx % n), j = (int)(idx / n);
  if (i < j) C[idx] = C[(size_t)i * n + j];
}

// Inverse of each CNB x CNB diagonal block of the lower-triangular L into
// Linv (same positions); one block of threads per diagonal block.
__global__ void __launch_bounds__(CNB) k_trinv_diag(const double* L, double* Linv, int n) {
  __shared__ double S[CNB][CNB + 1];
  const int j = blockIdx.x * CNB, b = min(CNB, n - j), t = threadIdx.x;
  for (int idx = t; idx < b * b; idx += blockDim.x) {
    const int r = idx % b, c = idx / b;
    S[r][c] = L[(size_t)(j + c) * n + j + r];
  }
  __syncthreads();
  if (t < b) {
    const int col = t;
    double x[CNB];
    for (int r = 0; r < b; ++r) x[r] = 0.0;
    x[col] = 1.0 / S[col][col];
    for (int r = col + 1; r < b; ++r) {
      double acc = 0.0;
      for (int k = col; k < r; ++k) acc += S[r][k] * x[k];
      x[r] = -acc / S[r][r];
    }
    for (int r = 0; r < b; ++r) Linv[(size_t)(j + col) * n + j + r] = x[r];
  }
}

}  // namespace

// Tile width for N columns: the least padded columns, weighted with the work a
// narrower tile adds per column (fragment loads per DMMA).
static int pick_bn(int N) {
  static const struct {
    int bn;
    double w;
  } opt[] = {{128, 1.0}, {96, 1.0}, {80, 1.0}, {64, 1.03}, {48, 1.06}, {40, 1.1}, {32, 1.1}, {16, 1.3}};
  int best = 128;
  double cost = 1e300;
  for (const auto& o : opt) {
    const double c = (double)((N + o.bn - 1) / o.bn) * o.bn * o.w;
    if (c < cost) {
      cost = c;
      best = o.bn;
    }
  }
  return best;
}

cudaError_t dgemm(const DGemm& g, cudaStream_t s) {
  if (g.M <= 0 || g.N <= 0 || g.batch <= 0) return cudaSuccess;
  if (g.c_lower && g.M != g.N) return cudaErrorInvalidValue;
  if (g.batch > 65535 || g.ksplit < 1 || g.ksplit > 65535) return cudaErrorInvalidValue;
  DGemm h = g;
  if (h.ksplit > 1 && h.beta != 1.0) {
    const long long tot = (long long)h.M * h.N;
    k_scale<<<dim3((unsigned)((tot + 255) / 256), h.batch), 256, 0, s>>>(h.C, h.M, h.N, h.scm, h.scn, h.bsc,
                                                                           h.beta);
    h.beta = 1.0;
  }
  const int bn = h.c_lower ? 128 : pick_bn(h.N);
  const int tm = (h.M + GBM - 1) / GBM, tn = (h.N + bn - 1) / bn;
  const long long tiles = h.c_lower ? (long long)tm * (tm + 1) / 2 : (long long)tm * tn;
  dim3 grid((unsigned)tiles, h.ksplit, h.batch);
  const bool ak1 = h.sak == 1, bn1 = h.sbn == 1;
  auto aligned = [](const double* p, long long s1, long long s2) {
    return ((uintptr_t)p & 15) == 0 && s1 % 2 == 0 && s2 % 2 == 0;
  };
  const bool va = (ak1 ? aligned(h.A, h.sam, h.bsa) : h.sam == 1 && aligned(h.A, h.sak, h.bsa));
  const bool vb = (bn1 ? aligned(h.B, h.sbk, h.bsb) : h.sbk == 1 && aligned(h.B, h.sbn, h.bsb));
  auto launch = [&](auto kern, int smem) {
    cudaError_t st = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (st != cudaSuccess) return st;
    kern<<<grid, GT, smem, s>>>(h, tn, va, vb);
    return cudaGetLastError();
  };
  auto pick = [&](auto width) {
    constexpr int W = decltype(width)::value;
    if (ak1 && bn1) return launch(k_dgemm<true, true, W>, gsmem(W));
    if (ak1) return launch(k_dgemm<true, false, W>, gsmem(W));
    if (bn1) return launch(k_dgemm<false, true, W>, gsmem(W));
    return launch(k_dgemm<false, false, W>, gsmem(W));
  };
  switch (bn) {
    case 16: return pick(std::integral_constant<int, 16>{});
    case 32: return pick(std::integral_constant<int, 32>{});
    case 40: return pick(std::integral_constant<int, 40>{});
    case 48: return pick(std::integral_constant<int, 48>{});
    case 64: return pick(std::integral_constant<int, 64>{});
    case 80: return pick(std::integral_constant<int, 80>{});
    case 96: return pick(std::integral_constant<int, 96>{});
    default: return pick(std::integral_constant<int, 128>{});
  }
}

// Blocks of a split-k GEMM over `tiles` output tiles: the split that leaves the
// last wave of one block per SM fullest, with at least 128 k per block.
int split_k(long long tiles, long long K, int nsm) {
  const long long most = std::max(1LL, std::min(65535LL, K / 128));
  int best = 1;
  double eff = 0.0;
  for (int waves = 1; waves <= 8; ++waves) {
    const long long ks = std::min(most, waves * (long long)nsm / tiles);
    if (ks < 1) continue;
    const long long blocks = tiles * ks, w = (blocks + nsm - 1) / nsm;
    const double e = (double)blocks / (double)(w * nsm);
    if (e > eff + 0.02) {
      eff = e;
      best = (int)ks;
    }
  }
  return best;
}

void mirror_lower(double* C, int n, cudaStream_t s) {
  const size_t nn = (size_t)n * n;
  k_mirror<<<(unsigned)((nn + 255) / 256), 256, 0, s>>>(C, n);
}

int cholesky(jk_engine* e, double* A, int n, double* work, int* info, cudaStream_t s) {
  cudaMemsetAsync(info, 0, sizeof(int), s);
  for (int j = 0; j < n; j += CNB) {
    const int b = std::min(CNB, n - j);
    k_potrf_diag<<<1, 4 * CNB, 0, s>>>(A, n, j, work, info);
    const int R = n - j - b;
    if (R <= 0) break;
    // L21 = A21 L11^-T, in place: at most 64 columns are one tile wide
    // (pick_bn), so each block reads only the rows it writes
    DGemm p;
    p.M = R;
    p.N = b;
    p.K = b;
    p.A = A + (size_t)j * n + j + b;
    p.sam = 1;
    p.sak = n;
    p.B = work;      // B(k, c) = Dinv(c, k)
    p.sbk = CNB;
    p.sbn = 1;
    p.C = A + (size_t)j * n + j + b;
    p.scm = 1;
    p.scn = n;
    cudaError_t st = dgemm(p, s);
    if (st != cudaSuccess) return check_cuda(e, st, "cholesky panel");
    // A22 -= L21 L21^T on the tiles on or below the diagonal
    DGemm u;
    u.M = R;
    u.N = R;
    u.K = b;
    u.A = A + (size_t)j * n + j + b;
    u.sam = 1;
    u.sak = n;
    u.B = A + (size_t)j * n + j + b;  // B(k, r') = L21(r', k)
    u.sbk = n;
    u.sbn = 1;
    u.C = A + (size_t)(j + b) * n + j + b;
    u.scm = 1;
    u.scn = n;
    u.alpha = -1.0;
    u.beta = 1.0;
    u.c_lower = true;
    st = dgemm(u, s);
    if (st != cudaSuccess) return check_cuda(e, st, "cholesky update");
  }
  const size_t nn = (size_t)n * n;
  k_zero_upper<<<(unsigned)((nn + 255) / 256), 256, 0, s>>>(A, n);
  return check_cuda(e, cudaGetLastError(), "cholesky");
}

// Linv[lo:hi, lo:hi] from its diagonal blocks (already inverted):
// Linv21 = -Linv22 L21 Linv11 for a split at `mid`.
static int tri_inverse_rec(jk_engine* e, const double* L, double* Linv, int n, int lo, int hi, double* work,
                           cudaStream_t s) {
  if (hi - lo <= CNB) return JK_OK;
  const int nb = (hi - lo + CNB - 1) / CNB;
  const int mid = lo + ((nb + 1) / 2) * CNB;
  int rc = tri_inverse_rec(e, L, Linv, n, lo, mid, work, s);
  if (!rc) rc = tri_inverse_rec(e, L, Linv, n, mid, hi, work, s);
  if (rc) return rc;
  const int r = hi - mid, c = mid - lo;
  // T (r x c, column-major ld r) = L21 Linv11
  DGemm a;
  a.M = r;
  a.N = c;
  a.K = c;
  a.A = L + (size_t)lo * n + mid;
  a.sam = 1;
  a.sak = n;
  a.B = Linv + (size_t)lo * n + lo;
  a.sbk = 1;
  a.sbn = n;
  a.b_lower = true;
  a.C = work;
  a.scm = 1;
  a.scn = r;
  cudaError_t st = dgemm(a, s);
  if (st != cudaSuccess) return check_cuda(e, st, "triangular inverse");
  DGemm b;
  b.M = r;
  b.N = c;
  b.K = r;
  b.A = Linv + (size_t)mid * n + mid;
  b.sam = 1;
  b.sak = n;
  b.a_lower = true;
  b.B = work;
  b.sbk = 1;
  b.sbn = r;
  b.C = Linv + (size_t)lo * n + mid;
  b.scm = 1;
  b.scn = n;
  b.alpha = -1.0;
  st = dgemm(b, s);
  return check_cuda(e, st, "triangular inverse");
}

int tri_inverse(jk_engine* e, const double* L, double* Linv, int n, double* work, cudaStream_t s) {
  cudaMemsetAsync(Linv, 0, sizeof(double) * (size_t)n * n, s);
  k_trinv_diag<<<(n + CNB - 1) / CNB, CNB, 0, s>>>(L, Linv, n);
  cudaError_t st = cudaGetLastError();
  if (st != cudaSuccess) return check_cuda(e, st, "triangular inverse (diagonal blocks)");
  return tri_inverse_rec(e, L, Linv, n, 0, n, work, s);
}

}  // namespace m2
