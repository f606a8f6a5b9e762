// Density-fitted RHF nuclear gradient: the gradient of the energy that the
// DF Fock build of compute_2body_fock_df (molecular2 src/fockbuild.cpp:585-660)
// defines, plus the one-body and nuclear terms of Fock::compute_forces
// (src/rhfgrad.cpp:15-89).  molecular2 only differentiates the 4-index
// energy (compute_2body_fock_deriv<1>); with density fitting the consistent
// gradient differentiates the fitted integrals (mn|P) V^-1 (Q|ls):
//   dE2 = sum_{P,mn} (mn|P)^x W3_{mn,P} + sum_{PQ} (P|Q)^x W2_{PQ}
// (weights in df_grad_kernels.cuh).  Everything before the derivative
// kernels is dense linear algebra on the B tensor kept by jk_df_setup:
//   X[x][K][i]  = sum_y B[x][K][y] C[y][i]                     (DGEMM)
//   bt[K](i,j)  = sum_x X[x][K][i] C[x][j]                     (batched DGEMM)
//   gt_K        = 2 sum_i bt[K](i,i),  c = L^-T gt              (TRSV)
//   d           = bt L^-1  over K (d^P_ij = sum_Q V^-1_PQ (Q|ij))   (TRSM)
//   W2          = d^T d - 1/2 c c^T                            (DGEMM + DGER)
//   Z^P         = C d^P C^T,  W3^P = c_P D - 2 Z^P              (batched DGEMM)
#include <algorithm>
#include <cmath>
#include <vector>

#include "df_grad_kernels.cuh"
#include "dense.cuh"
#include "engine.h"

namespace m2 {

int grad_rhf_device(jk_engine* e, const double* dD, const double* dW, double precision, double* g2e, double* g1e,
                    cudaStream_t s, bool with_2e);
void nuclear_repulsion_grad(const jk_engine* e, std::vector<double>& gn);

// gt_K = 2 sum_i bt[K](i,i)
__global__ void k_trace_bt(int naux, int o, const double* __restrict__ bt, double* __restrict__ g) {
  const int K = blockIdx.x * blockDim.x + threadIdx.x;
  if (K >= naux) return;
  double acc = 0.0;
  const double* b = bt + (size_t)K * o * o;
  for (int i = 0; i < o; ++i) acc += b[(size_t)i * o + i];
  g[K] = 2.0 * acc;
}

// W3[P] = c_P D - 2 Z[P], in place over n*n*naux elements
__global__ void k_w3(size_t nn, int naux, const double* __restrict__ c, const double* __restrict__ D,
                     double* __restrict__ Z) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nn * naux) return;
  const int P = (int)(i / nn);
  Z[i] = c[P] * D[i % nn] - 2.0 * Z[i];
}

// Ce = C diag(eps), C column-major n x o
__global__ void k_scale_cols(int n, int o, const double* __restrict__ C, const double* __restrict__ eps,
                             double* __restrict__ Ce) {
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx < (size_t)n * o) Ce[idx] = C[idx] * eps[idx / n];
}

int grad_df_2e_tiled(jk_engine* e, const double* dC, int nocc, const double* dD, double* g2e, cudaStream_t s);

// Cc (nc x o) = coefficients of the Cartesian functions for C (n x o), column-major
__global__ void k_cart_rows(int nc, int n, int o, const int* __restrict__ cshell, const int* __restrict__ ccomp,
                            const int* __restrict__ l, const int* __restrict__ pure, const int* __restrict__ foff,
                            const double* __restrict__ sph, const double* __restrict__ C, double* __restrict__ Cc) {
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (size_t)nc * o) return;
  const int a = (int)(idx % nc), i = (int)(idx / nc), sh = cshell[a], ic = ccomp[a], ls = l[sh], f0 = foff[sh];
  const double* c = C + (size_t)i * n + f0;
  double v = 0.0;
  if (pure[sh])
    for (int m = 0; m < 2 * ls + 1; ++m) v += sph[sph_off(ls) + m * ncart(ls) + ic] * c[m];
  else
    v = c[ic];
  Cc[idx] = v;
}
static void launch_cart_rows(const jk_engine* e, int o, const double* C, double* Cc, cudaStream_t s) {
  const int nc = e->obs.n_cart;
  k_cart_rows<<<(unsigned)(((size_t)nc * o + 255) / 256), 256, 0, s>>>(
      nc, e->obs.n_final, o, e->dobs.cart_shell.p, e->dobs.cart_comp.p, e->dobs.l.p, e->dobs.pure.p,
      e->dobs.final_off.p, e->dobs.sph.p, C, Cc);
}

// k_grad3 over every orbital pair class and the given fitting shells of each
// group, with W3 (Cartesian orbital functions) holding fitting functions from
// w3_f0 on; the launches add to the gradient and run on the side streams,
// longest first.
static cudaError_t launch_grad3_all(jk_engine* e, const int* const* shells, const int* counts, const double* W3,
                                    int w3_f0, double* g2e, cudaStream_t s) {
  static decltype(&launch_grad3_s) const launch[jk_engine::NAUXGROUP] = {
      launch_grad3_s, launch_grad3_p, launch_grad3_d_pure, launch_grad3_d_cart, launch_grad3_f_pure, launch_grad3_f_cart};
  static const double ncp[NPAIRCLASS] = {1, 3, 9, 6, 18, 36};
  static const int gl[jk_engine::NAUXGROUP] = {0, 1, 2, 2, 3, 3};
  struct Item {
    int g, pc;
    double cost;
  };
  std::vector<Item> items;
  for (int g = 0; g < jk_engine::NAUXGROUP; ++g)
    for (int pc = 0; pc < NPAIRCLASS; ++pc)
      if (counts[g] && e->pcls[pc].npair)
        items.push_back({g, pc, (double)e->pcls[pc].nent * counts[g] * ncp[pc] * (gl[g] + 1) * (gl[g] + 2)});
  std::stable_sort(items.begin(), items.end(), [](const Item& a, const Item& b) { return a.cost > b.cost; });
  ClassStreams cs(e, s);
  LaunchStatus status;
  for (const Item& it : items) {
    Grad3Params P{};
    P.nsm = e->nsm;
    P.aux = aux_group_view(e, shells[it.g], counts[it.g]);
    P.aux_atom = e->daux.atom.p;
    P.atom = e->dobs.atom.p;
    P.ent = entry_view(e->pcls[it.pc]);
    P.pairs = view(e->pcls[it.pc]);
    P.ox = e->dobs.x.p;
    P.oy = e->dobs.y.p;
    P.oz = e->dobs.z.p;
    P.coff = e->dobs.cart_off.p;
    P.sph = e->dobs.sph.p;
    P.boysp = e->boysp.p;
    P.nc = e->obs.n_cart;
    P.W3 = W3;
    P.w3_f0 = w3_f0;
    P.natom = e->natom;
    P.grad = g2e;
    status(launch[it.g](it.pc, P, cs.next(it.cost)));
  }
  cs.join();
  return status.st;
}

// k_grad2 over every ordered pair of fitting groups with the weights W2.
static cudaError_t launch_grad2_all(jk_engine* e, const double* W2, double* g2e, cudaStream_t s) {
  ClassStreams cs(e, s);
  LaunchStatus status;
  for (int gP = jk_engine::NAUXGROUP - 1; gP >= 0; --gP)
    for (int gQ = jk_engine::NAUXGROUP - 1; gQ >= 0; --gQ) {
      if (!e->aux_group_count[gP] || !e->aux_group_count[gQ]) continue;
      Grad2Params P{};
      P.P = aux_group_view(e, e->aux_group[gP].p, e->aux_group_count[gP]);
      P.Q = aux_group_view(e, e->aux_group[gQ].p, e->aux_group_count[gQ]);
      P.aux_atom = e->daux.atom.p;
      P.sph = e->dobs.sph.p;
      P.boysp = e->boysp.p;
      P.naux = e->aux.n_final;
      P.W2 = W2;
      P.grad = g2e;
      status(launch_grad2(gP, gQ, P, cs.next((double)P.P.count * P.Q.count)));
    }
  cs.join();
  return status.st;
}

// Z[P] = W3^P = c_P D - 2 C d^P C^T over Cartesian orbital functions (Cc: nc x o,
// Dc: nc x nc) for w fitting functions with coefficients c and d^P in dd; Y is
// scratch of w nc o elements.
static int w3_block(jk_engine* e, int o, int w, const double* Cc, const double* Dc, const double* dd, const double* c,
                    double* Y, double* Z, cudaStream_t s) {
  const int nc = e->obs.n_cart;
  const size_t ncc = (size_t)nc * nc;
  DGemm y;  // Y[P] = Cc d^P (nc x o)
  y.M = nc; y.N = o; y.K = o; y.batch = w;
  y.A = Cc; y.sam = 1; y.sak = nc;
  y.B = dd; y.sbk = 1; y.sbn = o; y.bsb = (long long)o * o;
  y.C = Y; y.scm = 1; y.scn = nc; y.bsc = (long long)nc * o;
  cudaError_t st = dgemm(y, s);
  if (st != cudaSuccess) return check_cuda(e, st, "DF gradient: Y = C d");
  DGemm z;  // Z[P] = Y[P] Cc^T (nc x nc)
  z.M = nc; z.N = nc; z.K = o; z.batch = w;
  z.A = Y; z.sam = 1; z.sak = nc; z.bsa = (long long)nc * o;
  z.B = Cc; z.sbk = nc; z.sbn = 1;
  z.C = Z; z.scm = 1; z.scn = nc; z.bsc = (long long)ncc;
  if ((st = dgemm(z, s)) != cudaSuccess) return check_cuda(e, st, "DF gradient: Z = Y C^T");
  k_w3<<<(unsigned)((ncc * w + 255) / 256), 256, 0, s>>>(ncc, w, c, Dc, Z);
  return check_cuda(e, cudaGetLastError(), "DF gradient: W3");
}

// W3 and its contraction with the derivative integrals, as many fitting shells
// at a time as the free memory holds (at least 16 functions).
static int grad3_blocks(jk_engine* e, int o, const double* Cc, const double* Dc, const double* dd, const double* c,
                        double* g2e, cudaStream_t s) {
  const int nc = e->obs.n_cart;
  const size_t ncc = (size_t)nc * nc, oo = (size_t)o * o;
  size_t fr = 0, tot = 0;
  dev_mem_info(&fr, &tot);
  const double per_f = 8.0 * ((double)ncc + (double)nc * o);
  const int wmax = (int)std::max(16.0, std::min<double>(e->aux.n_final, 0.6 * (double)fr / per_f));
  DevBuf<double> Y, Z;
  cudaError_t st = Y.alloc((size_t)nc * o * wmax);
  if (st == cudaSuccess) st = Z.alloc(ncc * wmax);
  if (st != cudaSuccess) return check_cuda(e, st, "DF gradient W3 block");
  const HostBasis& ab = e->aux;
  DevBuf<int> lists[jk_engine::NAUXGROUP];
  for (int s0 = 0; s0 < ab.nshell;) {
    int s1 = s0;
    while (s1 < ab.nshell && ab.off_final[s1 + 1] - ab.off_final[s0] <= wmax) ++s1;
    if (s1 == s0) return set_error(e, JK_ERR_ARG, "DF gradient: fitting shell wider than the block");
    const int f0 = ab.off_final[s0], w = ab.off_final[s1] - f0;
    int rc = w3_block(e, o, w, Cc, Dc, dd + (size_t)f0 * oo, c + f0, Y.p, Z.p, s);
    if (rc) return rc;
    std::vector<int> sh[jk_engine::NAUXGROUP];
    for (int k = s0; k < s1; ++k) sh[aux_group_of(ab.l[k], ab.pure[k])].push_back(k);
    const int* shells[jk_engine::NAUXGROUP];
    int counts[jk_engine::NAUXGROUP];
    for (int g = 0; g < jk_engine::NAUXGROUP; ++g) {
      if ((st = lists[g].upload(sh[g], s)) != cudaSuccess) return check_cuda(e, st, "DF gradient shells");
      shells[g] = lists[g].p;
      counts[g] = (int)sh[g].size();
    }
    st = launch_grad3_all(e, shells, counts, Z.p, f0, g2e, s);
    if (st == cudaSuccess) st = cudaStreamSynchronize(s);  // Y, Z and the shell lists are reused by the next block
    if (st != cudaSuccess) return check_cuda(e, st, "DF gradient block");
    s0 = s1;
  }
  return JK_OK;
}

// dC: n x nocc column-major occupied orbitals; dD = 2 C C^T; g2e receives
// the two-electron DF gradient (zeroed here).  Synchronises the stream.
int grad_df_2e_device(jk_engine* e, const double* dC, int nocc, const double* dD, double* g2e, cudaStream_t s) {
  DFState& d = e->df;
  if (e->tiled.metric_ready || (!d.ready && df_use_tiled(e))) return grad_df_2e_tiled(e, dC, nocc, dD, g2e, s);
  const int n = e->obs.n_final, naux = d.naux, o = nocc, na = e->natom;
  for (int k = 0; k < e->aux.nshell; ++k)
    if (e->aux.atom[k] < 0 || e->aux.atom[k] >= na)
      return set_error(e, JK_ERR_ARG, "DF gradient: every fitting shell needs an owning atom (jk_basis.atom)");
  const int nc = e->obs.n_cart;
  const size_t ncc = (size_t)nc * nc;
  if (!d.Linv.p) return set_error(e, JK_ERR_STATE, "DF gradient: L^-1 missing (run jk_df_setup)");
  DevBuf<double> X, bt, c, W2, Z, Cc, Dc, dd, gt;
  cudaError_t st = bt.alloc((size_t)o * o * naux);
  if (st == cudaSuccess) st = c.alloc(naux);
  if (st == cudaSuccess) st = W2.alloc((size_t)naux * naux);
  if (st == cudaSuccess) st = Cc.alloc((size_t)nc * o);
  if (st == cudaSuccess) st = Dc.alloc(ncc);
  if (st == cudaSuccess) st = dd.alloc((size_t)o * o * naux);
  if (st == cudaSuccess) st = gt.alloc(naux);
  // X, later Y, and the whole of W3; where W3 does not fit, it is made in blocks
  // in the place of X
  if (st == cudaSuccess) st = X.alloc((size_t)nc * naux * o);
  if (st == cudaSuccess) st = Z.alloc(ncc * naux);
  const bool whole = st == cudaSuccess;
  if (st == cudaErrorMemoryAllocation) st = X.alloc((size_t)n * naux * o);
  if (st != cudaSuccess) return check_cuda(e, st, "DF gradient allocation");
  auto gemm = [&](const DGemm& g, const char* what) {
    const cudaError_t r = dgemm(g, s);
    return r == cudaSuccess ? JK_OK : check_cuda(e, r, what);
  };
  int rc;
  // X[x][K][i] = sum_y B[x][K][y] C[y][i]
  {
    DGemm g;
    g.M = n * naux; g.N = o; g.K = n;
    g.A = d.B64.p; g.sam = n; g.sak = 1;
    g.B = dC; g.sbk = 1; g.sbn = n;
    g.C = X.p; g.scm = o; g.scn = 1;
    if ((rc = gemm(g, "DF gradient: X = B C"))) return rc;
  }
  // bt[K](i, j) = sum_x X[x][K][i] C[x][j]   (o x o, column-major, per K)
  {
    DGemm g;
    g.M = o; g.N = o; g.K = n; g.batch = naux;
    g.A = X.p; g.sam = 1; g.sak = (long long)naux * o; g.bsa = o;
    g.B = dC; g.sbk = 1; g.sbn = n;
    g.C = bt.p; g.scm = 1; g.scn = o; g.bsc = (long long)o * o;
    if ((rc = gemm(g, "DF gradient: C^T X"))) return rc;
  }
  k_trace_bt<<<(naux + 127) / 128, 128, 0, s>>>(naux, o, bt.p, gt.p);
  // c = L^-T gamma
  {
    DGemm g;
    g.M = naux; g.N = 1; g.K = naux;
    g.A = d.Linv.p; g.sam = naux; g.sak = 1;
    g.B = gt.p; g.sbk = 1; g.sbn = 0;
    g.C = c.p; g.scm = 1; g.scn = 0;
    if ((rc = gemm(g, "DF gradient: c = V^-1 gamma"))) return rc;
  }
  // d (o^2 x naux) = bt L^-1
  {
    DGemm g;
    g.M = o * o; g.N = naux; g.K = naux;
    g.A = bt.p; g.sam = 1; g.sak = (long long)o * o;
    g.B = d.Linv.p; g.sbk = 1; g.sbn = naux; g.b_lower = true;
    g.C = dd.p; g.scm = 1; g.scn = (long long)o * o;
    if ((rc = gemm(g, "DF gradient: d = V^-1 b"))) return rc;
  }
  // W2 = d^T d - 1/2 c c^T
  {
    DGemm g;
    g.M = naux; g.N = naux; g.K = o * o;
    g.A = dd.p; g.sam = (long long)o * o; g.sak = 1;
    g.B = dd.p; g.sbk = 1; g.sbn = (long long)o * o;
    g.C = W2.p; g.scm = 1; g.scn = naux;
    if ((rc = gemm(g, "DF gradient: W2"))) return rc;
    DGemm r;
    r.M = naux; r.N = naux; r.K = 1;
    r.A = c.p; r.sam = 1; r.sak = 0;
    r.B = c.p; r.sbk = 0; r.sbn = 1;
    r.C = W2.p; r.scm = 1; r.scn = naux;
    r.alpha = -0.5; r.beta = 1.0;
    if ((rc = gemm(r, "DF gradient: W2"))) return rc;
  }
  launch_cart_rows(e, o, dC, Cc.p, s);
  launch_final_to_cart(e, dD, Dc.p, s);
  cudaMemsetAsync(g2e, 0, sizeof(double) * 3 * na, s);
  // three-index derivatives
  if (whole) {
    if ((rc = w3_block(e, o, naux, Cc.p, Dc.p, dd.p, c.p, X.p, Z.p, s))) return rc;
    const int* shells[jk_engine::NAUXGROUP];
    for (int g = 0; g < jk_engine::NAUXGROUP; ++g) shells[g] = e->aux_group[g].p;
    st = launch_grad3_all(e, shells, e->aux_group_count, Z.p, 0, g2e, s);
  } else {
    X.reset();
    bt.reset();
    if ((rc = grad3_blocks(e, o, Cc.p, Dc.p, dd.p, c.p, g2e, s))) return rc;
  }
  // metric derivatives
  if (st == cudaSuccess) st = launch_grad2_all(e, W2.p, g2e, s);
  if (st == cudaSuccess) st = cudaStreamSynchronize(s);  // scratch dies on return
  return check_cuda(e, st, "DF gradient kernels");
}

}  // namespace m2

using namespace m2;

extern "C" int jk_grad_df(jk_engine* e, const double* Cocc, int nocc, const double* eps_occ, double* grad,
                          double* grad2e) {
  if (!e || !Cocc || !eps_occ || !grad) return JK_ERR_ARG;
  const int n = e->obs.n_final, na = e->natom;
  if (nocc <= 0 || nocc > n) return set_error(e, JK_ERR_ARG, "jk_grad_df: nocc out of range");
  if (e->df.k0 != 0 || (e->df.k1 >= 0 && e->df.k1 != e->aux.n_final))
    return set_error(e, JK_ERR_STATE, "jk_grad_df needs the whole fitting range (jk_df_set_range)");
  // tiled storage needs only the metric (df_tiled_metric, from the gradient itself)
  if (!e->df.ready && !e->tiled.metric_ready && !df_use_tiled(e)) {
    int rc = df_setup(e);
    if (rc) return rc;
  }
  cudaStream_t s = e->stream;
  DevBuf<double> dC, dCe, dD, dW, g2, g1, dEps;
  cudaError_t st = dC.alloc((size_t)n * nocc);
  if (st == cudaSuccess) st = dCe.alloc((size_t)n * nocc);
  if (st == cudaSuccess) st = dD.alloc((size_t)n * n);
  if (st == cudaSuccess) st = dW.alloc((size_t)n * n);
  if (st == cudaSuccess) st = dEps.alloc(nocc);
  if (st == cudaSuccess) st = g2.alloc(3 * na);
  if (st == cudaSuccess) st = g1.alloc(3 * na);
  if (st == cudaSuccess) st = cudaMemcpyAsync(dC.p, Cocc, sizeof(double) * n * nocc, cudaMemcpyHostToDevice, s);
  if (st == cudaSuccess) st = cudaMemcpyAsync(dEps.p, eps_occ, sizeof(double) * nocc, cudaMemcpyHostToDevice, s);
  if (st != cudaSuccess) return check_cuda(e, st, "jk_grad_df upload");
  // D = 2 C C^T, W = C diag(eps) C^T (src/rhfgrad.cpp:35-38)
  {
    DGemm g;
    g.M = n; g.N = n; g.K = nocc; g.alpha = 2.0;
    g.A = dC.p; g.sam = 1; g.sak = n;
    g.B = dC.p; g.sbk = n; g.sbn = 1;
    g.C = dD.p; g.scm = 1; g.scn = n;
    st = dgemm(g, s);
    if (st == cudaSuccess) {
      k_scale_cols<<<(unsigned)(((size_t)n * nocc + 255) / 256), 256, 0, s>>>(n, nocc, dC.p, dEps.p, dCe.p);
      g.alpha = 1.0;
      g.A = dCe.p;
      g.C = dW.p;
      st = dgemm(g, s);
    }
    if (st != cudaSuccess) return check_cuda(e, st, "jk_grad_df: densities");
  }
  int rc = grad_rhf_device(e, dD.p, dW.p, 0.0, nullptr, g1.p, s, false);
  if (rc) return rc;
  rc = grad_df_2e_device(e, dC.p, nocc, dD.p, g2.p, s);
  if (rc) return rc;
  std::vector<double> h2(3 * na), h1(3 * na), gn;
  st = cudaMemcpy(h2.data(), g2.p, sizeof(double) * 3 * na, cudaMemcpyDeviceToHost);
  if (st == cudaSuccess) st = cudaMemcpy(h1.data(), g1.p, sizeof(double) * 3 * na, cudaMemcpyDeviceToHost);
  if (st != cudaSuccess) return check_cuda(e, st, "jk_grad_df download");
  nuclear_repulsion_grad(e, gn);
  for (int i = 0; i < 3 * na; ++i) grad[i] = h1[i] + h2[i] + gn[i];
  if (grad2e)
    for (int i = 0; i < 3 * na; ++i) grad2e[i] = h2[i];
  return JK_OK;
}

namespace m2 {

// The same gradient for tiled DF storage, where neither B nor (P|mn) is kept:
// one streamed pass gives X'[x][P][i] = sum_y (P|xy) C[y][i] in occupied
// slices, hence b'[P] = C^T (P|..) C and b[K] = sum_P L^-1[K][P] b'[P]; the
// rest follows the unpacked path, with W3 formed and contracted one block of
// fitting shells at a time (W3 for all of them would be n^2 naux doubles).
int grad_df_2e_tiled(jk_engine* e, const double* dC, int nocc, const double* dD, double* g2e, cudaStream_t s) {
  int rc = df_tiled_metric(e);
  if (rc) return rc;
  DFState& d = e->df;
  TiledDF& T = e->tiled;
  const int n = e->obs.n_final, naux = e->aux.n_final, o = nocc, na = e->natom, npad = T.npad;
  const int nc = e->obs.n_cart;
  const size_t ncc = (size_t)nc * nc, oo = (size_t)o * o;
  for (int k = 0; k < e->aux.nshell; ++k)
    if (e->aux.atom[k] < 0 || e->aux.atom[k] >= na)
      return set_error(e, JK_ERR_ARG, "DF gradient: every fitting shell needs an owning atom (jk_basis.atom)");
  DevBuf<double> btp, bt, dd, gt, c, W2, Cp, Tt, Cc, Dc;
  cudaError_t st = btp.alloc(oo * naux);
  if (st == cudaSuccess) st = dd.alloc(oo * naux);
  if (st == cudaSuccess) st = gt.alloc(naux);
  if (st == cudaSuccess) st = c.alloc(naux);
  if (st == cudaSuccess) st = W2.alloc((size_t)naux * naux);
  if (st == cudaSuccess) st = Cp.alloc((size_t)npad * o);
  if (st == cudaSuccess) st = Tt.alloc((size_t)DF_TILE * naux * DF_TILE);
  if (st == cudaSuccess) st = Cc.alloc((size_t)nc * o);
  if (st == cudaSuccess) st = Dc.alloc(ncc);
  if (st != cudaSuccess) return check_cuda(e, st, "tiled DF gradient allocation");
  auto gemm = [&](const DGemm& g, const char* what) {
    const cudaError_t r = dgemm(g, s);
    return r == cudaSuccess ? JK_OK : check_cuda(e, r, what);
  };
  launch_pad_rows(n, npad, o, dC, Cp.p, s);
  {
    size_t fr = 0, tot = 0;
    dev_mem_info(&fr, &tot);
    int oc = (int)std::min<double>(o, std::floor(0.8 * (double)fr / (8.0 * npad * naux)));
    if (oc < 1) return set_error(e, JK_ERR_NOMEM, "tiled DF gradient: no room for X'");
    const int nch = (o + oc - 1) / oc;
    oc = (o + nch - 1) / nch;
    DevBuf<double> X;
    if ((st = X.alloc((size_t)npad * naux * oc)) != cudaSuccess) return check_cuda(e, st, "tiled DF gradient X'");
    for (int ch = 0; ch < nch; ++ch) {
      const int i0 = ch * oc, ocur = std::min(oc, o - i0);
      if ((rc = tiled_xprime_pass(e, Cp.p, i0, ocur, X.p, Tt.p, s, nullptr))) return rc;
      DGemm g;  // b'[P](i, j) = sum_x C[x][i] X'[x][P][j]
      g.M = o; g.N = ocur; g.K = n; g.batch = naux;
      g.A = dC; g.sam = n; g.sak = 1;
      g.B = X.p; g.sbk = (long long)naux * ocur; g.sbn = 1; g.bsb = ocur;
      g.C = btp.p + (size_t)i0 * o; g.scm = 1; g.scn = o; g.bsc = (long long)oo;
      if ((rc = gemm(g, "tiled DF gradient: C^T X'"))) return rc;
    }
  }
  Tt.reset();
  if ((st = bt.alloc(oo * naux)) != cudaSuccess) return check_cuda(e, st, "tiled DF gradient b");
  {
    DGemm g;  // b (o^2 x naux) = b' L^-T
    g.M = (int)oo; g.N = naux; g.K = naux;
    g.A = btp.p; g.sam = 1; g.sak = (long long)oo;
    g.B = d.Linv.p; g.sbk = naux; g.sbn = 1;
    g.C = bt.p; g.scm = 1; g.scn = (long long)oo;
    if ((rc = gemm(g, "tiled DF gradient: b = b' L^-T"))) return rc;
  }
  btp.reset();
  k_trace_bt<<<(naux + 127) / 128, 128, 0, s>>>(naux, o, bt.p, gt.p);
  {
    DGemm g;  // c = L^-T gamma
    g.M = naux; g.N = 1; g.K = naux;
    g.A = d.Linv.p; g.sam = naux; g.sak = 1;
    g.B = gt.p; g.sbk = 1; g.sbn = 0;
    g.C = c.p; g.scm = 1; g.scn = 0;
    if ((rc = gemm(g, "tiled DF gradient: c"))) return rc;
    DGemm h;  // d = b L^-1
    h.M = (int)oo; h.N = naux; h.K = naux;
    h.A = bt.p; h.sam = 1; h.sak = (long long)oo;
    h.B = d.Linv.p; h.sbk = 1; h.sbn = naux; h.b_lower = true;
    h.C = dd.p; h.scm = 1; h.scn = (long long)oo;
    if ((rc = gemm(h, "tiled DF gradient: d"))) return rc;
  }
  bt.reset();
  {
    DGemm g;  // W2 = d^T d - 1/2 c c^T
    g.M = naux; g.N = naux; g.K = (int)oo;
    g.A = dd.p; g.sam = (long long)oo; g.sak = 1;
    g.B = dd.p; g.sbk = 1; g.sbn = (long long)oo;
    g.C = W2.p; g.scm = 1; g.scn = naux;
    if ((rc = gemm(g, "tiled DF gradient: W2"))) return rc;
    DGemm r;
    r.M = naux; r.N = naux; r.K = 1;
    r.A = c.p; r.sam = 1; r.sak = 0;
    r.B = c.p; r.sbk = 0; r.sbn = 1;
    r.C = W2.p; r.scm = 1; r.scn = naux;
    r.alpha = -0.5; r.beta = 1.0;
    if ((rc = gemm(r, "tiled DF gradient: W2"))) return rc;
  }
  launch_cart_rows(e, o, dC, Cc.p, s);
  launch_final_to_cart(e, dD, Dc.p, s);
  cudaMemsetAsync(g2e, 0, sizeof(double) * 3 * na, s);
  if ((rc = grad3_blocks(e, o, Cc.p, Dc.p, dd.p, c.p, g2e, s))) return rc;
  st = launch_grad2_all(e, W2.p, g2e, s);
  if (st == cudaSuccess) st = cudaStreamSynchronize(s);
  return check_cuda(e, st, "tiled DF gradient kernels");
}

}  // namespace m2
