// Integral-direct J/K build (FP64) — the B200 replacement for
// Fock::formJKdirect (molecular2 src/fockbuild.cpp:64-164).
//
// Work decomposition.  Shell pairs (a,b) with l_a >= l_b are grouped into the
// six angular classes ss, ps, pp, ds, dp, dd and, inside a class, sorted by
// their Schwarz bound Q_ab (descending).  A unique shell quartet is a pair of
// pairs {ab, cd}: class(ab) > class(cd), or the same class with index(cd) <=
// index(ab).  Pairs are cut into entries of at most ENTRY_PRIMS primitive pairs
// (quartet.cuh) and the kernels work on entry pairs.  One kernel instantiation
// per class pair (21 for l <= 2), the 21 launches of a build spread longest
// first over the engine's side streams so that they run concurrently.  Because
// kets are Q-sorted, the kets that can pass Q_ab Q_cd Dmax >= precision form a
// prefix found by binary search; each ket then goes through molecular2's
// screen max6(|D| shell blocks) Q_ab Q_cd >= precision (:111-115) before a
// thread takes it.
//
// Digestion follows :121-153 (6 updates with the permutational degeneracy
// factor, symmetrised at the end with the 1/4 of :161-162).  J_ab is shared by
// the whole block and reduced in it before one atomic per element; the other
// five blocks are added per entry pair with FP64 atomics.  Everything runs in the Cartesian representation:
// D is transformed to Cartesian functions first and J, K back afterwards.
#include <algorithm>
#include <cmath>
#include <mutex>
#include <numeric>
#include <string>
#include <vector>

#include "engine.h"
#include "jk_kernels.cuh"

namespace m2 {

PairView view(const PairClassDev& c) { return PairView{c.sa.p, c.sb.p, c.prim_off.p, c.nprim.p, c.Q.p, c.npair}; }

EntryView entry_view(const PairClassDev& c) {
  return EntryView{c.ent_pair.p, c.ent_np.p, c.ent_first.p, c.ent_goff.p, c.ent_prim.p, c.nent};
}

PrimView prim_view(const jk_engine* e) { return PrimView{e->pp_p.p, e->pp_x.p, e->pp_y.p, e->pp_z.p, e->pp_K.p}; }

ShellView shell_view(const jk_engine* e) {
  return ShellView{e->dobs.x.p, e->dobs.y.p, e->dobs.z.p, e->dobs.cart_off.p};
}

// Entries of one sorted class (quartet.cuh): each pair's primitives, largest
// prefactor first, in slices of nearly equal length.
struct HostEntries {
  std::vector<int> pair, np, first;
  std::vector<long long> goff;
  std::vector<double> prim;
};
static void build_entries(const PairClassHost& c, const std::vector<double>* pp, HostEntries& E) {
  const std::vector<double>&p = pp[0], &x = pp[1], &y = pp[2], &z = pp[3], &K = pp[4], &al = pp[5];
  const int np = (int)c.sa.size();
  std::vector<int> order, prims;  // prims: primitive of each (entry, slot), entry by entry
  E.first.resize(np + 1);
  for (int i = 0; i < np; ++i) {
    E.first[i] = (int)E.pair.size();
    const int n = c.nprim[i], ne = (n + ENTRY_PRIMS - 1) / ENTRY_PRIMS;
    order.resize(n);
    std::iota(order.begin(), order.end(), c.prim_off[i]);
    if (n > 1)
      std::stable_sort(order.begin(), order.end(),
                       [&](int u, int v) { return std::fabs(K[u]) * p[v] > std::fabs(K[v]) * p[u]; });
    for (int k = 0, o = 0; k < ne; ++k) {
      const int m = (n - o + (ne - k) - 1) / (ne - k);
      E.pair.push_back(i);
      E.np.push_back(m);
      prims.insert(prims.end(), order.begin() + o, order.begin() + o + m);
      o += m;
    }
  }
  const int nent = (int)E.pair.size();
  E.first[np] = nent;
  E.goff.resize((nent + 31) / 32);
  long long tot = 0;
  for (int g = 0; g < (int)E.goff.size(); ++g) {
    E.goff[g] = tot;
    int mx = 0;
    for (int e = 32 * g; e < std::min(nent, 32 * g + 32); ++e) mx = std::max(mx, E.np[e]);
    tot += (long long)mx * ENTRY_FIELDS * 32;
  }
  E.prim.assign(tot, 0.0);
  const double c2pi = std::sqrt(PI25X2());
  for (int e = 0, o = 0; e < nent; ++e)
    for (int k = 0; k < E.np[e]; ++k, ++o) {
      const int i = prims[o];
      const double f[ENTRY_FIELDS] = {p[i], x[i], y[i], z[i], K[i] * c2pi / p[i], 0.5 / p[i], al[i]};
      double* q = E.prim.data() + E.goff[e / 32] + (long long)k * ENTRY_FIELDS * 32 + e % 32;
      for (int j = 0; j < ENTRY_FIELDS; ++j) q[j * 32] = f[j];
    }
}

// Appends v to a pool and returns its position there.
template <class T>
static size_t append(std::vector<T>& pool, const std::vector<T>& v) {
  const size_t o = pool.size();
  pool.insert(pool.end(), v.begin(), v.end());
  return o;
}

int build_pairs(jk_engine* e) {
  const HostBasis& hb = e->obs;
  std::vector<PairClassHost> cls(NPAIRCLASS);
  for (int la = 0; la <= MAX_L_OBS; ++la)
    for (int lb = 0; lb <= la; ++lb) {
      cls[pair_class(la, lb)].la = la;
      cls[pair_class(la, lb)].lb = lb;
    }
  std::vector<double> pp[6];
  std::vector<double>&pp_p = pp[0], &pp_x = pp[1], &pp_y = pp[2], &pp_z = pp[3], &pp_K = pp[4], &pp_a = pp[5];
  for (int i = 0; i < hb.nshell; ++i)
    for (int j = 0; j < hb.nshell; ++j) {
      const int li = hb.l[i], lj = hb.l[j];
      if (li < lj || (li == lj && j > i)) continue;  // canonical orientation l_a >= l_b
      PairClassHost& c = cls[pair_class(li, lj)];
      const double* A = &hb.xyz[3 * i];
      const double* B = &hb.xyz[3 * j];
      const double AB2 = (A[0] - B[0]) * (A[0] - B[0]) + (A[1] - B[1]) * (A[1] - B[1]) + (A[2] - B[2]) * (A[2] - B[2]);
      int off = (int)pp_p.size(), cnt = 0;
      for (int pa = 0; pa < hb.nprim[i]; ++pa)
        for (int pb = 0; pb < hb.nprim[j]; ++pb) {
          const double al = hb.exps[hb.prim_off[i] + pa], be = hb.exps[hb.prim_off[j] + pb];
          const double p = al + be;
          const double K = hb.coefs[hb.prim_off[i] + pa] * hb.coefs[hb.prim_off[j] + pb] * std::exp(-al * be / p * AB2);
          if (std::fabs(K) < 1e-18) continue;  // contributes below 1e-18 Eh to any integral
          pp_p.push_back(p);
          pp_x.push_back((al * A[0] + be * B[0]) / p);
          pp_y.push_back((al * A[1] + be * B[1]) / p);
          pp_z.push_back((al * A[2] + be * B[2]) / p);
          pp_K.push_back(K);
          pp_a.push_back(al);
          ++cnt;
        }
      if (cnt == 0) continue;  // every primitive product vanishes: the pair cannot contribute
      c.sa.push_back(i);
      c.sb.push_back(j);
      c.prim_off.push_back(off);
      c.nprim.push_back(cnt);
    }
  cudaStream_t s = e->stream;
  cudaError_t st = cudaSuccess;
  if (st == cudaSuccess) st = e->pp_p.upload(pp_p, s);
  if (st == cudaSuccess) st = e->pp_x.upload(pp_x, s);
  if (st == cudaSuccess) st = e->pp_y.upload(pp_y, s);
  if (st == cudaSuccess) st = e->pp_z.upload(pp_z, s);
  if (st == cudaSuccess) st = e->pp_K.upload(pp_K, s);
  if (st == cudaSuccess) st = e->pp_a.upload(pp_a, s);
  if (st != cudaSuccess) return check_cuda(e, st, "upload primitive pairs");

  // Schwarz bounds on the GPU, all classes from one upload
  const int ns = hb.nshell;
  e->schwarz_host.assign((size_t)ns * ns, 0.0);
  e->Qmax = 0.0;
  size_t ntot = 0;
  std::vector<int> ints;
  size_t io[NPAIRCLASS][4], qo[NPAIRCLASS];
  for (int k = 0; k < NPAIRCLASS; ++k) {
    PairClassHost& c = cls[k];
    PairClassDev& d = e->pcls[k];
    d.la = c.la;
    d.lb = c.lb;
    d.npair = (int)c.sa.size();
    io[k][0] = append(ints, c.sa);
    io[k][1] = append(ints, c.sb);
    io[k][2] = append(ints, c.prim_off);
    io[k][3] = append(ints, c.nprim);
    qo[k] = ntot;
    ntot += c.sa.size();
  }
  std::vector<double> Q(ntot);
  if (ntot > 0) {
    DevBuf<int> di;
    DevBuf<double> dq;
    st = di.upload(ints, s);
    if (st == cudaSuccess) st = dq.alloc(ntot);
    if (st != cudaSuccess) return check_cuda(e, st, "upload pairs");
    for (int k = 0; k < NPAIRCLASS; ++k) {
      if (e->pcls[k].npair == 0) continue;
      const PairView v{di.p + io[k][0], di.p + io[k][1], di.p + io[k][2], di.p + io[k][3], nullptr, e->pcls[k].npair};
      SchwarzParams P{v, prim_view(e), shell_view(e), e->dobs.l.p, e->dobs.pure.p, e->dobs.sph.p, e->boysp.p,
                      dq.p + qo[k]};
      if ((st = launch_schwarz(cls[k].la, cls[k].lb, P, s)) != cudaSuccess)
        return check_cuda(e, st, "schwarz launch");
    }
    st = cudaMemcpyAsync(Q.data(), dq.p, ntot * sizeof(double), cudaMemcpyDeviceToHost, s);
    if (st == cudaSuccess) st = cudaStreamSynchronize(s);
    if (st != cudaSuccess) return check_cuda(e, st, "schwarz kernel");
  }

  // sort each class, cut it into entries, and upload everything from one pool per type
  struct Pos {
    size_t sa, sb, off, np, Q, epair, enp, efirst, goff, prim;
  } pos[NPAIRCLASS];
  ints.clear();
  std::vector<double> dbls;
  std::vector<long long> offs;
  for (int k = 0; k < NPAIRCLASS; ++k) {
    PairClassHost& c = cls[k];
    PairClassDev& d = e->pcls[k];
    c.Q.assign(Q.begin() + qo[k], Q.begin() + qo[k] + d.npair);
    // sort the class by Q descending
    std::vector<int> order(d.npair);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return c.Q[x] > c.Q[y]; });
    // inside windows of PAIR_WINDOW, longest contractions first (warps of
    // kets with similar primitive counts; kernels round Q prefixes to windows)
    for (size_t w0 = 0; w0 < order.size(); w0 += PAIR_WINDOW) {
      const size_t w1 = std::min(order.size(), w0 + (size_t)PAIR_WINDOW);
      std::stable_sort(order.begin() + w0, order.begin() + w1,
                       [&](int x, int y) { return c.nprim[x] > c.nprim[y]; });
    }
    PairClassHost sorted;
    for (int o : order) {
      sorted.sa.push_back(c.sa[o]);
      sorted.sb.push_back(c.sb[o]);
      sorted.prim_off.push_back(c.prim_off[o]);
      sorted.nprim.push_back(c.nprim[o]);
      sorted.Q.push_back(c.Q[o]);
      e->schwarz_host[(size_t)c.sa[o] * ns + c.sb[o]] = c.Q[o];
      e->schwarz_host[(size_t)c.sb[o] * ns + c.sa[o]] = c.Q[o];
      e->Qmax = std::max(e->Qmax, c.Q[o]);
    }
    HostEntries E;
    build_entries(sorted, pp, E);
    d.nent = (int)E.pair.size();
    pos[k] = Pos{append(ints, sorted.sa), append(ints, sorted.sb), append(ints, sorted.prim_off),
                 append(ints, sorted.nprim), append(dbls, sorted.Q), append(ints, E.pair), append(ints, E.np),
                 append(ints, E.first), append(offs, E.goff), 0};
    dbls.resize((dbls.size() + 31) / 32 * 32);  // a warp's 32 doubles start on a 256-byte boundary
    pos[k].prim = append(dbls, E.prim);
  }
  st = e->pair_ints.upload(ints, s);
  if (st == cudaSuccess) st = e->pair_dbls.upload(dbls, s);
  if (st == cudaSuccess) st = e->pair_offs.upload(offs, s);
  if (st == cudaSuccess) st = cudaStreamSynchronize(s);  // host vectors die on return
  if (st != cudaSuccess) return check_cuda(e, st, "upload sorted pairs");
  for (int k = 0; k < NPAIRCLASS; ++k) {
    PairClassDev& d = e->pcls[k];
    const Pos& o = pos[k];
    int* pi = e->pair_ints.p;
    d.sa.p = pi + o.sa;
    d.sb.p = pi + o.sb;
    d.prim_off.p = pi + o.off;
    d.nprim.p = pi + o.np;
    d.Q.p = e->pair_dbls.p + o.Q;
    d.ent_pair.p = pi + o.epair;
    d.ent_np.p = pi + o.enp;
    d.ent_first.p = pi + o.efirst;
    d.ent_goff.p = e->pair_offs.p + o.goff;
    d.ent_prim.p = e->pair_dbls.p + o.prim;
  }
  return JK_OK;
}

// Ket entries per block: many, so that the bra set-up (Boys table, term
// products) is shared, but fewer for classes whose blocks would not fill the
// GPU otherwise.
static int ket_chunk(long long nbra, long long nket, int layers, int nsm) {
  int k = 4 * JK_LIST;
  nbra = std::max(nbra, 1LL);  // a rank's share of few entries; the grid's y limit is 65,535
  while (k > 32 && nbra * ((nket + k - 1) / k) * layers < (k > JK_THREADS ? 32 : 8) * nsm) k /= 2;
  return k;
}

// Rough relative cost of one class launch (Cartesian products of the pair
// classes ss ps pp ds dp dd times the pair counts): orders the launches
// longest first over the side streams.
static double class_cost(int A, int B, int nbra, int nket) {
  static const double ncp[6] = {1, 3, 9, 6, 18, 36};
  return (double)nbra * nket * ncp[A] * ncp[B] * (A == B ? 0.5 : 1.0);
}

// Every (bra class, ket class) launch of one build, longest first, spread over
// the engine's side streams so that the small d classes run beside the large
// ones instead of one after another; J, K and the counters are accumulated
// with atomics, so the launches commute.
template <class Launch>
static cudaError_t launch_classes(jk_engine* e, cudaStream_t s, Launch&& launch) {
  struct Item {
    int A, B;
    double cost;
  };
  std::vector<Item> items;
  for (int A = 0; A < NPAIRCLASS; ++A)
    for (int B = 0; B <= A; ++B)
      if (e->pcls[A].npair && e->pcls[B].npair)
        items.push_back({A, B, class_cost(A, B, e->pcls[A].npair, e->pcls[B].npair)});
  std::stable_sort(items.begin(), items.end(), [](const Item& a, const Item& b) { return a.cost > b.cost; });
  ClassStreams cs(e, s);
  LaunchStatus status;
  for (const Item& it : items) status(launch(it.A, it.B, cs.next(it.cost)));
  cs.join();
  return status.st;
}

static cudaError_t launch_jk(const jk_engine* e, int A, int B, const JKParams& Pin, cudaStream_t s) {
  JKParams P = Pin;
  const PairClassDev &ca = e->pcls[A], &cb = e->pcls[B];
  int nb = 0;
  bra_share(e, ca.npair, P.bra0, P.bra_step, nb);
  if (nb == 0) return cudaSuccess;
  P.bra = view(ca);
  P.ket = view(cb);
  P.bra_ent = entry_view(ca);
  P.ket_ent = entry_view(cb);
  P.same_class = (A == B);
  P.kchunk = ket_chunk((long long)ca.nent / P.bra_step, cb.nent, jk_layers(ca.la, ca.lb, cb.la, cb.lb), e->nsm);
  dim3 grid(ca.nent, (cb.nent + P.kchunk - 1) / P.kchunk);
  if (A <= 2) return launch_jk_bra_s(A, B, P, grid, s);
  if (A == 3) return launch_jk_bra_ds(B, P, grid, s);
  if (A == 4) return launch_jk_bra_dp(B, P, grid, s);
  return B < 4 ? launch_jk_bra_dd_lo(B, P, grid, s) : launch_jk_bra_dd_hi(B, P, grid, s);
}

int direct_jk_device(jk_engine* e, const double* dD, double precision, double mult, double* dJ, double* dK,
                     cudaStream_t s) {
  const int nc = e->obs.n_cart, ns = e->obs.nshell;
  cudaError_t st = cudaSuccess;
  if (st == cudaSuccess) st = e->Dcart.alloc((size_t)nc * nc);
  if (st == cudaSuccess) st = e->Jcart.alloc((size_t)nc * nc);
  if (st == cudaSuccess) st = e->Kcart.alloc((size_t)nc * nc);
  if (st == cudaSuccess) st = e->Dnorm.alloc((size_t)ns * ns);
  if (st == cudaSuccess) st = e->Dmax.alloc(2);
  if (st != cudaSuccess) return check_cuda(e, st, "jk_direct scratch");
  launch_shell_norms(e, dD, e->Dnorm.p, e->Dmax.p, s);
  launch_final_to_cart(e, dD, e->Dcart.p, s);
  cudaMemsetAsync(e->Jcart.p, 0, sizeof(double) * nc * nc, s);
  cudaMemsetAsync(e->Kcart.p, 0, sizeof(double) * nc * nc, s);
  unsigned long long* counter = reinterpret_cast<unsigned long long*>(e->Dmax.p + 1);
  e->last_counter = counter;
  cudaMemsetAsync(counter, 0, sizeof(unsigned long long), s);
  if ((st = e->class_work.alloc(3 * NPAIRCLASS * NPAIRCLASS)) != cudaSuccess)
    return check_cuda(e, st, "jk_direct work counters");
  cudaMemsetAsync(e->class_work.p, 0, sizeof(unsigned long long) * 3 * NPAIRCLASS * NPAIRCLASS, s);
  e->class_work_valid = true;
  JKParams P{};
  P.sh = shell_view(e);
  P.Dnorm = e->Dnorm.p;
  P.nshell = ns;
  P.Dmax = e->Dmax.p;
  P.nden = 1;
  P.Dc = e->Dcart.p;
  P.nc = nc;
  P.Jc = e->Jcart.p;
  P.Kc = e->Kcart.p;
  P.dstride = (size_t)nc * nc;
  P.precision = precision;
  P.eps = prim_eps(precision);
  P.boysp = e->boysp.p;
  P.counter = counter;
  const cudaError_t launched = launch_classes(e, s, [&](int A, int B, cudaStream_t cs) {
    JKParams Q = P;
    Q.work = e->class_work.p + 3 * (A * NPAIRCLASS + B);
    return launch_jk(e, A, B, Q, cs);
  });
  // J = 1/4 (J + J^T) mult, K = 1/2 * 1/4 (K + K^T) mult  (src/fockbuild.cpp:146-149, 161-162)
  launch_cart_to_final_sym(e, e->Jcart.p, 0.25 * mult, dJ, s);
  launch_cart_to_final_sym(e, e->Kcart.p, 0.125 * mult, dK, s);
  return check_cuda(e, launched != cudaSuccess ? launched : cudaGetLastError(), "jk_direct launch");
}

// J and K of two densities (UHF alpha and beta) from one pass over the shell
// quartets: UnrestrictedFock::formJKdirect (src/fockbuild.cpp:266-362), which
// screens with the shell-block norms of Da + Db and digests both densities from
// each integral batch.  Each J, K is w.r.t. its own full density.
int direct_jk_uhf_device(jk_engine* e, const double* dDa, const double* dDb, double precision, double mult,
                         double* dJa, double* dJb, double* dKa, double* dKb, cudaStream_t s) {
  const int n = e->obs.n_final, nc = e->obs.n_cart, ns = e->obs.nshell;
  const size_t ncc = (size_t)nc * nc, nn = (size_t)n * n;
  DevBuf<double> Dsum, Dc2, Jc2, Kc2;
  cudaError_t st = Dsum.alloc(nn);
  if (st == cudaSuccess) st = Dc2.alloc(2 * ncc);
  if (st == cudaSuccess) st = Jc2.alloc(2 * ncc);
  if (st == cudaSuccess) st = Kc2.alloc(2 * ncc);
  if (st == cudaSuccess) st = e->Dnorm.alloc((size_t)ns * ns);
  if (st == cudaSuccess) st = e->Dmax.alloc(2);
  if (st != cudaSuccess) return check_cuda(e, st, "jk_direct_uhf scratch");
  launch_add(dDa, dDb, Dsum.p, nn, s);
  launch_shell_norms(e, Dsum.p, e->Dnorm.p, e->Dmax.p, s);
  launch_final_to_cart(e, dDa, Dc2.p, s);
  launch_final_to_cart(e, dDb, Dc2.p + ncc, s);
  cudaMemsetAsync(Jc2.p, 0, sizeof(double) * 2 * ncc, s);
  cudaMemsetAsync(Kc2.p, 0, sizeof(double) * 2 * ncc, s);
  unsigned long long* counter = reinterpret_cast<unsigned long long*>(e->Dmax.p + 1);
  e->last_counter = counter;
  cudaMemsetAsync(counter, 0, sizeof(unsigned long long), s);
  JKParams P{};
  P.sh = shell_view(e);
  P.Dnorm = e->Dnorm.p;
  P.nshell = ns;
  P.Dmax = e->Dmax.p;
  P.nden = 2;
  P.Dc = Dc2.p;
  P.nc = nc;
  P.Jc = Jc2.p;
  P.Kc = Kc2.p;
  P.dstride = ncc;
  P.precision = precision;
  P.eps = prim_eps(precision);
  P.boysp = e->boysp.p;
  P.counter = counter;
  if ((st = e->class_work.alloc(3 * NPAIRCLASS * NPAIRCLASS)) != cudaSuccess)
    return check_cuda(e, st, "jk_direct_uhf work counters");
  cudaMemsetAsync(e->class_work.p, 0, sizeof(unsigned long long) * 3 * NPAIRCLASS * NPAIRCLASS, s);
  e->class_work_valid = true;
  const cudaError_t launched = launch_classes(e, s, [&](int A, int B, cudaStream_t cs) {
    JKParams Q = P;
    Q.work = e->class_work.p + 3 * (A * NPAIRCLASS + B);
    return launch_jk(e, A, B, Q, cs);
  });
  launch_cart_to_final_sym(e, Jc2.p, 0.25 * mult, dJa, s);
  launch_cart_to_final_sym(e, Jc2.p + ncc, 0.25 * mult, dJb, s);
  launch_cart_to_final_sym(e, Kc2.p, 0.125 * mult, dKa, s);
  launch_cart_to_final_sym(e, Kc2.p + ncc, 0.125 * mult, dKb, s);
  st = launched != cudaSuccess ? launched : cudaGetLastError();
  if (st == cudaSuccess) st = cudaStreamSynchronize(s);  // the scratch dies on return
  return check_cuda(e, st, "jk_direct_uhf");
}

// ---------------------------------------------------------------- no-allocation variant
// Scratch of jk_direct_noalloc: one fixed array in device global memory.  Every
// GPU that loads this library holds it (6.8 MB) until the process exits, and
// every call on a device shares it.  Layout (in doubles): Cartesian D, J, K
// (NOALLOC_MAX_CART^2 each), the shell-block norms (NOALLOC_MAX_SHELLS^2), then
// Dmax and the quartet counter.
constexpr int NOALLOC_MAX_CART = 512;
constexpr int NOALLOC_MAX_SHELLS = 256;
constexpr size_t NOALLOC_CC = (size_t)NOALLOC_MAX_CART * NOALLOC_MAX_CART;
constexpr size_t NOALLOC_SS = (size_t)NOALLOC_MAX_SHELLS * NOALLOC_MAX_SHELLS;
constexpr size_t NOALLOC_DOUBLES = 3 * NOALLOC_CC + NOALLOC_SS + 2;
static __device__ __align__(256) double g_noalloc_scratch[NOALLOC_DOUBLES];

// Device address of the scratch array on `device`, looked up once per device
// with that device current (the host-side symbol is not a device address).
static cudaError_t noalloc_scratch(int device, double** out) {
  static std::mutex mu;
  static std::vector<double*> addr;
  std::lock_guard<std::mutex> lock(mu);
  if ((int)addr.size() <= device) addr.resize(device + 1, nullptr);
  if (!addr[device]) {
    int prev = -1;
    cudaError_t st = cudaGetDevice(&prev);
    if (st == cudaSuccess && prev != device) st = cudaSetDevice(device);
    double* p = nullptr;
    if (st == cudaSuccess) st = cudaGetSymbolAddress((void**)&p, g_noalloc_scratch);
    if (prev >= 0 && prev != device) cudaSetDevice(prev);
    if (st != cudaSuccess) return st;
    addr[device] = p;
  }
  *out = addr[device];
  return cudaSuccess;
}

int direct_jk_noalloc(jk_engine* e, const double* dD, double precision, double mult, double* dJ, double* dK,
                      cudaStream_t s) {
  const int nc = e->obs.n_cart, ns = e->obs.nshell;
  if (nc > NOALLOC_MAX_CART || ns > NOALLOC_MAX_SHELLS)
    return set_error(e, JK_ERR_ARG,
                     "jk_direct_noalloc: basis too large for the fixed scratch (" + std::to_string(nc) +
                         " Cartesian functions, max " + std::to_string(NOALLOC_MAX_CART) + "; " + std::to_string(ns) +
                         " shells, max " + std::to_string(NOALLOC_MAX_SHELLS) + "); use jk_direct_device");
  // the array's address is per device: launching on another GPU than the
  // engine's would hand its kernels a foreign address
  int cur = -1;
  cudaError_t st = cudaGetDevice(&cur);
  if (st != cudaSuccess) return check_cuda(e, st, "jk_direct_noalloc: cudaGetDevice");
  if (cur != e->device)
    return set_error(e, JK_ERR_ARG,
                     "jk_direct_noalloc: the current CUDA device (" + std::to_string(cur) +
                         ") is not the engine's device (" + std::to_string(e->device) + ")");
  double* base = nullptr;
  st = noalloc_scratch(e->device, &base);
  if (st != cudaSuccess) return check_cuda(e, st, "jk_direct_noalloc: cudaGetSymbolAddress");
  double* Dc = base;
  double* Jc = base + NOALLOC_CC;
  double* Kc = base + 2 * NOALLOC_CC;
  double* Dn = base + 3 * NOALLOC_CC;
  double* Dmax = Dn + NOALLOC_SS;
  unsigned long long* counter = reinterpret_cast<unsigned long long*>(Dmax + 1);
  e->last_counter = counter;
  e->class_work_valid = false;  // this build keeps no per-class counters
  // the array keeps the previous call's contents: clear the accumulators
  launch_shell_norms(e, dD, Dn, Dmax, s);  // zeroes Dmax itself
  launch_final_to_cart(e, dD, Dc, s);
  cudaMemsetAsync(Jc, 0, sizeof(double) * nc * nc, s);
  cudaMemsetAsync(Kc, 0, sizeof(double) * nc * nc, s);
  cudaMemsetAsync(counter, 0, sizeof(unsigned long long), s);
  JKParams P{};
  P.sh = shell_view(e);
  P.Dnorm = Dn;
  P.nshell = ns;
  P.Dmax = Dmax;
  P.nden = 1;
  P.Dc = Dc;
  P.nc = nc;
  P.Jc = Jc;
  P.Kc = Kc;
  P.precision = precision;
  P.eps = prim_eps(precision);
  P.boysp = e->boysp.p;
  P.counter = counter;
  P.dstride = NOALLOC_CC;
  const cudaError_t launched = launch_classes(e, s, [&](int A, int B, cudaStream_t cs) {
    return launch_jk(e, A, B, P, cs);
  });
  launch_cart_to_final_sym(e, Jc, 0.25 * mult, dJ, s);
  launch_cart_to_final_sym(e, Kc, 0.125 * mult, dK, s);
  return check_cuda(e, launched != cudaSuccess ? launched : cudaGetLastError(), "jk_direct_noalloc launch");
}

}  // namespace m2

using namespace m2;

extern "C" {

int jk_direct_uhf_device(jk_engine* e, const double* dDa, const double* dDb, double precision, double multiplier,
                         double* dJa, double* dJb, double* dKa, double* dKb, void* stream) {
  if (!e || !dDa || !dDb || !dJa || !dJb || !dKa || !dKb) return JK_ERR_ARG;
  if (!(precision >= 0.0)) return set_error(e, JK_ERR_ARG, "jk_direct_uhf: precision must be >= 0");
  PartitionScope part(e);
  return direct_jk_uhf_device(e, dDa, dDb, precision, multiplier, dJa, dJb, dKa, dKb,
                              stream ? (cudaStream_t)stream : e->stream);
}

int jk_direct_uhf(jk_engine* e, const double* Da, const double* Db, double precision, double multiplier, double* Ja,
                  double* Jb, double* Ka, double* Kb) {
  if (!e || !Da || !Db || !Ja || !Jb || !Ka || !Kb) return JK_ERR_ARG;
  const int n = e->obs.n_final;
  const size_t nn = (size_t)n * n, bytes = sizeof(double) * nn;
  DevBuf<double> d;
  cudaError_t st = d.alloc(6 * nn);
  if (st == cudaSuccess) st = cudaMemcpyAsync(d.p, Da, bytes, cudaMemcpyHostToDevice, e->stream);
  if (st == cudaSuccess) st = cudaMemcpyAsync(d.p + nn, Db, bytes, cudaMemcpyHostToDevice, e->stream);
  if (st != cudaSuccess) return check_cuda(e, st, "jk_direct_uhf upload");
  int rc = jk_direct_uhf_device(e, d.p, d.p + nn, precision, multiplier, d.p + 2 * nn, d.p + 3 * nn, d.p + 4 * nn,
                                d.p + 5 * nn, nullptr);
  if (rc) return rc;
  double* outs[4] = {Ja, Jb, Ka, Kb};
  for (int k = 0; k < 4 && st == cudaSuccess; ++k)
    st = cudaMemcpyAsync(outs[k], d.p + (2 + k) * nn, bytes, cudaMemcpyDeviceToHost, e->stream);
  if (st == cudaSuccess) st = cudaStreamSynchronize(e->stream);
  return check_cuda(e, st, "jk_direct_uhf download");
}

int jk_last_class_work(const jk_engine* e, long long* out, int nmax, int* nwritten) {
  if (!e || !out || !nwritten) return JK_ERR_ARG;
  *nwritten = 0;
  if (!e->class_work_valid || !e->class_work.p) return JK_ERR_STATE;
  std::vector<unsigned long long> h(3 * NPAIRCLASS * NPAIRCLASS);
  if (cudaMemcpyAsync(h.data(), e->class_work.p, h.size() * sizeof(h[0]), cudaMemcpyDeviceToHost, e->stream) !=
          cudaSuccess ||
      cudaStreamSynchronize(e->stream) != cudaSuccess)
    return JK_ERR_CUDA;
  const int k = std::min<int>(nmax, (int)h.size());
  for (int i = 0; i < k; ++i) out[i] = (long long)h[i];
  *nwritten = k;
  return JK_OK;
}

int jk_direct_noalloc(jk_engine* e, const double* dD, double precision, double multiplier, double* dJ, double* dK,
                      void* stream) {
  if (!e || !dD || !dJ || !dK) return JK_ERR_ARG;
  if (!(precision >= 0.0)) return set_error(e, JK_ERR_ARG, "jk_direct_noalloc: precision must be >= 0");
  cudaStream_t s = stream ? (cudaStream_t)stream : e->stream;
  PartitionScope part(e);
  return direct_jk_noalloc(e, dD, precision, multiplier, dJ, dK, s);
}

int jk_direct_device(jk_engine* e, const double* dD, double precision, double multiplier, double* dJ, double* dK,
                     void* stream) {
  if (!e || !dD || !dJ || !dK) return JK_ERR_ARG;
  if (!(precision >= 0.0)) return set_error(e, JK_ERR_ARG, "jk_direct: precision must be >= 0");
  cudaStream_t s = stream ? (cudaStream_t)stream : e->stream;
  PartitionScope part(e);
  return direct_jk_device(e, dD, precision, multiplier, dJ, dK, s);
}

int jk_direct_set_partition(jk_engine* e, int rank, int nranks) {
  if (!e) return JK_ERR_ARG;
  if (nranks < 1 || rank < 0 || rank >= nranks)
    return set_error(e, JK_ERR_ARG, "jk_direct_set_partition: need 0 <= rank < nranks");
  e->part_rank = rank;
  e->part_size = nranks;
  return JK_OK;
}

int jk_direct(jk_engine* e, const double* D, double precision, double multiplier, double* J, double* K) {
  if (!e || !D || !J || !K) return JK_ERR_ARG;
  const int n = e->obs.n_final;
  const size_t bytes = sizeof(double) * n * n;
  cudaError_t st = cudaSuccess;
  if (st == cudaSuccess) st = e->Dfinal.alloc((size_t)n * n);
  if (st == cudaSuccess) st = e->Jfinal.alloc((size_t)n * n);
  if (st == cudaSuccess) st = e->Kfinal.alloc((size_t)n * n);
  if (st == cudaSuccess) st = cudaMemcpyAsync(e->Dfinal.p, D, bytes, cudaMemcpyHostToDevice, e->stream);
  if (st != cudaSuccess) return check_cuda(e, st, "jk_direct upload");
  int rc = jk_direct_device(e, e->Dfinal.p, precision, multiplier, e->Jfinal.p, e->Kfinal.p, nullptr);
  if (rc) return rc;
  st = cudaMemcpyAsync(J, e->Jfinal.p, bytes, cudaMemcpyDeviceToHost, e->stream);
  if (st == cudaSuccess) st = cudaMemcpyAsync(K, e->Kfinal.p, bytes, cudaMemcpyDeviceToHost, e->stream);
  if (st == cudaSuccess) st = cudaStreamSynchronize(e->stream);
  return check_cuda(e, st, "jk_direct download");
}

}  // extern "C"
