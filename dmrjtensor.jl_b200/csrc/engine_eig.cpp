// engine_eig.cpp -- batched eigensolve of the density-matrix blocks of one truncation:
// the tridiagonal path (one CTA per block, or clusters) for all that it may solve, block Jacobi for
// the rest (with the one-CTA shared-memory Jacobi up to 100 states).
#include <algorithm>

#include "engine.hpp"

namespace dmrg {

namespace {
void check_trid(const std::vector<TridTask>& ts, int64_t nbase, bool vectors) {
  for (const TridTask& t : ts) {
    const int64_t nn = int64_t(t.n) * t.n;
    if (t.n <= 0 || t.n > (t.mid ? SYEVT_MID_NMAX : SYEVT_NMAX) || t.a_off < 0 || t.a_off + nn > nbase ||
        t.w_off < 0 || t.w_off + t.n > nbase || t.ws_off < 0 || t.ws_off + 3 * t.n > nbase)
      fail(DMRG_ERR_ARG, "internal plan check failed: tridiagonal eigensolver task");
    if (vectors && (t.keep < 0 || t.keep > t.n || t.u_off < 0 ||
                    t.u_off + int64_t(t.n) * t.keep > nbase))
      fail(DMRG_ERR_ARG, "internal plan check failed: tridiagonal eigenvector task");
  }
}
}  // namespace

void set_trid_paths(std::vector<TridTask>& t) {
  int nmax = 0;
  for (const TridTask& x : t) nmax = std::max(nmax, x.n);
  for (TridTask& x : t) x.mid = nmax > SYEVT_ROUTE ? 1 : 0;
}

void put_trid_values(Upload& u, const std::vector<TridTask>& t, TridValues& v) {
  v = TridValues{};
  for (const TridTask& x : t) {
    if (!x.mid) { v.small.push_back(x); v.ns = std::max(v.ns, x.n); }
    else { v.mid.push_back(x); v.sum += x.n; }
  }
  // the largest first: not all clusters of a long list are resident at once
  std::stable_sort(v.mid.begin(), v.mid.end(),
                   [](const TridTask& a, const TridTask& b) { return a.n > b.n; });
  v.o_small = u.put(v.small);
  v.o_mid = u.put(v.mid);
}

void run_trid_values(dmrg_ctx* c, double* base, int64_t nbase, const TridValues& v, char* db) {
  check_trid(v.small, nbase, false);
  check_trid(v.mid, nbase, false);
  if (!v.small.empty())
    launch_trid_eigvals(c->stream, base, reinterpret_cast<const TridTask*>(db + v.o_small),
                        int(v.small.size()), v.ns);
  if (!v.mid.empty())
    launch_trid_cluster(c->stream, base, reinterpret_cast<const TridTask*>(db + v.o_mid),
                        int(v.mid.size()), v.mid[0].n, v.sum);
  cuda_check(cudaGetLastError(), "tridiagonal eigenvalues");
}

void run_trid_vectors(dmrg_ctx* c, double* base, int64_t nbase, std::vector<TridTask> t,
                      int slot) {
  check_trid(t, nbase, true);
  std::vector<TridTask> small, mid;
  int ns = 0, ks = 0, nm = 0, km = 0;
  int64_t xw = 0;
  for (TridTask x : t) {
    if (x.keep <= 0) continue;
    if (!x.mid) {
      small.push_back(x);
      ns = std::max(ns, x.n);
      ks = std::max(ks, x.keep);
    } else {
      x.x_off = xw;
      xw += syevt_mid_workspace(x.n, x.keep);
      mid.push_back(x);
      nm = std::max(nm, x.n);
      km = std::max(km, x.keep);
    }
  }
  if (small.empty() && mid.empty()) return;
  if (xw > 0) ensure(c, c->W, xw);
  Upload u;
  const size_t o1 = u.put(small), o2 = u.put(mid);
  char* db = u.send(c, slot);
  if (!small.empty())
    launch_trid_vectors(c->stream, base, reinterpret_cast<const TridTask*>(db + o1),
                        int(small.size()), ns, ks);
  if (!mid.empty())
    launch_trid_mid_vectors(c->stream, base, reinterpret_cast<const TridTask*>(db + o2),
                            int(mid.size()), nm, km, c->W.p);
  cuda_check(cudaGetLastError(), "tridiagonal eigenvectors");
}

int64_t eig_workspace(const std::vector<EigTask>& tasks) {
  int64_t ws = 0;
  for (const EigTask& t : tasks) {
    if (t.n <= 100) continue;
    const int64_t N = block_eig_padded(t.n);
    ws += 2 * N * N + N * 32;
  }
  return ws;
}

void run_eigs(dmrg_ctx* c, double* base, int64_t nbase, const std::vector<EigTask>& tasks,
              int64_t ws_off, int* sweeps) {
  if (sweeps) *sweeps = 0;
  if (tasks.empty()) return;   // nothing to solve: no status read, no synchronisation
  std::vector<EigTask> small;
  std::vector<BlockEigGroup> big;
  int nsmall = 0, maxN = 0, maxn = 0;
  int64_t ws = ws_off;
  for (const EigTask& t : tasks) {
    if (t.n <= 0) continue;
    if (t.n <= 100) {
      small.push_back(t);
      nsmall = std::max(nsmall, t.n);
      continue;
    }
    BlockEigGroup g{};
    g.a_off = t.a_off;
    g.w_off = t.w_off;
    g.n = t.n;
    g.N = block_eig_padded(t.n);
    g.ap_off = ws;
    g.vp_off = ws + int64_t(g.N) * g.N;
    g.q_off = ws + 2 * int64_t(g.N) * g.N;
    ws += 2 * int64_t(g.N) * g.N + int64_t(g.N) * 32;
    maxN = std::max(maxN, g.N);
    maxn = std::max(maxn, g.n);
    big.push_back(g);
  }
  check_eig(small, nbase);
  if (ws > nbase) fail(DMRG_ERR_ARG, "internal plan check failed: eigensolver workspace");
  for (const BlockEigGroup& g : big) {
    EigTask t{g.a_off, g.a_off, g.w_off, g.n, 0};
    check_eig({t}, nbase);
  }
  if (int(big.size()) > c->max_groups) fail(DMRG_ERR_SHAPE, "too many large density-matrix blocks");
  if (!small.empty()) {
    Upload u;
    const size_t off = u.put(small);
    char* db = u.send(c, 4);
    cuda_check(cudaMemsetAsync(c->d_status, 0, sizeof(int), c->stream), "status");
    launch_jacobi(c->stream, base, reinterpret_cast<const EigTask*>(db + off), int(small.size()),
                  nsmall, c->d_status);
  }
  if (!big.empty()) {
    std::vector<int2> pairs;
    std::vector<int4> tiles;
    for (int gi = 0; gi < int(big.size()); ++gi) {
      const int nb = big[gi].N / 16, np = nb / 2;
      for (int k = 0; k < np; ++k) pairs.push_back(make_int2(gi, k));
      for (int P = 0; P < np; ++P)
        for (int Q = 0; Q < np; ++Q) tiles.push_back(make_int4(gi, 0, P, Q));
      for (int rc = 0; rc < big[gi].N / 32; ++rc)
        for (int P = 0; P < np; ++P) tiles.push_back(make_int4(gi, 1, rc, P));
    }
    Upload u;
    const size_t go = u.put(big), po = u.put(pairs), to = u.put(tiles);
    char* db = u.send(c, 5);
    BlockEigPlan pl{};
    pl.groups = reinterpret_cast<const BlockEigGroup*>(db + go);
    pl.ngroups = int(big.size());
    pl.pairs = reinterpret_cast<const int2*>(db + po);
    pl.npairs = int(pairs.size());
    pl.tiles = reinterpret_cast<const int4*>(db + to);
    pl.ntiles = int(tiles.size());
    pl.maxN = maxN;
    pl.maxn = maxn;
    pl.max_sweeps = 30;
    int sw = 0;
    cuda_check(cudaGetLastError(), "block Jacobi set-up");
    launch_block_jacobi(c->stream, base, pl, c->d_flags, c->h_flags, c->d_floors, &sw);
    cuda_check(cudaGetLastError(), "block Jacobi");
    if (sweeps) *sweeps = sw;
    if (sw >= pl.max_sweeps) fail(DMRG_ERR_CUDA, "block Jacobi eigensolver did not converge");
  }
  int stat = 0;
  cuda_check(cudaMemcpyAsync(&stat, c->d_status, sizeof(int), cudaMemcpyDeviceToHost, c->stream),
             "status");
  cuda_check(cudaStreamSynchronize(c->stream), "eigen sync");
  cuda_check(cudaGetLastError(), "eigensolve");
  if (!small.empty() && stat != 0) fail(DMRG_ERR_CUDA, "Jacobi eigensolver did not converge");
}

}  // namespace dmrg
