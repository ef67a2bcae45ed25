// engine_eig.cpp -- batched eigensolve of the density-matrix blocks of one truncation:
// the tridiagonal path (one CTA per block, or clusters) for all that it may solve, block Jacobi for
// the rest (with the one-CTA shared-memory Jacobi up to 100 states).
#include <algorithm>

#include "engine.hpp"

namespace dmrg {

namespace {
constexpr int TRID_NMAX[3] = {SYEVT_NMAX, SYEVT_MID_NMAX, SYEVT_RESOLVE_NMAX};   // by path
void check_trid(const std::vector<TridTask>& ts, int64_t nbase, bool vectors) {
  for (const TridTask& t : ts) {
    const int64_t nn = int64_t(t.n) * t.n;
    if (t.n <= 0 || t.n > TRID_NMAX[t.path] || t.a_off < 0 || t.a_off + nn > nbase ||
        t.w_off < 0 || t.w_off + t.n > nbase || t.ws_off < 0 || t.ws_off + 3 * t.n > nbase)
      fail(DMRG_ERR_ARG, "internal plan check failed: tridiagonal eigensolver task");
    if (vectors && (t.keep < 0 || t.keep > t.n || t.u_off < 0 ||
                    t.u_off + int64_t(t.n) * t.keep > nbase))
      fail(DMRG_ERR_ARG, "internal plan check failed: tridiagonal eigenvector task");
  }
}
const TridTask* at(const char* db, size_t off) {
  return reinterpret_cast<const TridTask*>(db + off);
}
}  // namespace

bool fixed_order(const dmrg_params& P, int L, bool tdvp) {
  return split_form(P.precision) != 0 || (!tdvp && P.krylov > FIXED_KRYLOV && L > FIXED_SITES);
}

void set_trid_paths(std::vector<TridTask>& t, bool fixed) {
  int nmax = 0;
  for (const TridTask& x : t) nmax = std::max(nmax, x.n);
  for (TridTask& x : t)
    x.path = fixed ? (x.n <= SYEVT_NMAX ? TRID_SMALL : TRID_BLOCK)
                   : (nmax > SYEVT_ROUTE ? TRID_CLUSTER : TRID_SMALL);
}

void put_trid_values(Upload& u, const std::vector<TridTask>& t, TridValues& v) {
  v = TridValues{};
  for (const TridTask& x : t) {
    v.t[x.path].push_back(x);
    v.nmax[x.path] = std::max(v.nmax[x.path], x.n);
    if (x.path == TRID_CLUSTER) v.sum += x.n;
  }
  // the largest first: not all clusters of a long list are resident at once
  std::stable_sort(v.t[TRID_CLUSTER].begin(), v.t[TRID_CLUSTER].end(),
                   [](const TridTask& a, const TridTask& b) { return a.n > b.n; });
  for (int p = 0; p < 3; ++p) v.off[p] = u.put(v.t[p]);
}

void run_trid_values(dmrg_ctx* c, double* base, int64_t nbase, const TridValues& v, char* db) {
  for (int p = 0; p < 3; ++p) {
    const int n = int(v.t[p].size());
    if (n == 0) continue;
    check_trid(v.t[p], nbase, false);
    const TridTask* tasks = at(db, v.off[p]);
    if (p == TRID_SMALL) launch_trid_eigvals(c->stream, base, tasks, n, v.nmax[p]);
    else if (p == TRID_BLOCK) launch_trid_block_eigvals(c->stream, base, tasks, n, v.nmax[p]);
    else launch_trid_cluster(c->stream, base, tasks, n, v.nmax[p], v.sum);
  }
  cuda_check(cudaGetLastError(), "tridiagonal eigenvalues");
}

void run_trid_vectors(dmrg_ctx* c, double* base, int64_t nbase, std::vector<TridTask> t,
                      int slot) {
  check_trid(t, nbase, true);
  // one launch per path; TRID_BLOCK in two: the blocks whose Gram matrix fits in shared memory
  // beside their vectors, and the rest (which keep the whole L1 for their global-memory Gram)
  std::vector<TridTask> list[4];
  int nmax[4] = {0, 0, 0, 0}, kmax[4] = {0, 0, 0, 0}, nblock = 0;
  for (const TridTask& x : t)
    if (x.keep > 0 && x.path == TRID_BLOCK) nblock = std::max(nblock, x.n);
  const int kg = nblock > 0 ? syevt_block_gram_limit(nblock) : 0;
  int64_t xw = 0;
  for (TridTask x : t) {
    if (x.keep <= 0) continue;
    if (x.path != TRID_SMALL) {
      x.x_off = xw;
      xw += x.path == TRID_BLOCK ? syevt_block_workspace(x.n, x.keep)
                                 : syevt_mid_workspace(x.n, x.keep);
    }
    const int l = x.path == TRID_BLOCK && x.keep > kg ? 3 : x.path;
    list[l].push_back(x);
    nmax[l] = std::max(nmax[l], x.n);
    kmax[l] = std::max(kmax[l], x.keep);
  }
  Upload u;
  size_t off[4];
  bool any = false;
  for (int l = 0; l < 4; ++l) {
    off[l] = u.put(list[l]);
    any |= !list[l].empty();
  }
  if (!any) return;
  if (xw > 0) ensure(c, c->W, xw);
  char* db = u.send(c, slot);
  for (int l = 0; l < 4; ++l) {
    const int n = int(list[l].size());
    if (n == 0) continue;
    const TridTask* tasks = at(db, off[l]);
    if (l == TRID_SMALL) launch_trid_vectors(c->stream, base, tasks, n, nmax[l], kmax[l]);
    else if (l == TRID_CLUSTER)
      launch_trid_mid_vectors(c->stream, base, tasks, n, nmax[l], kmax[l], c->W.p);
    else launch_trid_block_vectors(c->stream, base, tasks, n, nmax[l], kmax[l], c->W.p);
  }
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
