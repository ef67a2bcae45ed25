// syevt_mid.cu -- eigenvectors of the density-matrix blocks of a step whose largest has more than
// SYEVT_ROUTE (up to SYEVT_MID_NMAX) states (their tridiagonal matrices and eigenvalues come from
// syevt_cluster.cu). Every part runs on many CTAs; one CTA per block for all of it took 1.6 + 0.54 ms
// at n = 345 with 200 kept vectors.
//   * k_mid_invit: inverse iteration, one thread per kept vector, a few vectors per CTA so that
//     their LU factors and the vectors stay in shared memory (with 32 vectors per CTA and the
//     factors in global memory 290 us at n = 345). Bound by the latency of the recurrences.
//   * k_mid_runs: vectors of (nearly) equal eigenvalues, which come out as independent but not
//     orthogonal vectors of their common eigenspace, are orthonormalised among themselves.
//   * up to three rounds of k_mid_gram and k_mid_apply: G = Z^T Z = I + E with a small E (vectors
//     of separated eigenvalues are orthogonal to eps ||A|| / gap), then Z <- Z (I - E_up), E_up =
//     the strict upper triangle and half the diagonal of E: the first-order Cholesky QR, which
//     squares E each round and is two matrix products instead of an elimination of k dependent
//     steps. A round whose predecessor left nothing to do returns at once.
//   * k_mid_cholqr: blocks that round zero cannot treat (long runs of equal or numerically zero
//     eigenvalues, nearly dependent vectors) take the Cholesky QR or Gram-Schmidt of one CTA; it
//     returns at once for all others.
//   * k_mid_back: U = H_0 ... H_{n-3} Z, two vectors per warp in registers, the reflectors two at
//     a time through a shared-memory ring.
#include <algorithm>

#include "kernels.cuh"
#include "launch.cuh"
#include "trid_solve.cuh"

namespace dmrg {
namespace {

constexpr int MT = 512;             // threads per CTA
constexpr int NW = MT / 32;         // warps
constexpr size_t MID_SMEM_LIMIT = 227 * 1024 - 2048;

// Workspace of one task, in doubles from x_off: Z (n x (k|1), row-major), Gram matrix (k x k,
// row-major, upper triangle), control words.
struct MidCtl {
  unsigned long long emax[3];   // largest |E| of each round (bits of a non-negative double)
  unsigned long long slow;      // set: the block goes to k_mid_cholqr
};
__host__ __device__ inline int64_t mid_g_off(int n, int k) { return int64_t(n) * (k | 1); }
__host__ __device__ inline int64_t mid_vec_workspace(int n, int k) {
  return mid_g_off(n, k) + int64_t(k) * k + 8;
}
__device__ __forceinline__ MidCtl* mid_ctl(double* X, int n, int k) {
  return reinterpret_cast<MidCtl*>(X + mid_g_off(n, k) + int64_t(k) * k);
}

// ---- inverse iteration: `lanes` vectors per CTA (the first lanes of its one warp), blockIdx.x =
// group of vectors, blockIdx.y = task
__global__ void __launch_bounds__(32)
k_mid_invit(double* __restrict__ base, const TridTask* __restrict__ tasks,
            double* __restrict__ xws, int lanes) {
  grid_entry();
  const TridTask tk = tasks[blockIdx.y];
  const int n = tk.n, kk = tk.keep, lane = threadIdx.x, j0 = blockIdx.x * lanes, j = j0 + lane;
  if (j0 >= kk) return;
  extern __shared__ __align__(16) double sm[];
  double* d = sm;                          // n
  double* e = d + n;                       // n
  double* F = e + n;                       // u0, u1, l, z: n x lanes each; pivots
  const double* ws = base + tk.ws_off;
  const double* W = base + tk.w_off;
  for (int i = lane; i < n; i += 32) { d[i] = ws[i]; e[i] = ws[n + i]; }
  __syncwarp();
  const size_t nl = size_t(n) * lanes;
  double* z = F + 3 * nl;
  if (lane < lanes && j < kk) {
    const double tn = fmax(fmax(fabs(W[0]), fabs(W[n - 1])), 1e-300);   // descending
    LeanSlot f{F + lane, F + nl + lane, F + 2 * nl + lane, reinterpret_cast<int*>(F + 4 * nl) + lane,
             lanes};
    // kept eigenvalues that are numerically zero keep the pseudo-random vector alone
    if (W[j] > 1e-13 * tn) lean_inverse_iteration(d, e, n, W[j], z + lane, lanes, j, tn, f);
    else for (int r = 0; r < n; ++r) z[r * lanes + lane] = prand(r, j);
  }
  __syncwarp();
  double* Z = xws + tk.x_off;
  const int w = min(lanes, kk - j0), ldz = kk | 1;
  for (int x = lane; x < n * lanes; x += 32) {
    const int r = x / lanes, q = x - r * lanes;
    if (q < w) Z[int64_t(r) * ldz + j0 + q] = z[x];
  }
}
size_t invit_smem(int n, int lanes) {
  return sizeof(double) * (2 * size_t(n) + 4 * size_t(n) * lanes) + sizeof(int) * size_t(n) * lanes;
}

// ---- runs of nearly equal eigenvalues (neighbours within 1e-12 ||T||): modified Gram-Schmidt
// inside each run, twice, one warp per run. Runs longer than RUN_MAX go to k_mid_cholqr.
constexpr int RUN_THREADS = 256, RUN_MAX = 32;
__global__ void __launch_bounds__(RUN_THREADS)
k_mid_runs(double* __restrict__ base, const TridTask* __restrict__ tasks,
           double* __restrict__ xws) {
  grid_entry();
  const TridTask tk = tasks[blockIdx.x];
  const int n = tk.n, kk = tk.keep;
  if (n < 1 || kk <= 0) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double* W = base + tk.w_off;
  const double tol = 1e-12 * fmax(fmax(fabs(W[0]), fabs(W[n - 1])), 1e-300);
  double* X = xws + tk.x_off;
  double* Z = X;
  MidCtl* ctl = mid_ctl(X, n, kk);
  const int ldz = kk | 1;
  if (threadIdx.x < 4) (threadIdx.x < 3 ? ctl->emax[threadIdx.x] : ctl->slow) = 0ull;
  __syncthreads();
  for (int j = warp; j < kk; j += RUN_THREADS / 32) {
    if (j > 0 && !(W[j - 1] - W[j] > tol)) continue;       // not the first of its run
    int len = 1;
    while (j + len < kk && !(W[j + len - 1] - W[j + len] > tol)) ++len;
    if (len > RUN_MAX) {
      if (lane == 0) ctl->slow = 1ull;
      continue;
    }
    for (int c = 0; c < len && len > 1; ++c) {
      double* zc = Z + j + c;
      for (int pass = 0; pass < 2; ++pass)
        for (int p = 0; p < c; ++p) {
          const double* zp = Z + j + p;
          double s = 0.0;
          for (int r = lane; r < n; r += 32) s += zp[int64_t(r) * ldz] * zc[int64_t(r) * ldz];
          s = wsum(s);
          for (int r = lane; r < n; r += 32) zc[int64_t(r) * ldz] -= s * zp[int64_t(r) * ldz];
        }
      double s = 0.0;
      for (int r = lane; r < n; r += 32) s += zc[int64_t(r) * ldz] * zc[int64_t(r) * ldz];
      s = sqrt(wsum(s));
      if (!(s > 1e-4)) {                                    // nearly dependent
        if (lane == 0) ctl->slow = 1ull;
        break;
      }
      const double inv = 1.0 / s;
      for (int r = lane; r < n; r += 32) zc[int64_t(r) * ldz] *= inv;
    }
  }
}

// Whether round `pass` has anything to do: not for a block handed to k_mid_cholqr, nor after a
// round that found |E| < 1e-9 (its own correction leaves E^2).
__device__ __forceinline__ bool round_active(const MidCtl* ctl, int pass) {
  if (ctl->slow) return false;
  return pass == 0 || __longlong_as_double(ctl->emax[pass - 1]) >= 1e-9;
}

// ---- G = Z^T Z, one 32 x 32 tile of its upper triangle per CTA (blockIdx.x; blockIdx.y = task),
// rows of Z in chunks of 32 through shared memory, the next chunk on its way in registers
constexpr int GT = 256;
__global__ void __launch_bounds__(GT)
k_mid_gram(double* __restrict__ base, const TridTask* __restrict__ tasks, double* __restrict__ xws,
           int pass) {
  grid_entry();
  const TridTask tk = tasks[blockIdx.y];
  const int n = tk.n, kk = tk.keep;
  if (n < 1 || kk <= 0) return;
  const int nt = (kk + 31) >> 5;
  if (int(blockIdx.x) >= nt * (nt + 1) / 2) return;
  int I = 0, x = blockIdx.x;
  while (x >= nt - I) { x -= nt - I; ++I; }
  const int J = I + x;
  double* X = xws + tk.x_off;
  MidCtl* ctl = mid_ctl(X, n, kk);
  if (!round_active(ctl, pass)) return;
  const double* Z = X;
  double* G = X + mid_g_off(n, kk);
  const int ldz = kk | 1;
  __shared__ double sa[32][33], sb[32][33];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double pa[4], pb[4];
  auto fetch = [&](int r0) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int r = r0 + warp + 8 * u, ca = 32 * I + lane, cb = 32 * J + lane;
      pa[u] = (r < n && ca < kk) ? Z[int64_t(r) * ldz + ca] : 0.0;
      pb[u] = (r < n && cb < kk) ? Z[int64_t(r) * ldz + cb] : 0.0;
    }
  };
  const int tp = 2 * (tid >> 4), tq = 2 * (tid & 15);
  double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
  fetch(0);
  for (int r0 = 0; r0 < n; r0 += 32) {
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      sa[warp + 8 * u][lane] = pa[u];
      sb[warp + 8 * u][lane] = pb[u];
    }
    __syncthreads();
    if (r0 + 32 < n) fetch(r0 + 32);
#pragma unroll 8
    for (int r = 0; r < 32; ++r) {
      const double a0 = sa[r][tp], a1 = sa[r][tp + 1], b0 = sb[r][tq], b1 = sb[r][tq + 1];
      acc[0][0] += a0 * b0;
      acc[0][1] += a0 * b1;
      acc[1][0] += a1 * b0;
      acc[1][1] += a1 * b1;
    }
  }
  double mx = 0.0;
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      const int p = 32 * I + tp + u, q = 32 * J + tq + v;
      if (p <= q && q < kk) {
        G[int64_t(p) * kk + q] = acc[u][v];
        const double ev = fabs(acc[u][v] - (p == q ? 1.0 : 0.0));
        mx = ev > mx || ev != ev ? ev : mx;
      }
    }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double t = __shfl_xor_sync(FULL, mx, o);
    mx = t > mx || t != t ? t : mx;
  }
  if (lane == 0)
    atomicMax(&ctl->emax[pass], (unsigned long long)(__double_as_longlong(mx)) & ~(1ull << 63));
}

// ---- Z <- Z (I - E_up), AR rows per CTA (blockIdx.x; blockIdx.y = task)
template <int AR>
__global__ void __launch_bounds__(GT)
k_mid_apply(double* __restrict__ base, const TridTask* __restrict__ tasks,
            double* __restrict__ xws, int pass) {
  grid_entry();
  const TridTask tk = tasks[blockIdx.y];
  const int n = tk.n, kk = tk.keep, r0 = blockIdx.x * AR;
  if (n < 1 || kk <= 0 || r0 >= n) return;
  double* X = xws + tk.x_off;
  MidCtl* ctl = mid_ctl(X, n, kk);
  if (!round_active(ctl, pass)) return;
  // the rounds square E: what is not small enough for the rounds that remain goes to k_mid_cholqr
  const double lim = pass == 0 ? 1e-3 : (pass == 1 ? 1e-5 : 1e-9);
  if (!(__longlong_as_double(ctl->emax[pass]) <= lim)) {
    if (threadIdx.x == 0) ctl->slow = 1ull;
    return;
  }
  double* Z = X;
  const double* G = X + mid_g_off(n, kk);
  const int ldz = kk | 1;
  extern __shared__ __align__(16) double sm[];         // kk x AR: row r of the slab at [p * AR + r]
  const int tid = threadIdx.x;
  for (int x = tid; x < AR * kk; x += GT) {
    const int r = x / kk, p = x - r * kk;
    sm[p * AR + r] = r0 + r < n ? Z[int64_t(r0 + r) * ldz + p] : 0.0;
  }
  __syncthreads();
  for (int q = tid; q < kk; q += GT) {
    double acc[AR];
#pragma unroll
    for (int r = 0; r < AR; ++r) acc[r] = 0.0;
#pragma unroll 4
    for (int p = 0; p < q; ++p) {
      const double g = G[int64_t(p) * kk + q];
      const double2* zp = reinterpret_cast<const double2*>(sm + p * AR);
#pragma unroll
      for (int r = 0; r < AR / 2; ++r) {
        const double2 z = zp[r];
        acc[2 * r] += z.x * g;
        acc[2 * r + 1] += z.y * g;
      }
    }
    const double h = 0.5 * (G[int64_t(q) * kk + q] - 1.0);
#pragma unroll
    for (int r = 0; r < AR; ++r)
      if (r0 + r < n) {
        const double z = sm[q * AR + r];
        Z[int64_t(r0 + r) * ldz + q] = z - fma(h, z, acc[r]);
      }
  }
}

// Packed upper triangle by rows of a k x k matrix: row p starts at gpk(p, k).
__host__ __device__ __forceinline__ int gpk(int p, int k) { return p * k - (p * (p - 1)) / 2; }

// Shared memory of k_mid_cholqr: rinv, sq (k each) and, for k <= kg, the
// packed Gram matrix. kg = the largest k for which all of it fits.
__host__ __device__ inline size_t mid_vec_smem_k(int k, bool gram) {
  return sizeof(double) * (2 * size_t(k) +
                           (gram ? size_t(k) * (k + 1) / 2 : 0)) + 64;
}
int mid_vec_kg() {
  int kg = 0;
  while (mid_vec_smem_k(kg + 1, true) <= MID_SMEM_LIMIT) ++kg;
  return kg;
}

__global__ void __launch_bounds__(MT, 1)
k_mid_cholqr(double* __restrict__ base, const TridTask* __restrict__ tasks,
             double* __restrict__ xws, int kg) {
  grid_entry();
  const TridTask tk = tasks[blockIdx.x];
  const int n = tk.n, kk = tk.keep;
  if (n < 1 || kk <= 0) return;
  double* X = xws + tk.x_off;
  if (mid_ctl(X, n, kk)->slow == 0ull) return;
  const int ldz = kk | 1;
  extern __shared__ double sm[];
  double* rinv = sm;                       // kk
  double* sq = rinv + kk;                  // kk
  __shared__ double red[32];
  __shared__ int s_flag, s_need2;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* Z = X;                        // n x ldz
  double* G = X + mid_g_off(n, kk);                        // kk x kk row-major, upper triangle
  if (tid == 0) { s_flag = 0; s_need2 = 0; }
  __syncthreads();
  // ---- Cholesky QR: G = Z^T Z = R^T R with R = D^(1/2) U (U unit upper), Z <- Z U^-1 D^(-1/2);
  // a second pass unless G was within 1e-3/k of the identity. When the packed upper triangle of
  // G fits in shared memory (kk <= kg) it lives there: the Gram matrix by 4 x 4 register tiles,
  // the elimination by one warp per row, the solve by one thread per row in blocks of 32
  // columns held in registers. Otherwise G stays in the global workspace.
  const bool gsm = kk <= kg;
  double* Gs = sq + kk;                    // packed: G(p, q), q >= p, at gpk(p) + q - p
  for (int pass = 0; pass < 2; ++pass) {
    if (gsm) {
      const int nb4 = (kk + 3) >> 2, ntile = nb4 * (nb4 + 1) / 2;
      for (int x = tid; x < ntile; x += MT) {
        int I = 0;
        while ((I + 1) * nb4 - ((I + 1) * I) / 2 <= x) ++I;
        const int J = I + (x - (I * nb4 - (I * (I - 1)) / 2));
        double acc[16];
#pragma unroll
        for (int c = 0; c < 16; ++c) acc[c] = 0.0;
        for (int r = 0; r < n; ++r) {
          const double* zr = Z + int64_t(r) * ldz;
          double a[4], b[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int ca = 4 * I + u, cb = 4 * J + u;
            a[u] = ca < kk ? zr[ca] : 0.0;
            b[u] = cb < kk ? zr[cb] : 0.0;
          }
#pragma unroll
          for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int w2 = 0; w2 < 4; ++w2) acc[u * 4 + w2] += a[u] * b[w2];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int w2 = 0; w2 < 4; ++w2) {
            const int pp = 4 * I + u, q = 4 * J + w2;
            if (pp <= q && q < kk) {
              const double gv = acc[u * 4 + w2];
              Gs[gpk(pp, kk) + q - pp] = gv;
              if (pass == 0 && fabs(gv - (pp == q ? 1.0 : 0.0)) > 1e-3 / kk) s_need2 = 1;
            }
          }
      }
      __syncthreads();
      for (int j = 0; j < kk; ++j) {
        const double* rowj = Gs + gpk(j, kk) - j;      // rowj[q] = G(j, q), q >= j
        const double gjj = rowj[j];
        if (!(gjj > 1e-8) && tid == 0) s_flag = 1;
        const double inv = 1.0 / fmax(gjj, 1e-300);
        for (int pr = j + 1 + warp; pr < kk; pr += NW) {
          const double f = rowj[pr] * inv;
          double* rowp = Gs + gpk(pr, kk) - pr;
          for (int q = pr + lane; q < kk; q += 32) rowp[q] -= f * rowj[q];
        }
        __syncthreads();
      }
      for (int q = tid; q < kk; q += MT) {
        const double g = fmax(Gs[gpk(q, kk)], 1e-300);
        rinv[q] = 1.0 / g;
        sq[q] = sqrt(g);
      }
      __syncthreads();
      if (s_flag) break;
      for (int r = tid; r < n; r += MT) {
        double* zr = Z + int64_t(r) * ldz;
        for (int q0 = 0; q0 < kk; q0 += 32) {
          const int qb = min(32, kk - q0);
          double acc[32];
#pragma unroll
          for (int c = 0; c < 32; ++c) acc[c] = c < qb ? zr[q0 + c] : 0.0;
#pragma unroll 4
          for (int pp = 0; pp < q0; ++pp) {
            const double y = zr[pp];
            const double* gr = Gs + gpk(pp, kk) - pp;  // gr[q] = G(pp, q)
#pragma unroll
            for (int c = 0; c < 32; ++c)
              if (c < qb) acc[c] -= y * gr[q0 + c];
          }
#pragma unroll
          for (int c = 0; c < 32; ++c) {
            if (c < qb) {
              const double* gc = Gs + gpk(q0, kk) - q0;  // row q0, then down the block
              double sacc = acc[c];
              int off = 0;
#pragma unroll
              for (int c2 = 0; c2 < 32; ++c2) {
                if (c2 < c) sacc -= acc[c2] * gc[off + q0 + c];
                off += kk - (q0 + c2) - 1;             // gpk(p + 1) - (p + 1) - (gpk(p) - p)
              }
              acc[c] = sacc * rinv[q0 + c];
            }
          }
#pragma unroll
          for (int c = 0; c < 32; ++c)
            if (c < qb) zr[q0 + c] = acc[c];
        }
        for (int q = 0; q < kk; ++q) zr[q] *= sq[q];
      }
      __syncthreads();
      if (!s_need2) break;
      continue;
    }
    for (int x = tid; x < kk * kk; x += MT) {
      const int pp = x / kk, q = x - pp * kk;
      if (pp > q) continue;
      double s0 = 0.0, s1 = 0.0;
      int r = 0;
      for (; r + 2 <= n; r += 2) {
        s0 += Z[int64_t(r) * ldz + pp] * Z[int64_t(r) * ldz + q];
        s1 += Z[int64_t(r + 1) * ldz + pp] * Z[int64_t(r + 1) * ldz + q];
      }
      if (r < n) s0 += Z[int64_t(r) * ldz + pp] * Z[int64_t(r) * ldz + q];
      const double g = s0 + s1;
      G[int64_t(pp) * kk + q] = g;
      if (pass == 0 && fabs(g - (pp == q ? 1.0 : 0.0)) > 1e-3 / kk) s_need2 = 1;
    }
    __syncthreads();
    for (int j = 0; j < kk; ++j) {
      const double gjj = G[int64_t(j) * kk + j];
      if (!(gjj > 1e-8) && tid == 0) s_flag = 1;
      const double inv = 1.0 / fmax(gjj, 1e-300);
      const int t = kk - j - 1;
      for (int x = tid; x < t * t; x += MT) {
        const int pp = j + 1 + x / t, q = j + 1 + x % t;
        if (pp <= q)
          G[int64_t(pp) * kk + q] -= G[int64_t(j) * kk + pp] * G[int64_t(j) * kk + q] * inv;
      }
      __syncthreads();
    }
    for (int q = tid; q < kk; q += MT) {
      const double g = fmax(G[int64_t(q) * kk + q], 1e-300);
      rinv[q] = 1.0 / g;
      sq[q] = sqrt(g);
    }
    __syncthreads();
    if (s_flag) break;
    for (int r = tid; r < n; r += MT) {
      double* zr = Z + int64_t(r) * ldz;
      for (int q = 0; q < kk; ++q) {
        double s0 = zr[q], s1 = 0.0;
        int pp = 0;
        for (; pp + 2 <= q; pp += 2) {
          s0 -= zr[pp] * G[int64_t(pp) * kk + q];
          s1 -= zr[pp + 1] * G[int64_t(pp + 1) * kk + q];
        }
        if (pp < q) s0 -= zr[pp] * G[int64_t(pp) * kk + q];
        zr[q] = (s0 + s1) * rinv[q];
      }
      for (int q = 0; q < kk; ++q) zr[q] *= sq[q];
    }
    __syncthreads();
    if (!s_need2) break;
  }
  if (s_flag) {
    // two passes of classical Gram-Schmidt, largest eigenvalue first, with fresh starts for
    // vectors that lie (numerically) in the span of the previous ones
    int attempt = 0;
    for (int c = 0; c < kk; ++c) {
      for (int pass = 0; pass < 2; ++pass) {
        {
          const int g8 = tid >> 3, l8 = tid & 7, ng8 = MT >> 3;
          for (int qb = 0; qb < c; qb += ng8) {
            const int q = qb + g8;
            double s = 0.0;
            if (q < c)
              for (int r = l8; r < n; r += 8) s += Z[int64_t(r) * ldz + q] * Z[int64_t(r) * ldz + c];
            s += __shfl_xor_sync(FULL, s, 4, 8);
            s += __shfl_xor_sync(FULL, s, 2, 8);
            s += __shfl_xor_sync(FULL, s, 1, 8);
            if (q < c && l8 == 0) G[q] = s;      // G reused as the coefficient row
          }
        }
        __syncthreads();
        for (int r = tid; r < n; r += MT) {
          double s = Z[int64_t(r) * ldz + c];
          for (int q = 0; q < c; ++q) s -= G[q] * Z[int64_t(r) * ldz + q];
          Z[int64_t(r) * ldz + c] = s;
        }
        __syncthreads();
      }
      double part = 0.0;
      for (int r = tid; r < n; r += MT) part += Z[int64_t(r) * ldz + c] * Z[int64_t(r) * ldz + c];
      const double nr = sqrt(bsum(part, red));
      if (nr < 1e-8 && attempt < 8) {
        ++attempt;
        for (int r = tid; r < n; r += MT) Z[int64_t(r) * ldz + c] = prand(r, c + 1000 * attempt);
        __syncthreads();
        --c;
        continue;
      }
      attempt = 0;
      for (int r = tid; r < n; r += MT) Z[int64_t(r) * ldz + c] /= fmax(nr, 1e-300);
      __syncthreads();
    }
  }
}

// Sums of s[0..5) over the warp, in every lane: exchanges that halve the values a lane carries,
// then one broadcast each.
__device__ __forceinline__ void wsum5(double (&s)[5], int lane) {
  const bool b0 = lane & 1, b1 = lane & 2, b2 = lane & 4;
  const double u0 = (b0 ? s[1] : s[0]) + __shfl_xor_sync(FULL, b0 ? s[0] : s[1], 1);
  const double u1 = (b0 ? s[3] : s[2]) + __shfl_xor_sync(FULL, b0 ? s[2] : s[3], 1);
  const double u2 = (b0 ? 0.0 : s[4]) + __shfl_xor_sync(FULL, b0 ? s[4] : 0.0, 1);
  const double w0 = (b1 ? u1 : u0) + __shfl_xor_sync(FULL, b1 ? u0 : u1, 2);
  const double w1 = (b1 ? 0.0 : u2) + __shfl_xor_sync(FULL, b1 ? u2 : 0.0, 2);
  double v = (b2 ? w1 : w0) + __shfl_xor_sync(FULL, b2 ? w0 : w1, 4);
  v += __shfl_xor_sync(FULL, v, 8);
  v += __shfl_xor_sync(FULL, v, 16);
#pragma unroll
  for (int q = 0; q < 5; ++q) s[q] = __shfl_sync(FULL, v, q);
}

// Back-transformation U = H_0 H_1 ... H_{n-3} Z: two kept vectors per warp in registers (lane l
// has rows l, l + 32, ...), n <= 32 RM. Two reflectors per step, a = v_k and b = v_{k-1}: their
// four products with the vectors and a.b are one warp sum. The pairs come through a ring of
// BSTAGES shared-memory stages, several steps ahead (cp.async): read straight from L2 one pair
// ahead, a step waited for them (n = 345, 200 vectors: 191 us against 128 us).
// Bound by the latency of the warp sum: blocks of more reflectors would add products that the two
// warps per scheduler have no free issue slots for.
constexpr int BW = 4, BSTAGES = 6;       // warps per CTA, stages of the ring
template <int RM, int NV>                // NV vectors per warp
__global__ void __launch_bounds__(32 * BW)
k_mid_back(double* __restrict__ base, const TridTask* __restrict__ tasks,
           const double* __restrict__ xws) {
  grid_entry();
  constexpr int LD = 32 * RM;
  constexpr int KR = RM <= 16 ? RM : 1;          // reflectors kept in registers between their uses
  const TridTask tk = tasks[blockIdx.y];
  const int n = tk.n, kk = tk.keep, tid = threadIdx.x, lane = tid & 31;
  if (n < 1 || n > LD || int(blockIdx.x) * NV * BW >= kk) return;
  extern __shared__ __align__(16) double sm[];
  double* stau = sm + BSTAGES * 2 * LD;          // n
  const int q0 = NV * (blockIdx.x * BW + (tid >> 5));
  const bool one = q0 < kk, two = NV > 1 && q0 + 1 < kk;
  const int ldz = kk | 1;
  const double* Z = xws + tk.x_off;
  const double* V = base + tk.a_off;             // reflector k: V[k n + r], r >= 32 (k / 32)
  const double* tau = base + tk.ws_off + 2 * n;
  const int np = (n - 1) / 2;                    // pairs (k, k - 1), k = n - 3, n - 5, ...
  auto fill = [&](int t) {
    const int k = n - 3 - 2 * t;
    if (t < np) {
      double* st = sm + (t % BSTAGES) * 2 * LD;
      for (int i = (k & ~31) + tid; i < n; i += 32 * BW) {
        const unsigned da = unsigned(__cvta_generic_to_shared(st + i));
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" :: "r"(da), "l"(V + int64_t(k) * n + i));
        if (k >= 1)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;"
                       :: "r"(da + 8 * LD), "l"(V + int64_t(k - 1) * n + i));
        else
          st[LD + i] = 0.0;                      // no partner: tb = 0 alone would let a NaN through
      }
    }
    asm volatile("cp.async.commit_group;");
  };
  // rows past the block stay zero in every stage
  for (int x = tid; x < BSTAGES * 2 * LD; x += 32 * BW)
    if (x % LD >= n) sm[x] = 0.0;
  __syncthreads();
  for (int t = 0; t < BSTAGES - 1; ++t) fill(t);
  for (int i = tid; i < n; i += 32 * BW) stau[i] = i < n - 2 ? tau[i] : 0.0;
  double z0[RM], z1[NV > 1 ? RM : 1];
#pragma unroll
  for (int r = 0; r < RM; ++r) {
    const int i = lane + 32 * r;
    z0[r] = i < n && one ? Z[int64_t(i) * ldz + q0] : 0.0;
    if (NV > 1) z1[r] = i < n && two ? Z[int64_t(i) * ldz + q0 + 1] : 0.0;
  }
  for (int t = 0; t < np; ++t) {
    const int k = n - 3 - 2 * t;
    asm volatile("cp.async.wait_group %0;" :: "n"(BSTAGES - 2) : "memory");
    __syncthreads();                             // pair t is there, pair t - 1 is done with
    fill(t + BSTAGES - 1);
    if (!one) continue;
    const double* st = sm + (t % BSTAGES) * 2 * LD + lane;
    const double ta = stau[k], tb = k >= 1 ? stau[k - 1] : 0.0;   // tb = 0: no partner
    double s[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    double a[KR], b[KR];
    if (KR == RM) {                              // all at once: rows above the pair's are not used
#pragma unroll
      for (int r = 0; r < KR; ++r) {
        a[r] = st[32 * r];
        b[r] = st[LD + 32 * r];
      }
    }
#pragma unroll
    for (int r = 0; r < RM; ++r) {
      if (32 * r + 31 >= k && 32 * r < n) {
        const double av = KR == RM ? a[r % KR] : st[32 * r];
        const double bv = KR == RM ? b[r % KR] : st[LD + 32 * r];
        s[0] = fma(av, z0[r], s[0]);
        s[2] = fma(bv, z0[r], s[2]);
        if (NV > 1) {
          s[1] = fma(av, z1[r], s[1]);
          s[3] = fma(bv, z1[r], s[3]);
        }
        s[4] = fma(av, bv, s[4]);
      }
    }
    wsum5(s, lane);
    const double x0 = ta * s[0], x1 = ta * s[1];
    const double y0 = tb * fma(-x0, s[4], s[2]), y1 = tb * fma(-x1, s[4], s[3]);
#pragma unroll
    for (int r = 0; r < RM; ++r) {
      if (32 * r + 31 >= k && 32 * r < n) {
        const double av = KR == RM ? a[r % KR] : st[32 * r];
        const double bv = KR == RM ? b[r % KR] : st[LD + 32 * r];
        z0[r] = fma(-y0, bv, fma(-x0, av, z0[r]));
        if (NV > 1) z1[r] = fma(-y1, bv, fma(-x1, av, z1[r]));
      }
    }
  }
  double* U = base + tk.u_off;
#pragma unroll
  for (int r = 0; r < RM; ++r) {
    const int i = lane + 32 * r;
    if (i < n) {
      if (one) U[int64_t(q0) * n + i] = z0[r];
      if (NV > 1 && two) U[int64_t(q0 + 1) * n + i] = z1[r];
    }
  }
}
template <int RM, int NV>
void launch_back(cudaStream_t s, double* base, const TridTask* tasks, int ntasks, int max_n,
                 int max_k, const double* xws) {
  const size_t sm = sizeof(double) * (BSTAGES * 2 * 32 * RM + size_t(max_n));
  raise_smem_limit(reinterpret_cast<const void*>(k_mid_back<RM, NV>), sm);
  launch_k(k_mid_back<RM, NV>, dim3((max_k + NV * BW - 1) / (NV * BW), ntasks), 32 * BW, sm, s, base,
           tasks, xws);
}

}  // namespace

int64_t syevt_mid_workspace(int n, int k) { return mid_vec_workspace(n, k); }

void launch_trid_mid_vectors(cudaStream_t s, double* base, const TridTask* tasks, int ntasks,
                             int max_n, int max_k, double* xws) {
  launch_trid_mid_inner(s, base, tasks, ntasks, max_n, max_k, xws);
  launch_trid_mid_back(s, base, tasks, ntasks, max_n, max_k, xws);
}

void launch_trid_mid_inner(cudaStream_t s, double* base, const TridTask* tasks, int ntasks,
                           int max_n, int max_k, double* xws) {
  if (ntasks <= 0) return;
  int lanes = 8;                           // 152 KB at n = 512
  while (lanes > 1 && invit_smem(max_n, lanes) > MID_SMEM_LIMIT) lanes /= 2;
  const size_t si = invit_smem(max_n, lanes);
  raise_smem_limit(reinterpret_cast<const void*>(k_mid_invit), si);
  launch_k(k_mid_invit, dim3((max_k + lanes - 1) / lanes, ntasks), 32, si, s, base, tasks, xws,
           lanes);
  launch_k(k_mid_runs, ntasks, RUN_THREADS, 0, s, base, tasks, xws);
  const int nt = (max_k + 31) / 32;
  const int ar = sizeof(double) * 16 * size_t(max_k) <= MID_SMEM_LIMIT ? 16 : 8;
  const auto apply = ar == 16 ? k_mid_apply<16> : k_mid_apply<8>;
  const size_t sa = sizeof(double) * ar * size_t(max_k);
  raise_smem_limit(reinterpret_cast<const void*>(apply), sa);
  for (int pass = 0; pass < 3; ++pass) {
    launch_k(k_mid_gram, dim3(nt * (nt + 1) / 2, ntasks), GT, 0, s, base, tasks, xws, pass);
    launch_k(apply, dim3((max_n + ar - 1) / ar, ntasks), GT, sa, s, base, tasks, xws, pass);
  }
  const int kg = mid_vec_kg();
  const size_t sm = std::max(mid_vec_smem_k(std::min(max_k, kg), true), mid_vec_smem_k(max_k, false));
  raise_smem_limit(reinterpret_cast<const void*>(k_mid_cholqr), sm);
  launch_k(k_mid_cholqr, ntasks, MT, sm, s, base, tasks, xws, kg);
  count_launch(9);
}

void launch_trid_mid_back(cudaStream_t s, double* base, const TridTask* tasks, int ntasks,
                          int max_n, int max_k, const double* xws) {
  if (ntasks <= 0) return;
  auto back = [&](auto launch) { launch(s, base, tasks, ntasks, max_n, max_k, xws); };
  if (max_n <= 128) back(launch_back<4, 2>);
  else if (max_n <= 160) back(launch_back<5, 2>);
  else if (max_n <= 256) back(launch_back<8, 2>);
  else if (max_n <= 352) back(launch_back<11, 2>);
  else if (max_n <= 512) back(launch_back<16, 2>);
  else if (max_n <= 1024) back(launch_back<32, 2>);
  else back(launch_back<64, 1>);
  count_launch();
}

}  // namespace dmrg
