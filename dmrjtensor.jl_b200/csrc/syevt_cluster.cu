// syevt_cluster.cu -- tridiagonalisation of larger density-matrix blocks by a thread-block
// cluster, and the eigenvalues of the tridiagonal matrices by the whole chip.
//
// k_trid_cluster: one cluster of c CTAs per block (c = 8, or 16 for large blocks). The matrix is
// kept in full in the cluster's registers: a warp owns up to CC whole columns (column s c + rank
// of warp s mod 16, so the trailing block stays evenly dealt), lane l their rows l, l + 32, ...
// The owner of column j therefore has the whole product p_j = tau B(:,j).v, and a Householder
// step exchanges one message per column instead of partial sums:
//   * pass: every warp applies the previous step's rank-2 update to its columns and multiplies
//     them by the new reflector in the same sweep. (x.B(:,j), B(k+1, j)) and the CTA's share of
//     x.B x go to every CTA with st.async, which also counts the bytes into the receiver's mbarrier.
//     B(k+1, :) is the next pivot column by symmetry, so no CTA ever sends a column;
//   * every CTA then forms w and the next reflector by itself, from the same numbers in the same
//     order (bit-identical in all CTAs). The reflector stays unscaled (x, with v = s x and
//     v_first = 1) until its norm is known: an extra warp sums the squares and takes the root
//     and the reciprocal while the others sweep their columns and exchange messages.
// Blocks above HN = 512 rows start in k_trid_lead, a cluster of 16 CTAs that takes the same steps
// on the matrix in global memory (L2-resident) until 512 or fewer rows are left.
// What bounds it: the latency of a step's chain (sweep, warp sums, message, elementwise update:
// ~1,500 cycles for small blocks, ~2,500 at n = 345) and the issue rate of the two warps per
// scheduler, not bandwidth or arithmetic. Fewer warps with more columns each beat more warps: the
// work per warp that does not depend on its columns is over half of the instructions (n = 345, 16
// column warps: 0.86 ms; 7 column warps and the reflector warp, 8 CTAs: 0.57 ms; 16 CTAs: 0.48 ms;
// one CTA with the matrix in global and shared memory: 4.6 ms with the eigenvalues).
#include <cstring>

#include "cluster.cuh"
#include "kernels.cuh"
#include "launch.cuh"
#include "trid_solve.cuh"

namespace dmrg {
namespace {

constexpr int HW = 7;                // column warps per CTA
constexpr int HT = 32 * HW;          // threads of the column warps
constexpr int HN = 512;              // largest block of k_trid_cluster
constexpr int HTX = HT + 32;         // and of the reflector warp
// Bit pattern (a NaN) that k_trid_cluster leaves in d[0] when a wait gave up.
constexpr long long TRID_GAVE_UP = 0x7ff8000000d06e0fLL;

// stores into another CTA that count their bytes into its mbarrier
__device__ __forceinline__ void async_store(unsigned addr, unsigned bar, double a, double b) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];"
               :: "r"(addr), "l"(__double_as_longlong(a)), "l"(__double_as_longlong(b)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void async_store(unsigned addr, unsigned bar, double a) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];"
               :: "r"(addr), "l"(__double_as_longlong(a)), "r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
// Waits for the phase; false after about a second.
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity) {
  if (mbar_try(bar, parity)) return true;
  unsigned long long t0 = 0, t;
  for (unsigned it = 1;; ++it) {
    if (mbar_try(bar, parity)) return true;
    if ((it & 255u) == 0) {
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
      if (t0 == 0) t0 = t;
      else if (t - t0 > 1000000000ull) return false;
    }
  }
}

// Sums s[0..N) over the warp's lanes: lane l returns the sum of s[l % G], G the power of two from
// N up (0 for the lanes of a missing column).
template <int N, int MASK>
__device__ __forceinline__ double wsum_cols(const double (&s)[N], int lane) {
  if constexpr (N == 1) {
    double v = s[0];
#pragma unroll
    for (int m = MASK; m < 32; m <<= 1) v += __shfl_xor_sync(FULL, v, m);
    return v;
  } else {
    constexpr int H = (N + 1) / 2;
    const bool up = lane & MASK;
    double u[H];
#pragma unroll
    for (int p = 0; p < H; ++p) {
      const double lo = s[2 * p], hi = 2 * p + 1 < N ? s[(2 * p + 1) % N] : 0.0;
      u[p] = (up ? hi : lo) + __shfl_xor_sync(FULL, up ? lo : hi, MASK);
    }
    return wsum_cols<H, 2 * MASK>(u, lane);
  }
}

constexpr int LC = 16;               // CTAs of k_trid_lead's cluster
constexpr int LT = 512;              // threads of each
constexpr int LWARPS = LT / 32;
constexpr int LCOLS = 4;             // columns per warp and sweep

// First column that k_trid_cluster takes (a multiple of 32, so that both kernels store reflectors
// from the same 32-row boundaries).
__host__ __device__ __forceinline__ int trid_lead_steps(int n) {
  return n <= HN ? 0 : (n - HN + 31) / 32 * 32;
}

// The first trid_lead_steps(n) Householder steps of a block above HN rows: columns dealt cyclically
// to the CTAs, four per warp and sweep; each sweep applies the previous step's rank-2 update,
// stores, and multiplies by the new reflector (unscaled, as in k_trid_cluster). One cluster
// barrier per step. Bound by the L2 bandwidth of 16 SMs: the trailing block is read and written
// once a step.
__global__ void __launch_bounds__(LT, 1)
k_trid_lead(double* __restrict__ base, const TridTask* __restrict__ tasks) {
  grid_entry();
  const TridTask tk = tasks[blockIdx.x / LC];
  const int n = tk.n, ks = trid_lead_steps(n);
  if (ks == 0) return;                     // the same in every CTA of the cluster
  const int rank = cluster_rank();
  extern __shared__ __align__(16) double sm[];
  double2* pc = reinterpret_cast<double2*>(sm);   // 2 x n: (x.B(:,j), pivot-row element j)
  double* xb = sm + 4 * size_t(n);         // 2 x n: unscaled reflectors, by parity
  double* w = xb + 2 * size_t(n);          // n
  __shared__ double kw[2][LC * LWARPS];    // shares of x.B x, every warp of every CTA
  __shared__ double red[LWARPS];
  __shared__ double s_alpha;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* Ag = base + tk.a_off;
  double* ws = base + tk.ws_off;           // d | e | tau
  const bool head = rank == 0;

  double part = 0.0;
  for (int i = tid; i < n; i += LT) {
    const double a = Ag[i];
    xb[i] = i >= 2 ? a : 0.0;
    xb[n + i] = 0.0;
    w[i] = 0.0;
    if (i >= 2) part += a * a;
    if (i == 1) s_alpha = a;
    if (i == 0 && head) ws[0] = a;
  }
  part = wsum(part);
  if (lane == 0) red[warp] = part;
  cluster_sync_all();                      // every CTA runs before any remote store

  double sc_p = 0.0, tau = 0.0, sc = 0.0, first = 0.0;   // first: the reflector's first element
  auto reflect = [&](int k) {              // reflector k's scalars, and the reflector into column k
    double t[LWARPS];
#pragma unroll
    for (int q = 0; q < LWARPS; ++q) t[q] = red[q];
#pragma unroll
    for (int h = LWARPS / 2; h > 0; h >>= 1)
#pragma unroll
      for (int q = 0; q < h; ++q) t[q] += t[q + h];
    const double alpha = s_alpha;
    double beta = alpha;
    tau = 0.0;
    sc = 0.0;
    first = 0.0;
    if (t[0] != 0.0) {
      beta = -copysign(sqrt(fma(alpha, alpha, t[0])), alpha);
      tau = (beta - alpha) / beta;
      first = alpha - beta;
      sc = 1.0 / first;
    }
    if (head && tid == 0) { ws[n + k] = beta; ws[2 * n + k] = tau; }
    if (rank == k % LC) {
      const double* x = xb + (k & 1) * n;
      for (int i = (k & ~31) + tid; i < n; i += LT)
        Ag[int64_t(k) * n + i] = i > k + 1 ? x[i] * sc : (i == k + 1 ? 1.0 : 0.0);
    }
  };
  // columns j >= f of this CTA: pending update, and (dot) the product with x
  auto sweep = [&](int f, const double* x, const double* xp, bool dot, double2* pck) {
    const int s0 = (f - rank + LC - 1) / LC, i0 = f & ~31;
    double kpart = 0.0;
    for (int s = s0 + warp; s * LC + rank < n; s += LCOLS * LWARPS) {
      double* col[LCOLS];
      double wj[LCOLS], xj[LCOLS], acc[LCOLS];
      const int jl = s * LC + rank;
      const int nq = min(LCOLS, (n - jl + LC * LWARPS - 1) / (LC * LWARPS));
#pragma unroll
      for (int q = 0; q < LCOLS; ++q) {
        const int j = jl + (q < nq ? q : 0) * LC * LWARPS;   // a missing column repeats the first
        col[q] = Ag + int64_t(j) * n;
        wj[q] = -sc_p * w[j];
        xj[q] = -sc_p * xp[j];
        acc[q] = 0.0;
      }
#pragma unroll 4
      for (int i = i0 + lane; i < n; i += 32) {
        const bool live = i >= f;
        const double xi = x[i], xpi = xp[i], wi = w[i];
        double v[LCOLS];
#pragma unroll
        for (int q = 0; q < LCOLS; ++q) v[q] = col[q][i];
#pragma unroll
        for (int q = 0; q < LCOLS; ++q) {
          v[q] = fma(wi, xj[q], fma(xpi, wj[q], v[q]));
          if (live && q < nq) col[q][i] = v[q];
          if (live) acc[q] = fma(v[q], xi, acc[q]);
        }
      }
      if (dot) {
        const double dt = wsum_cols<LCOLS, 1>(acc, lane);
        __syncwarp();
        const int q = lane & 3, j = jl + q * LC * LWARPS;
        if (j < n) {
          kpart += dt * x[j];
          const double piv = Ag[int64_t(j) * n + f];
          const unsigned dst = smem_addr(&pck[j]);
          for (int r = lane >> 2; r < LC; r += 8) peer_store(peer_addr(dst, r), dt, piv);
        }
      }
    }
    return kpart;
  };
  reflect(0);
  for (int k = 0; k < ks; ++k) {
    const int par = k & 1, f = k + 1;
    const double* x = xb + par * n;                // reflector k, x[k+1] = 0
    double* xn = xb + (par ^ 1) * n;               // reflector k-1, then k+1
    double2* pck = pc + size_t(par) * n;
    double kpart = sweep(f, x, xn, true, pck);
    kpart += __shfl_xor_sync(FULL, kpart, 1);
    kpart += __shfl_xor_sync(FULL, kpart, 2);
    if (lane < LC) peer_store(peer_addr(smem_addr(&kw[par][rank * LWARPS + warp]), lane), kpart);
    cluster_sync_all();
    double K = 0.0;
#pragma unroll
    for (int q = 0; q < LC * LWARPS / 32; ++q) K += kw[par][lane + 32 * q];
    K = wsum(K);
    const double2 pf = pck[f];
    const double hk = 0.5 * tau * (tau * fma(sc, fma(sc, K, 2.0 * pf.x), pf.y));
    const double w0 = tau * fma(sc, pf.x, pf.y) - hk;
    part = 0.0;
    for (int i = f + tid; i < n; i += LT) {
      const double2 pi = pck[i];
      const double vi = i == f ? 1.0 : sc * x[i];
      const double wi = tau * fma(sc, pi.x, pi.y) - hk * vi;
      const double ci = pi.y - fma(vi, w0, wi);
      w[i] = wi;
      xn[i] = i >= f + 2 ? ci : 0.0;
      if (i >= f + 2) part = fma(ci, ci, part);
      if (i == f && head) ws[f] = ci;              // d[k+1]
      if (i == f + 1) s_alpha = ci;
    }
    part = wsum(part);
    if (lane == 0) red[warp] = part;
    __syncthreads();
    sc_p = sc;
    if (k + 1 < ks) reflect(f);
  }
  // the pending update of step ks - 1, its pivot row included, so that the trailing block is a
  // problem of its own
  if (tid == 0) xb[((ks - 1) & 1) * n + ks] = first;
  __syncthreads();
  sweep(ks, xb + (ks & 1) * n, xb + ((ks - 1) & 1) * n, false, pc);
  cluster_sync_all();                      // no CTA leaves before the others have read its stores
}

template <int V>
struct Lo {
  static constexpr int v = V;
};

// Blocks of n <= HN with up to 32 RM rows and HW CC C columns.
template <int RM, int CC, int C>
__global__ void __launch_bounds__(HTX, 1)
k_trid_cluster(double* __restrict__ base, const TridTask* __restrict__ tasks) {
  grid_entry();
  constexpr int G = CC <= 1 ? 1 : (CC <= 2 ? 2 : (CC <= 4 ? 4 : 8));   // lanes per column group
  constexpr int EPT = (32 * RM + HTX - 1) / HTX;          // elements per thread
  const TridTask tk = tasks[blockIdx.x / C];
  const int k0 = trid_lead_steps(tk.n), ld = tk.n, n = ld - k0;   // the block from column k0 on
  if (n > 32 * RM || n > HW * CC * C) return;      // the same in all of the cluster
  if (n < 3) {                                     // tridiagonal as it is
    if (cluster_rank() == 0 && threadIdx.x == 0 && n > 0) {
      const double* A = base + tk.a_off;
      double* ws = base + tk.ws_off;
      for (int i = 0; i < n; ++i) {
        ws[i] = A[i * (n + 1)];
        ws[n + i] = i + 1 < n ? A[i * n + i + 1] : 0.0;
        ws[2 * n + i] = 0.0;
      }
    }
    return;
  }
  __shared__ __align__(16) double2 pc[2][HN];      // (x.B(:,j), pivot-row element j), by parity
  __shared__ __align__(16) double kw[2][C];        // the CTAs' shares of x.B x
  __shared__ __align__(16) double kp[HW + 1];      // the warps' shares
  __shared__ double s_pv[HW][CC];                  // the warps' pivot-row elements
  __shared__ double xb[2][HN];                     // unscaled reflectors, by parity
  __shared__ double w[HN];
  __shared__ double s_alpha, s_tau, s_sc;
  __shared__ __align__(8) unsigned long long mbar[2];
  const int rank = cluster_rank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* Ag = base + tk.a_off + int64_t(k0) * (ld + 1);
  double* ws = base + tk.ws_off + k0;              // d | e | tau, ld apart
  const bool head = rank == 0;
  const unsigned bar0 = smem_addr(&mbar[0]);

  double a[CC][RM];                                // the warp's columns
  int jc[CC];
#pragma unroll
  for (int q = 0; q < CC; ++q) {
    jc[q] = warp < HW ? (q * HW + warp) * C + rank : n;
#pragma unroll
    for (int r = 0; r < RM; ++r) {
      const int i = lane + 32 * r;
      a[q][r] = (jc[q] < n && i < n) ? Ag[int64_t(jc[q]) * ld + i] : 0.0;
    }
  }
  double xi[EPT];                                  // this thread's elements of the reflector
#pragma unroll
  for (int u = 0; u < EPT; ++u) {
    const int i = tid + u * HTX;
    const double a0 = i < n ? Ag[i] : 0.0;
    xi[u] = i >= 2 ? a0 : 0.0;
    if (i < HN) {
      xb[0][i] = xi[u];
      xb[1][i] = 0.0;
      w[i] = 0.0;
    }
    if (i == 1) s_alpha = a0;
    if (i == 0 && head) ws[0] = a0;
  }
  if (tid == 0) {
    kp[HW] = 0.0;
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(bar0));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(bar0 + 8));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  cluster_sync_all();                              // every CTA is ready to receive
  double sc_p = 0.0;
  bool ok = true;
  for (int k = 0; k + 2 < n; ++k) {
    const int par = k & 1, f = k + 1;
    const unsigned bar = bar0 + 8 * par;
    const double* x = xb[par];
    const double* xp = xb[par ^ 1];
    if (warp == HW) {
      // reflector k from x and alpha: beta = -sign(alpha) |(alpha, x)|, tau = 1 + |alpha|/|beta|,
      // v = x / (alpha - beta)
      double s2 = 0.0;
#pragma unroll
      for (int r = 0; r < RM; ++r) {
        const double xv = x[lane + 32 * r];
        s2 += xv * xv;
      }
      s2 = wsum(s2);
      const double al = s_alpha;
      double t = 0.0, sv = 0.0, be = al;
      if (s2 != 0.0) {
        const double n2 = fma(al, al, s2), nr = sqrt(n2);
        be = -copysign(nr, al);
        t = (be - al) / be;
        sv = 1.0 / (al - be);
      }
      if (lane == 0) { s_tau = t; s_sc = sv; }
      if (head && lane == 0) { ws[ld + k] = be; ws[2 * ld + k] = t; }
      // reflector k, its unit entry and the zeros above it in its first 32 rows included: the
      // back-transformation reads whole 32-row chunks of column k
      if (rank == k % C)
        for (int i = (k & ~31) + lane; i < n; i += 32)
          Ag[int64_t(k) * ld + i] = i > f ? x[i] * sv : (i == f ? 1.0 : 0.0);
    } else {
      if (tid == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                     :: "r"(bar), "r"(16 * (n - f) + 8 * C) : "memory");
      // ---- pass: pending rank-2 update and product with x over the columns j >= f
      double acc[CC], wj[CC], xj[CC];
#pragma unroll
      for (int q = 0; q < CC; ++q) {
        const bool on = jc[q] >= f && jc[q] < n;
        wj[q] = on ? -sc_p * w[jc[q]] : 0.0;
        xj[q] = on ? -sc_p * xp[jc[q]] : 0.0;
        acc[q] = 0.0;
      }
      // columns in the order of q finish first: once the lower half is done, the upper alone
      auto sweep = [&](auto lo) {
        const int ib = (f & ~31) + lane;           // the next chunk's vectors are loaded ahead
        double xv = x[ib], xpv = xp[ib], wv = w[ib];
#pragma unroll
        for (int r = 0; r < RM; ++r) {
          if (32 * r + 31 >= f && 32 * r < n) {
            const int i = lane + 32 * r;
            const double xc = xv, xpc = xpv, wc = wv;
            if (r + 1 < RM) { xv = x[i + 32]; xpv = xp[i + 32]; wv = w[i + 32]; }
#pragma unroll
            for (int q = lo.v; q < CC; ++q) {
              const double v = fma(wc, xj[q], fma(xpc, wj[q], a[q][r]));
              a[q][r] = v;
              acc[q] = fma(v, xc, acc[q]);
            }
            if (32 * r <= f && i == f) {
#pragma unroll
              for (int q = lo.v; q < CC; ++q) s_pv[warp][q] = a[q][r];
            }
          }
        }
      };
      double kpart = 0.0;
      if (jc[CC - 1] >= f) {
        if (CC == 1 || jc[CC / 2 - (CC > 1)] >= f) sweep(Lo<0>{});
        else sweep(Lo<CC / 2>{});
        const double dot = wsum_cols<CC, 1>(acc, lane);
        const int ql = lane % G;
        const int j = ql < CC ? (ql * HW + warp) * C + rank : n;
        __syncwarp();
        if (j >= f && j < n) {
          kpart = dot * x[j];
          const double piv = s_pv[warp][ql];
          const unsigned dst = smem_addr(&pc[par][j]);
#pragma unroll
          for (int r0 = 0; r0 < C; r0 += 32 / G) {
            const int r = r0 + lane / G;
            if (C % (32 / G) == 0 || r < C)
              async_store(peer_addr(dst, r), peer_addr(bar, r), dot, piv);
          }
        }
#pragma unroll
        for (int m = 1; m < G; m <<= 1) kpart += __shfl_xor_sync(FULL, kpart, m);
      }
      if (lane == 0) kp[warp] = kpart;
      asm volatile("bar.sync 2, %0;" :: "n"(HT) : "memory");
      if (warp == HW - 1 && lane < C) {
        double t[HW + 1];
#pragma unroll
        for (int q = 0; q <= HW; ++q) t[q] = kp[q];
#pragma unroll
        for (int h = (HW + 1) / 2; h > 0; h >>= 1)
#pragma unroll
          for (int q = 0; q < h; ++q) t[q] += t[q + h];
        async_store(peer_addr(smem_addr(&kw[par][rank]), lane), peer_addr(bar, lane), t[0]);
      }
    }
    // ---- w and the pivot column of the next step, by all threads. With v = sc x and
    // v_f = 1: p_j = tau (sc dot_j + B_fj), and p.v = tau (B_ff + 2 sc dot_f + sc^2 x.dot)
    ok = mbar_wait(bar, unsigned(k >> 1) & 1u);
    __syncthreads();                               // tau and sc of reflector k
    const double tau = s_tau, sc = s_sc;
    double t[C];
#pragma unroll
    for (int q = 0; q < C; ++q) t[q] = kw[par][q];
#pragma unroll
    for (int h = C / 2; h > 0; h >>= 1)
#pragma unroll
      for (int q = 0; q < h; ++q) t[q] += t[q + h];
    const double2 pf = pc[par][f];
    const double hk = 0.5 * tau * (tau * fma(sc, fma(sc, t[0], 2.0 * pf.x), pf.y));
    const double w0 = tau * fma(sc, pf.x, pf.y) - hk;
#pragma unroll
    for (int u = 0; u < EPT; ++u) {
      const int i = tid + u * HTX;
      if (i >= f && i < n) {
        const double2 pi = pc[par][i];
        const double vi = i == f ? 1.0 : sc * xi[u];
        const double wi = tau * fma(sc, pi.x, pi.y) - hk * vi;
        const double ci = pi.y - fma(vi, w0, wi);
        w[i] = wi;
        xi[u] = i >= f + 2 ? ci : 0.0;
        xb[par ^ 1][i] = xi[u];
        if (i == f && head) ws[f] = ci;          // d[k+1]
        if (i == f + 1) {
          s_alpha = ci;
          if (head && k + 3 == n) ws[ld + n - 2] = ci;
        }
      }
    }
    sc_p = sc;
    if (__syncthreads_or(!ok)) {                   // a wait gave up: the same in the whole CTA
      ok = false;
      break;
    }
  }
  if (ok) {
    // d[n-1]: the last diagonal element with the last update
#pragma unroll
    for (int q = 0; q < CC; ++q)
      if (jc[q] == n - 1) {
#pragma unroll
        for (int r = 0; r < RM; ++r)
          if (lane + 32 * r == n - 1)
            ws[n - 1] = a[q][r] - 2.0 * (sc_p * xb[(n - 3) & 1][n - 1]) * w[n - 1];
      }
    if (head && tid == 0) {
      ws[ld + n - 1] = 0.0;
      ws[2 * ld + n - 2] = 0.0;
      ws[2 * ld + n - 1] = 0.0;
    }
  } else {
    for (int r = 0; r < 1000; ++r) __nanosleep(1000);   // messages still in flight land
  }
  cluster_sync_all();                              // no CTA leaves before the others are done
  if (!ok && tid == 0) ws[-k0] = __longlong_as_double(TRID_GAVE_UP);
}

constexpr int CT = 64;               // threads of k_trid_sturm
constexpr int CWARPS = CT / 32;

// Eigenvalues of the tridiagonal matrices, on the whole chip, in CTAs of two warps (one wave over
// all schedulers at n = 345: 55 us against 121 us with 256-thread CTAs, which leave most idle), by
// multisection, P lanes per eigenvalue (each counts at
// one of the P interior points of the interval, which shrinks by P + 1 per round), CT / P
// eigenvalues per CTA: blockIdx.x = chunk, blockIdx.y = task.
template <int P>
__global__ void __launch_bounds__(CT)
k_trid_sturm(double* __restrict__ base, const TridTask* __restrict__ tasks) {
  grid_entry();
  const TridTask tk = tasks[blockIdx.y];
  const int n = tk.n;
  if (int(blockIdx.x) * (CT / P) >= n) return;
  extern __shared__ double sm[];
  double* d = sm;
  double* e2 = sm + n;
  __shared__ double s_lo[CWARPS], s_hi[CWARPS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double* ws = base + tk.ws_off;
  if (__double_as_longlong(ws[0]) == TRID_GAVE_UP) {   // no tridiagonal matrix: pass it on
    const int ei = int(blockIdx.x) * (CT / P) + tid / P;
    if (tid % P == 0 && ei < n) base[tk.w_off + ei] = ws[0];
    return;
  }
  double lo = 1e300, hi = -1e300;          // Gershgorin interval
  bool fin = true;
  for (int i = tid; i < n; i += CT) {
    const double di = ws[i], ei = i + 1 < n ? ws[n + i] : 0.0, ep = i > 0 ? ws[n + i - 1] : 0.0;
    d[i] = di;
    e2[i] = ei;
    const double r = fabs(ei) + fabs(ep);
    lo = fmin(lo, di - r);
    hi = fmax(hi, di + r);
    fin &= isfinite(di) && isfinite(ei);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(FULL, lo, o));
    hi = fmax(hi, __shfl_xor_sync(FULL, hi, o));
  }
  if (lane == 0) { s_lo[warp] = lo; s_hi[warp] = hi; }
  if (!__syncthreads_and(fin)) {           // no eigenvalue of a NaN or an infinity is a number
    const int ei = int(blockIdx.x) * (CT / P) + tid / P;
    if (tid % P == 0 && ei < n) base[tk.w_off + ei] = __longlong_as_double(0x7ff8000000000000LL);
    return;
  }
#pragma unroll
  for (int q = 0; q < CWARPS; ++q) {
    lo = fmin(lo, s_lo[q]);
    hi = fmax(hi, s_hi[q]);
  }
  double back;                             // the counts run on T with a norm in [1, 2)
  const double scale = unit_scale(fmax(fabs(lo), fabs(hi)), back);
  lo *= scale;
  hi *= scale;
  for (int i = tid; i < n; i += CT) {
    const double ei = e2[i] * scale;
    d[i] *= scale;
    e2[i] = ei * ei;
  }
  __syncthreads();
  const double pad = 2.2e-16 * fmax(fabs(lo), fabs(hi)) + 1e-300;
  lo -= pad;
  hi += pad;
  const double tol = 8.9e-16 * fmax(fabs(lo), fabs(hi));
  const int ei = int(blockIdx.x) * (CT / P) + tid / P, h = tid % P;
  const int target = n - 1 - ei;           // i-th largest = (n-1-i)-th smallest
  const double frac = 1.0 / double(P + 1);
  bool done = ei >= n;
  double a = lo, b = hi;
  for (int it = 0; it < 200; ++it) {
    if (__all_sync(FULL, done)) break;
    bool below = false;
    const double wd = b - a;
    if (!done) {
      const double xl = a + wd * frac, xh = a + wd * (double(P) * frac);
      if (wd <= tol || !(a < xl && xl < xh && xh < b)) done = true;   // converged / no progress
      else below = sturm_lagged(d, e2, n, a + wd * (double(h + 1) * frac)) > target;
    }
    const unsigned bal = __ballot_sync(FULL, below);
    if (!done) {
      const unsigned bits = (bal >> (lane - h)) & ((1u << P) - 1u);
      if (bits == 0) {
        a = a + wd * (double(P) * frac);
      } else {
        const int g = __ffs(bits) - 1;
        const double xg = a + wd * (double(g + 1) * frac);
        if (g > 0) a = a + wd * (double(g) * frac);
        b = xg;
      }
    }
  }
  if (h == 0 && ei < n) base[tk.w_off + ei] = 0.5 * (a + b) * back;
}

}  // namespace

bool trid_gave_up(double w) {
  long long b;
  std::memcpy(&b, &w, sizeof b);
  return b == TRID_GAVE_UP;
}

void launch_trid_cluster(cudaStream_t s, double* base, const TridTask* tasks, int ntasks,
                         int max_n, int64_t sum_n) {
  if (ntasks <= 0) return;
  if (max_n > HN) {                    // such blocks come first
    const size_t sl = sizeof(double) * 7 * size_t(max_n);
    raise_smem_limit(reinterpret_cast<const void*>(k_trid_lead), sl);
    allow_wide_clusters(reinterpret_cast<const void*>(k_trid_lead));
    launch_cluster_k(k_trid_lead, LC, ntasks * LC, LT, sl, s, base, tasks);
    count_launch();
  }
  auto go = [&](auto kernel, int c) {
    allow_wide_clusters(reinterpret_cast<const void*>(kernel));
    launch_cluster_k(kernel, c, ntasks * c, HTX, 0, s, base, tasks);
  };
  // 16 CTAs halve the sweep, which is what a step of a larger block spends its time on (n = 345:
  // 0.49 against 0.57 ms; below 256 rows the two are equal), but only eight such clusters fit on
  // the chip at once
  const bool wide = max_n > 352 || ntasks <= 8;
  if (max_n <= 112) go(k_trid_cluster<4, 2, 8>, 8);
  else if (max_n <= 160) go(k_trid_cluster<5, 3, 8>, 8);
  else if (max_n <= 224) go(k_trid_cluster<7, 4, 8>, 8);
  else if (max_n <= 256) go(k_trid_cluster<8, 5, 8>, 8);
  else if (!wide) go(k_trid_cluster<11, 7, 8>, 8);
  else if (max_n <= 320) go(k_trid_cluster<10, 3, 16>, 16);
  else if (max_n <= 352) go(k_trid_cluster<11, 4, 16>, 16);
  else if (max_n <= 448) go(k_trid_cluster<14, 4, 16>, 16);
  else go(k_trid_cluster<16, 5, 16>, 16);
  count_launch();
  const size_t ss = sizeof(double) * 2 * size_t(max_n);
  // 16 lanes per eigenvalue need 13 rounds and 8 lanes 16, but twice the warps: worth it while
  // they are fewer than the schedulers
  if (sum_n * 16 <= int64_t(device_sm_count()) * 128) {
    const dim3 g((max_n + CT / 16 - 1) / (CT / 16), ntasks);
    launch_k(k_trid_sturm<16>, g, CT, ss, s, base, tasks);
  } else {
    const dim3 g((max_n + CT / 8 - 1) / (CT / 8), ntasks);
    launch_k(k_trid_sturm<8>, g, CT, ss, s, base, tasks);
  }
  count_launch();
}

}  // namespace dmrg
