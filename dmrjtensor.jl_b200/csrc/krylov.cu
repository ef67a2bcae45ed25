// krylov.cu -- the vector part of a Krylov step in ONE launch: one cluster of 16 CTAs holds the
// vector in registers (up to KRY_MAX elements) and takes every dot product, subtraction and
// normalisation between two Heff applications, where the general kernels (vec_kernels.cu) need a
// launch for each: nine for a Lanczos iteration with re-orthogonalisation (45 us of kernels at
// n = 40,000), three for the first half of the 2-vector step and three for its end, two for a
// normalisation.
//
// The dot products are summed in the order of the general kernels: 256-element blocks (a warp's
// 32 elements by shuffles over 16, 8, 4, 2, 1, the block's eight warps one after the other), then
// the block sums the same way. The numbers are therefore the same bit for bit, and the line at
// KRY_MAX, where the general kernels' bandwidth begins to count, changes none.
//
// What bounds it: latency -- ~0.8 us per set of dot products (shuffles, exchange of block sums
// through distributed shared memory, one cluster barrier), not the ~1 MB it reads.
#include <algorithm>

#include "cluster.cuh"
#include "kernels.cuh"
#include "launch.cuh"

namespace dmrg {
namespace {

constexpr int KC = 16;               // CTAs of the cluster
constexpr int KT = 512;              // threads of a CTA: two blocks of the summation order
constexpr int KW = KT / 32;
constexpr int64_t KST = KC * KT;     // elements of one round over the cluster
static_assert(KRY_MAX == 8 * KST, "at most eight elements per thread");
constexpr size_t KRY_SMEM = 227 * 1024 - 1024;
constexpr unsigned FULLM = 0xffffffffu;

// Dynamic shared memory, in doubles: block sums of the dot products of a set, by parity (2 x nd x
// nb, nb = 2 KC nq), the warps' sums (nd x nq x KW), the final warp sums (nd x 8), the results
// (nd), and the cached slices of Krylov vectors (nq KT each).
__host__ __device__ inline size_t kry_fixed(int nd, int nq) {
  return size_t(nd) * (2 * 2 * KC * nq + nq * KW + 8 + 1);
}

// Sums v[0..N) over the warp in the shuffle order 16, 8, ..., 1; lane l returns the sum of v[idx]
// with idx = the bits 4, 3, ... of l as bits 0, 1, ... (all lanes that share them agree).
template <int N, int MASK>
__device__ __forceinline__ double wsum_down(const double (&v)[N], int lane) {
  if constexpr (N == 1) {
    double s = v[0];
#pragma unroll
    for (int m = MASK; m > 0; m >>= 1) s += __shfl_xor_sync(FULLM, s, m);
    return s;
  } else {
    constexpr int H = (N + 1) / 2;
    const bool up = lane & MASK;
    double u[H];
#pragma unroll
    for (int p = 0; p < H; ++p) {
      const double lo = v[2 * p], hi = 2 * p + 1 < N ? v[(2 * p + 1) % N] : 0.0;
      u[p] = (up ? hi : lo) + __shfl_xor_sync(FULLM, up ? lo : hi, MASK);
    }
    return wsum_down<H, MASK / 2>(u, lane);
  }
}

struct Sums {
  double *part, *red, *red2, *dot;
  int nd, nq, rank, par;
};

// The k dot products with the threads' elements: term(d, q) = this thread's product of dot d for
// its q-th element. Results in su.dot[0..k), the same in every CTA.
template <int NQ, class F>
__device__ __forceinline__ void dots(Sums& su, int k, F term) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nq = su.nq, nb = 2 * KC * nq;
  // lane bits 4, 3, 2 select the element whose sum a lane ends up with
  const int idx = NQ == 1 ? 0 : NQ == 2 ? (lane >> 4) & 1
                  : NQ == 4 ? ((lane >> 4) & 1) | ((lane >> 2) & 2)
                            : ((lane >> 4) & 1) | ((lane >> 2) & 2) | (lane & 4);
  const bool writer = (lane & (32 / NQ - 1)) == 0 && idx < nq;
#pragma unroll 2
  for (int d = 0; d < k; ++d) {
    double v[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) v[q] = term(d, q);
    const double s = wsum_down<NQ, 16>(v, lane);
    if (writer) su.red[(d * nq + idx) * KW + warp] = s;
  }
  __syncthreads();
  double* part = su.part + size_t(su.par) * su.nd * nb;
  for (int x = tid; x < k * nq * 2; x += KT) {
    const int d = x / (2 * nq), y = x - d * 2 * nq, q = y >> 1, half = y & 1;
    const double* r = su.red + (d * nq + q) * KW + half * 8;
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < 8; ++w) s += r[w];
    const unsigned a = smem_addr(&part[d * nb + (q * KC + su.rank) * 2 + half]);
#pragma unroll
    for (int c = 0; c < KC; ++c) peer_store(peer_addr(a, c), s);
  }
  cluster_sync_all();
  const int w8 = warp & 7;
  for (int d = warp >> 3; d < k; d += 2) {
    const int b = w8 * 32 + lane;              // block sums past the vector's end are zero
    double s = b < nb ? part[d * nb + b] : 0.0;
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) s += __shfl_xor_sync(FULLM, s, m);
    if (lane == 0) su.red2[d * 8 + w8] = s;
  }
  __syncthreads();
  if (tid < k) {
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += su.red2[tid * 8 + w];
    su.dot[tid] = t;
  }
  __syncthreads();
  su.par ^= 1;
}

// Lowest eigenpair (c0, c1) of [[a0, b], [b, a1]] by the rotations of the general Ritz kernel, in
// its arithmetic; b = 0 after a breakdown: the first vector alone.
__device__ __forceinline__ double ritz2(double a0, double b, double a1, double& c0, double& c1) {
  c0 = 1.0;
  c1 = 0.0;
  if (!(b > 0.0)) return a0;
  double A00 = a0, A10 = b, A01 = b, A11 = a1, V00 = 1.0, V10 = 0.0, V01 = 0.0, V11 = 1.0;
  for (int sweep = 0; sweep < 100; ++sweep) {
    const double off = __dmul_rn(A01, A01);
    const double dg = __dadd_rn(__dmul_rn(A00, A00), __dmul_rn(A11, A11));
    if (off < 1e-300 || off <= 1e-32 * dg) break;
    const double apq = A01;
    const double theta = (A11 - A00) / (2.0 * apq);
    const double t = (theta >= 0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
    const double c = 1.0 / sqrt(t * t + 1.0), sn = t * c;
    auto rotate = [&](double& p, double& q) {
      const double ap = p, aq = q;
      p = fma(c, ap, -__dmul_rn(sn, aq));   // the roundings of the general kernel
      q = fma(sn, ap, __dmul_rn(c, aq));
    };
    rotate(A00, A10);
    rotate(A01, A11);
    rotate(A00, A01);
    rotate(A10, A11);
    rotate(V00, V01);
    rotate(V10, V11);
  }
  const bool second = A11 < A00;
  c0 = second ? V01 : V00;
  c1 = second ? V11 : V10;
  return second ? A11 : A00;
}

// One cluster; n <= NQ KST. nd: dot products of the largest set; the last ncache of the Krylov
// vectors 0..j are held in shared memory (every thread its own elements).
template <int NQ>
__global__ void __launch_bounds__(KT)
k_krylov(int mode, double* __restrict__ K, double* __restrict__ H, int64_t n, double* s, int j,
         double betatest, int nd, int ncache) {
  grid_entry();
  extern __shared__ __align__(16) double smk[];
  const int rank = cluster_rank(), tid = threadIdx.x;
  const int nq = int((n + KST - 1) / KST);
  const int64_t i0 = int64_t(rank) * KT + tid;     // element q of this thread: i0 + q KST
  const int nb = 2 * KC * nq;
  Sums su;
  su.part = smk;
  su.red = su.part + size_t(2) * nd * nb;
  su.red2 = su.red + size_t(nd) * nq * KW;
  su.dot = su.red2 + size_t(nd) * 8;
  su.nd = nd; su.nq = nq; su.rank = rank; su.par = 0;
  double* cache = smk + (kry_fixed(nd, nq) + 1) / 2 * 2;
  bool in[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) in[q] = i0 + q * KST < n;
  const int c0 = j + 1 - ncache;                   // first cached vector
  if (mode == KRY_STEP) {                          // all on their way at once, vector j first
    for (int d = j; d >= c0; --d) {
#pragma unroll
      for (int q = 0; q < NQ; ++q)
        if (in[q])
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;"
                       :: "r"(smem_addr(cache + size_t((d - c0) * nq + q) * KT + tid)),
                          "l"(K + int64_t(d) * n + i0 + q * KST));
      if (d == j) asm volatile("cp.async.commit_group;");
    }
    asm volatile("cp.async.commit_group;");
  }
  double h[NQ];
  const double* src = mode == KRY_NORMALISE ? K : H;
#pragma unroll
  for (int q = 0; q < NQ; ++q) h[q] = in[q] ? src[i0 + q * KST] : 0.0;
  cluster_sync_all();                              // every CTA runs before any remote store
  if (mode == KRY_NORMALISE) {                     // K *= 1/|K|; s[j] = <K,K>
    dots<NQ>(su, 1, [&](int, int q) { return h[q] * h[q]; });
    const double v = su.dot[0];
    const double a = (v > 0.0) ? 1.0 / sqrt(v) : 1.0;
#pragma unroll
    for (int q = 0; q < NQ; ++q)
      if (in[q]) K[i0 + q * KST] = h[q] * a;
    if (rank == 0 && tid == 0) s[j] = v;
  } else if (mode == KRY_ALPHA) {
    const double* Kj = K + int64_t(j) * n + i0;
    dots<NQ>(su, 1, [&](int, int q) { return in[q] ? Kj[q * KST] * h[q] : 0.0; });
    if (rank == 0 && tid == 0) s[lz::ALPHA + j] = su.dot[0];
  } else if (mode == KRY_LAST2) {
    double k[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) k[q] = in[q] ? K[n + i0 + q * KST] : 0.0;
    const double a0 = s[lz::ALPHA], b = s[lz::BETA];
    dots<NQ>(su, 1, [&](int, int q) { return k[q] * h[q]; });
    const double a1 = su.dot[0];
    double c0, c1;
    const double en = ritz2(a0, b, a1, c0, c1);
#pragma unroll
    for (int q = 0; q < NQ; ++q)
      if (in[q]) H[i0 + q * KST] = fma(c1, k[q], __dmul_rn(c0, K[i0 + q * KST]));
    if (rank == 0 && tid == 0) {
      s[lz::ALPHA + 1] = a1;
      s[lz::EN] = en;
      s[lz::COEF] = c0;
      s[lz::COEF + 1] = c1;
    }
  } else {
    double b2;
    if (mode == KRY_FIRST) {
      double k[NQ];
#pragma unroll
      for (int q = 0; q < NQ; ++q) k[q] = in[q] ? K[i0 + q * KST] : 0.0;
      dots<NQ>(su, 2, [&](int d, int q) { return k[q] * (d == 0 ? k[q] : h[q]); });
      const double kk = su.dot[0], kh = su.dot[1];
      __syncthreads();
      const double nn = sqrt(kk), inv = 1.0 / nn, a1 = kh / nn;
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        k[q] *= inv;
        h[q] = h[q] - a1 * k[q];
        if (in[q]) K[i0 + q * KST] = k[q];
      }
      if (rank == 0 && tid == 0) {
        s[lz::KK] = kk;
        s[lz::KH] = kh;
        s[lz::ALPHA] = a1;
      }
    } else {
      // element q of K_d, 0 past the end
      auto kv = [&](int d, int q) {
        if (!in[q]) return 0.0;
        return d >= c0 ? cache[size_t((d - c0) * nq + q) * KT + tid]
                       : K[int64_t(d) * n + i0 + q * KST];
      };
      const double be = j > 0 ? -1.0 * s[lz::BETA + j - 1] : 0.0;
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      dots<NQ>(su, 1, [&](int, int q) { return kv(j, q) * h[q]; });
      const double al = -1.0 * su.dot[0];
      if (rank == 0 && tid == 0) s[lz::ALPHA + j] = su.dot[0];
      __syncthreads();
      asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        h[q] = al * kv(j, q) + h[q];
        if (j > 0) h[q] = be * kv(j - 1, q) + h[q];
      }
      for (int pass = 0; pass < 2; ++pass) {       // full re-orthogonalisation (CGS2)
        dots<NQ>(su, j + 1, [&](int d, int q) { return kv(d, q) * h[q]; });
#pragma unroll 2
        for (int d = 0; d <= j; ++d) {
          const double c = su.dot[d];
#pragma unroll
          for (int q = 0; q < NQ; ++q) h[q] -= c * kv(d, q);
        }
        __syncthreads();
      }
    }
    dots<NQ>(su, 1, [&](int, int q) { return h[q] * h[q]; });
    b2 = su.dot[0];
    const bool act = (j == 0) || (s[lz::ACT + j] != 0.0);
    const double b = sqrt(b2);
    const bool ok = act && (b > betatest);
    const double r = ok ? 1.0 / b : 0.0;
    double* Kn = K + int64_t(j + 1) * n;           // the next vector
#pragma unroll
    for (int q = 0; q < NQ; ++q)
      if (in[q]) Kn[i0 + q * KST] = ok ? r * h[q] : 0.0;
    if (rank == 0 && tid == 0) {
      s[lz::B2 + j] = b2;
      s[lz::BETA + j] = ok ? b : 0.0;
      s[lz::ACT + j + 1] = ok ? 1.0 : 0.0;
    }
  }
  cluster_sync_all();                              // no CTA leaves before the others' stores landed
}

template <int NQ>
void go(cudaStream_t s, int mode, double* K, double* H, int64_t n, double* scal, int j,
        double betatest) {
  const int nq = int((n + KST - 1) / KST);
  const int nd = mode == KRY_STEP ? j + 1 : (mode == KRY_FIRST ? 2 : 1);
  const size_t fixed = (kry_fixed(nd, nq) + 1) / 2 * 2 * sizeof(double);
  const size_t slice = size_t(nq) * KT * sizeof(double);
  const int ncache = mode == KRY_STEP ? int(std::min<size_t>(j + 1, (KRY_SMEM - fixed) / slice)) : 0;
  const size_t sm = fixed + ncache * slice;
  raise_smem_limit(reinterpret_cast<const void*>(k_krylov<NQ>), sm);
  allow_wide_clusters(reinterpret_cast<const void*>(k_krylov<NQ>));
  launch_cluster_k(k_krylov<NQ>, KC, KC, KT, sm, s, mode, K, H, n, scal, j, betatest, nd, ncache);
  count_launch();
}

}  // namespace

bool launch_krylov(cudaStream_t s, int mode, double* K, double* H, int64_t n, double* scal, int j,
                   double betatest) {
  if (n <= 0 || n > KRY_MAX) return false;
  if (n <= KST) go<1>(s, mode, K, H, n, scal, j, betatest);
  else if (n <= 2 * KST) go<2>(s, mode, K, H, n, scal, j, betatest);
  else if (n <= 4 * KST) go<4>(s, mode, K, H, n, scal, j, betatest);
  else go<8>(s, mode, K, H, n, scal, j, betatest);
  return true;
}

}  // namespace dmrg
