// gemm_f64.cu -- persistent grouped FP64 GEMM on the FP64 tensor-core path (DMMA, m8n8k4).
//
// One launch executes every block product of one contraction step (all QN block triples), as a
// flat list of output tiles; each CTA walks tiles with a stride of gridDim.x. A tile accumulates
// over the K-segments of its task (stacked MPO channels, physical states). Operands may be
// transposed (NN, NT, TN) so that no permute copies are needed anywhere in the sweep. B200 has no
// tcgen05 FP64 kind; mma.sync f64 is the FP64 tensor-core instruction on sm_100a, and one warp per
// scheduler that issues nothing else reaches its 37 TFLOP/s.
//
// What bounds it is how much else those warps issue: a DMMA holds its warp's issue for about 18
// cycles, so copies, address arithmetic and barriers in the same warp add to that time. The warps
// of a CTA are therefore split: four fill a four-stage ring of shared-memory slices with cp.async
// (16 bytes where the operand's address and leading dimension allow, 8 otherwise), four only load
// fragments and issue DMMAs. The two sides meet at two named barriers per stage (filled, free),
// and the filling warps run ahead into the next tile. Slices lie in shared memory along the
// operand's own contiguous direction, padded so that both the copies and the fragment loads are
// free of bank conflicts; where that is the row direction one 16-byte load brings two fragments
// (rows 2g and 2g + 1 of a pair, a relabelling of the tile's rows).
//
// Every element of C is one chain of fused multiply-adds in the order of k, whatever the tile, so
// the tile shapes give the same bits. Measured (one CTA per tile-stride of three per SM; the
// kernel before had 64 x 64 or 32 x 32 tiles whose four warps did everything, best of the two):
//   1920 x 768 x 384    72 -> 45 us   (25 TFLOP/s)     5 GF, 2560 x 2048 x 512   228 -> 182 us
//   500 x 400 x 100    7.8 -> 5.1 us                   4 of 100 x 100 x 500       18 -> 7.1 us
//   225 x 180 x 45     4.0 -> 3.4 us                   24 ragged blocks, 0.3 GF   53 -> 30 us
#include <map>
#include <mutex>
#include <utility>
#include <atomic>

#include "kernels.cuh"
#include "launch.cuh"

namespace dmrg {
namespace {

constexpr int BK = 32, STAGES = 4;
constexpr int FILL_WARPS = 4, WARPS_M = 2, WARPS_N = 2, MMA_WARPS = WARPS_M * WARPS_N;
constexpr int FILL = 32 * FILL_WARPS, THREADS = FILL + 32 * MMA_WARPS;
constexpr int PER_SM = 3;         // CTAs per SM: 74 KB of shared memory, 80 registers a thread
static_assert(2 * STAGES + 1 <= 16, "two named barriers per stage, and barrier 0");

__device__ __forceinline__ void cp_async8(uint32_t smem, const double* gmem, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(smem), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_async16(uint32_t smem, const double* gmem, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem), "l"(gmem),
               "r"(bytes));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
// Barrier of all threads of the block: one side waits, the other only reports.
__device__ __forceinline__ void bar_sync(int id) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(THREADS) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(THREADS) : "memory");
}

// D(8x8) += A(8x4, row) * B(4x8, col). Lane l holds A[l>>2][l&3], B[l&3][l>>2],
// D[l>>2][2*(l&3) + {0,1}].
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

// The owner of `tile` in a list sorted by first tile, looked up by each warp on its own (the two
// sides of a block are at different tiles): one round of loads for up to 32 tasks.
__device__ __forceinline__ int find_task_warp(const GemmTask* __restrict__ tasks, int ntasks,
                                              int tile, int lane) {
  int lo = 0, n = ntasks;                  // the owner is in [lo, lo + n)
  while (n > 1) {
    const int step = (n + 31) / 32;
    const int i = lane * step;
    const int c = __popc(__ballot_sync(0xffffffffu, i < n && tasks[lo + i].tile0 <= tile));
    lo += (c - 1) * step;
    n = min(step, n - (c - 1) * step);
  }
  return lo;
}

// Slices of R rows (of A; columns of B) x BK of one operand. KF: K is the contiguous direction.
// A filling thread copies elements (f along memory, s + i hops across it) of every slice.
template <int R, bool KF>
struct Slice {
  static constexpr int LD = (KF ? BK : R) + 4;
  static constexpr int SIZE = (KF ? R : BK) * LD;       // doubles per stage
  static constexpr int F = KF ? BK : R;
  static constexpr int PER8 = R * BK / FILL, ACROSS8 = FILL / F;
  static constexpr int PER16 = PER8 / 2, ACROSS16 = 2 * ACROSS8;
  static_assert(PER16 >= 1 && F % 2 == 0 && FILL % F == 0, "whole rounds of copies");
  __device__ static __forceinline__ int at(int r, int k) { return KF ? r * LD + k : k * LD + r; }

  const double *src, *safe;   // this thread's first element of the next slice; any valid address
  int64_t hop, step;
  int f, s, rows;             // rows: of the tile, from its first one
  bool wide;
  __device__ __forceinline__ void start(const double* base, int ld, int r0, int nrows, int tid) {
    wide = ((reinterpret_cast<uintptr_t>(base) | (uintptr_t(ld) * sizeof(double))) & 15) == 0;
    f = wide ? (tid % (F / 2)) * 2 : tid % F;
    s = wide ? tid / (F / 2) : tid / F;
    safe = base;
    src = base + (KF ? int64_t(r0 + s) * ld + f : int64_t(s) * ld + r0 + f);
    hop = int64_t(wide ? ACROSS16 : ACROSS8) * ld;
    step = KF ? int64_t(BK) : int64_t(BK) * ld;
    rows = nrows - r0;
  }
  // Copies the next slice, of which k < kleft is inside the segment; the rest becomes zero.
  __device__ __forceinline__ void issue(uint32_t dst, int kleft) {
    const uint32_t d = dst + (s * LD + f) * sizeof(double);
    const double* p = src;
    if (rows >= R && kleft >= BK) {
      if (wide) {
#pragma unroll
        for (int i = 0; i < PER16; ++i, p += hop) cp_async16(d + i * ACROSS16 * LD * 8, p, 16);
      } else {
#pragma unroll
        for (int i = 0; i < PER8; ++i, p += hop) cp_async8(d + i * ACROSS8 * LD * 8, p, 8);
      }
    } else {
      const int along = (KF ? kleft : rows) - f, across = (KF ? rows : kleft) - s;
      if (wide) {
        const int bytes = max(0, min(2, along)) * 8;
#pragma unroll
        for (int i = 0; i < PER16; ++i, p += hop) {
          const int n = i * ACROSS16 < across ? bytes : 0;
          cp_async16(d + i * ACROSS16 * LD * 8, n ? p : safe, n);
        }
      } else {
        const int bytes = along > 0 ? 8 : 0;
#pragma unroll
        for (int i = 0; i < PER8; ++i, p += hop) {
          const int n = i * ACROSS8 < across ? bytes : 0;
          cp_async8(d + i * ACROSS8 * LD * 8, n ? p : safe, n);
        }
      }
    }
    src += step;
  }
};

// A warp's fragments over its W rows (columns): element g of fragment i is row row(i, g).
template <int W, bool KF>
struct Frag {
  static constexpr int N = W / 8;
  static constexpr bool PAIRS = !KF && W % 16 == 0;
  __device__ static __forceinline__ int row(int i, int g) {
    return PAIRS ? 16 * (i / 2) + 2 * g + (i & 1) : 8 * i + g;
  }
  // fragments with a row below `rows`
  __device__ static __forceinline__ int used(int rows) {
    return min(N, max(0, PAIRS ? (rows + 15) / 16 * 2 : (rows + 7) / 8));
  }
  // p: the lane's element of fragment 0
  template <class S>
  __device__ static __forceinline__ void load(double (&v)[N], const double* p, int k) {
    p += k * (KF ? 1 : S::LD);
    if constexpr (PAIRS) {
#pragma unroll
      for (int i = 0; i < N; i += 2) {
        const double2 w = *reinterpret_cast<const double2*>(p + S::at(8 * i, 0));
        v[i] = w.x;
        v[i + 1] = w.y;
      }
    } else {
#pragma unroll
      for (int i = 0; i < N; ++i) v[i] = p[S::at(8 * i, 0)];
    }
  }
};

template <int BM, int BN, bool TA, bool TB>
__global__ void __launch_bounds__(THREADS, PER_SM)
k_gemm_f64(const double* __restrict__ A0, const double* __restrict__ B0, double* __restrict__ C0,
           const GemmTask* __restrict__ tasks, int ntasks, const GemmSeg* __restrict__ segs,
           int total_tiles, GemmBatch batch) {
  grid_entry();
  using SA = Slice<BM, TA>;
  using SB = Slice<BN, !TB>;
  constexpr int WM = BM / WARPS_M, WN = BN / WARPS_N;
  using FA = Frag<WM, TA>;
  using FB = Frag<WN, !TB>;
  constexpr int MI = FA::N, NI = FB::N;
  constexpr int STAGE = SA::SIZE + SB::SIZE;
  constexpr int FILLED = 1, FREE = 1 + STAGES;    // named barriers of stage 0
  extern __shared__ __align__(16) double smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int all_tiles = total_tiles * batch.n;

  if (warp >= MMA_WARPS) {   // ---- the filling side
    const uint32_t ring = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    const int tid = threadIdx.x - 32 * MMA_WARPS;
    int n = 0, st = 0, done = 0;   // slices issued, their next stage, the next stage to report
    for (int all = blockIdx.x; all < all_tiles; all += gridDim.x) {
      const int set = batch.n > 1 ? all / total_tiles : 0, tile = all - set * total_tiles;
      const double* A = set == batch.n - 1 && batch.a_last ? batch.a_last : A0 + set * batch.a;
      const double* B = B0 + set * batch.b;
      const GemmTask tk = tasks[find_task_warp(tasks, ntasks, tile, lane)];
      const int local = tile - tk.tile0;
      const int m0 = (local % tk.tiles_m) * BM, n0 = (local / tk.tiles_m) * BN;
      for (int q = 0; q < tk.nseg; ++q) {
        const GemmSeg sg = segs[tk.seg0 + q];
        SA a;
        SB b;
        a.start(A + sg.a_off, sg.lda, m0, tk.M, tid);
        b.start(B + sg.b_off, sg.ldb, n0, tk.N, tid);
        for (int left = sg.K; left > 0; left -= BK) {
          if (n >= STAGES) bar_sync(FREE + st);
          const uint32_t d = ring + st * STAGE * sizeof(double);
          a.issue(d, left);
          b.issue(d + SA::SIZE * sizeof(double), left);
          cp_commit();
          if (++st == STAGES) st = 0;
          if (++n >= STAGES - 1) {
            cp_wait<STAGES - 2>();
            bar_arrive(FILLED + done);
            if (++done == STAGES) done = 0;
          }
        }
      }
    }
    cp_wait<0>();
    for (int open = min(n, STAGES - 2); open > 0; --open) {
      bar_arrive(FILLED + done);
      if (++done == STAGES) done = 0;
    }
    for (int i = 0; i < STAGES; ++i) {   // no report of the other side stays open
      if (n + i >= STAGES) bar_sync(FREE + st);
      if (++st == STAGES) st = 0;
    }
    return;
  }

  // ---- the multiplying side
  const int wm = warp % WARPS_M, wn = warp / WARPS_M;
  const int g = lane >> 2, t = lane & 3;
  const int a0 = SA::at(wm * WM + FA::row(0, g), t);
  const int b0 = SA::SIZE + SB::at(wn * WN + FB::row(0, g), t);
  int st = 0;
  for (int all = blockIdx.x; all < all_tiles; all += gridDim.x) {
    const int set = batch.n > 1 ? all / total_tiles : 0, tile = all - set * total_tiles;
    const GemmTask tk = tasks[find_task_warp(tasks, ntasks, tile, lane)];
    const int local = tile - tk.tile0;
    const int m0 = (local % tk.tiles_m) * BM + wm * WM;
    const int n0 = (local / tk.tiles_m) * BN + wn * WN;
    double acc[MI][NI][2];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < NI; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    const int mi_n = FA::used(tk.M - m0), ni_n = FB::used(tk.N - n0);
    const bool full = mi_n == MI && ni_n == NI;
    for (int q = 0; q < tk.nseg; ++q) {
      for (int left = segs[tk.seg0 + q].K; left > 0; left -= BK) {
        bar_sync(FILLED + st);
        const double* as = smem + st * STAGE + a0;
        const double* bs = smem + st * STAGE + b0;
        if (full && left >= BK) {
          double a[2][MI], b[2][NI];
          FA::template load<SA>(a[0], as, 0);
          FB::template load<SB>(b[0], bs, 0);
#pragma unroll
          for (int kk = 0; kk < BK / 4; ++kk) {
            if (kk + 1 < BK / 4) {
              FA::template load<SA>(a[(kk + 1) & 1], as, 4 * (kk + 1));
              FB::template load<SB>(b[(kk + 1) & 1], bs, 4 * (kk + 1));
            }
#pragma unroll
            for (int i = 0; i < MI; ++i)
#pragma unroll
              for (int j = 0; j < NI; ++j) dmma(acc[i][j], a[kk & 1][i], b[kk & 1][j]);
          }
        } else if (mi_n > 0 && ni_n > 0) {   // the remainder of K, the last rows and columns
          const int kn = min(BK, left);
#pragma unroll 1
          for (int kk = 0; kk < kn; kk += 4) {
            double a[MI], b[NI];
            FA::template load<SA>(a, as, kk);
            FB::template load<SB>(b, bs, kk);
#pragma unroll
            for (int i = 0; i < MI; ++i)
#pragma unroll
              for (int j = 0; j < NI; ++j)
                if (i < mi_n && j < ni_n) dmma(acc[i][j], a[i], b[j]);
          }
        }
        bar_arrive(FREE + st);
        if (++st == STAGES) st = 0;
      }
    }
    double* C = C0 + set * batch.c + tk.c_off;
#pragma unroll
    for (int i = 0; i < MI; ++i) {
      const int row = m0 + FA::row(i, g);
      if (row >= tk.M) continue;
#pragma unroll
      for (int j = 0; j < NI; ++j) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int col = n0 + FB::row(j, 2 * t + e);
          if (col < tk.N) {
            const int64_t idx = row + int64_t(col) * tk.ldc;
            double v = tk.alpha * acc[i][j][e];
            if (tk.beta != 0.0) v += tk.beta * C[idx];
            C[idx] = v;
          }
        }
      }
    }
  }
}

template <int BM, int BN, bool TA, bool TB>
void launch_variant(cudaStream_t s, const double* A, const double* B, double* C,
                    const GemmTask* tasks, int ntasks, const GemmSeg* segs, int total_tiles,
                    int nsm, const GemmBatch& batch) {
  constexpr size_t SM = sizeof(double) * STAGES * (Slice<BM, TA>::SIZE + Slice<BN, !TB>::SIZE);
  raise_smem_limit(reinterpret_cast<const void*>(k_gemm_f64<BM, BN, TA, TB>), SM);
  const int64_t all = int64_t(total_tiles) * batch.n;
  const int grid = int(all < int64_t(nsm) * PER_SM ? all : int64_t(nsm) * PER_SM);
  launch_k(k_gemm_f64<BM, BN, TA, TB>, grid, THREADS, SM, s, A, B, C, tasks, ntasks, segs,
           total_tiles, batch);
  count_launch();
}

template <int BM, int BN>
void dispatch_f64(cudaStream_t s, bool transA, bool transB, const double* A, const double* B,
                  double* C, const GemmTask* tasks, int ntasks, const GemmSeg* segs,
                  int total_tiles, int nsm, const GemmBatch& batch) {
  if (!transA && !transB)
    launch_variant<BM, BN, false, false>(s, A, B, C, tasks, ntasks, segs, total_tiles, nsm, batch);
  else if (!transA && transB)
    launch_variant<BM, BN, false, true>(s, A, B, C, tasks, ntasks, segs, total_tiles, nsm, batch);
  else if (transA && !transB)
    launch_variant<BM, BN, true, false>(s, A, B, C, tasks, ntasks, segs, total_tiles, nsm, batch);
  else
    launch_variant<BM, BN, true, true>(s, A, B, C, tasks, ntasks, segs, total_tiles, nsm, batch);
}

}  // namespace

void launch_gemm_f64(cudaStream_t s, int bn, bool transA, bool transB, const double* A,
                     const double* B, double* C, const GemmTask* tasks, int ntasks,
                     const GemmSeg* segs, int total_tiles, int nsm, const GemmBatch& batch) {
  if (total_tiles <= 0 || ntasks <= 0 || batch.n <= 0) return;
  if (bn == GEMM_BN_SMALL)
    dispatch_f64<GEMM_BM, GEMM_BN_SMALL>(s, transA, transB, A, B, C, tasks, ntasks, segs,
                                         total_tiles, nsm, batch);
  else
    dispatch_f64<GEMM_BM, GEMM_BN>(s, transA, transB, A, B, C, tasks, ntasks, segs, total_tiles,
                                   nsm, batch);
}

// Raises (never lowers) the dynamic shared-memory limit of a kernel on the current device. The
// limit is a property of the kernel shared by every host thread, so launchers on different
// threads (one context each) must never lower it below what another thread launches with.
void raise_smem_limit(const void* func, size_t bytes) {
  static std::mutex mu;
  static std::map<std::pair<int, const void*>, size_t> cur;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(mu);
  size_t& c = cur[{dev, func}];
  if (bytes > c &&
      cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes)) ==
          cudaSuccess)
    c = bytes;
}

void allow_wide_clusters(const void* func) {
  static std::mutex mu;
  static std::map<std::pair<int, const void*>, bool> done;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(mu);
  bool& d = done[{dev, func}];
  if (!d) d = cudaFuncSetAttribute(func, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
              cudaSuccess;
}

static std::atomic<long long> g_launches{0};
void count_launch(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
long long launch_count() { return g_launches.load(std::memory_order_relaxed); }

int device_sm_count() {
  int dev = 0, n = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n;
}

}  // namespace dmrg
