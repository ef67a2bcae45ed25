// launch.cuh -- kernel launches with programmatic dependent launch (sm_90 and later).
//
// A bond step is two dozen short kernels in one stream, each depending on the one before. With
// an ordinary launch the next kernel is scheduled only after its predecessor has finished and
// its writes have been flushed, so every boundary costs a full launch latency on the device.
// Every kernel of this library therefore begins with grid_entry(): griddepcontrol.wait blocks
// until all kernels it depends on in the stream have COMPLETED and their memory operations are
// visible, then griddepcontrol.launch_dependents lets the next kernel in the stream be
// scheduled. Every launch goes through launch_k, which sets the programmatic-serialisation
// attribute, so the next kernel's launch and block set-up overlap the running kernel and its
// blocks start work the moment the running kernel completes.
//
// Ordering is unchanged: no thread touches global memory before its wait returns, so a kernel
// still sees every write of the kernels before it and never overwrites what they read. The
// trigger comes after the wait, so at most one kernel runs ahead in its set-up. A kernel whose
// predecessor in the stream is not a kernel (a copy, a memset, an event wait) is ordered after
// it as usual, and both instructions are no-ops in a kernel launched without the attribute.
#pragma once
#include <cuda_runtime.h>
#include <utility>

namespace dmrg {

__device__ __forceinline__ void grid_entry() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// The task that owns `tile` in a list sorted by first tile (tile0): the whole block looks at
// blockDim.x evenly spread tasks at once and narrows the range to the gap between two of them, so
// a list of up to blockDim.x tasks costs one round of loads where a binary search by every thread
// costs log2(ntasks) dependent ones (~600 cycles each from L2: the mixing and copy launches of a
// U(1) sweep took 9.4 and 6.1 us on average against 7.8 and 5.3 us). All threads call it.
template <class Task>
__device__ __forceinline__ int find_task(const Task* __restrict__ tasks, int ntasks, int tile) {
  int lo = 0, n = ntasks;                  // the owner is in [lo, lo + n)
  while (n > 1) {
    const int step = (n + int(blockDim.x) - 1) / int(blockDim.x);
    const int i = int(threadIdx.x) * step;
    const int c = __syncthreads_count(i < n && tasks[lo + i].tile0 <= tile);
    lo += (c - 1) * step;
    n = min(step, n - (c - 1) * step);
  }
  return lo;
}

// kernel<<<grid, block, smem, s>>>(args...) with programmatic stream serialisation allowed.
// Errors are left for the caller's cudaGetLastError().
template <typename... P, typename... A>
inline void launch_k(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                     A&&... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  (void)cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

// The same with thread-block clusters of c CTAs (grid: a multiple of c). Above 8 CTAs the size is
// not portable and has to be allowed first (allow_wide_clusters).
template <typename... P, typename... A>
inline void launch_cluster_k(void (*kernel)(P...), int c, dim3 grid, dim3 block, size_t smem,
                             cudaStream_t s, A&&... args) {
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = unsigned(c);
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  (void)cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

}  // namespace dmrg
