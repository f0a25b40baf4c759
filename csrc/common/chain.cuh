// Kernels that follow one another in a stream without the gap between them (programmatic dependent launch).
#pragma once
#include <cuda_runtime.h>
#include <utility>

namespace st {

// First statement (before any access to global memory) of a kernel that st::chained launches: waits until the kernel before it
// in the stream has completed and its writes are visible, then lets the next kernel's blocks be scheduled.  Without the launch
// attribute both are no-ops.  The arguments are the kernel's `const __restrict__` pointers: a compiler may move loads through
// those across anything, as what they point at counts as constant, so their addresses are made to depend on the wait.
template <typename... P>
__device__ __forceinline__ void chain_begin(P&... pointers) {
  int zero;
  asm volatile("griddepcontrol.wait;\nmov.u32 %0, 0;" : "=r"(zero)::"memory");
  ((pointers += zero), ...);
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Launch whose start-up overlaps the end of the kernel before it in the stream: the blocks are scheduled while that kernel's
// last ones drain, and chain_begin(), which every such kernel calls before it touches global memory, waits for its completion.
// Between two kernels of a forward pass this saves the 1 to 2 us of launch latency and ramp-up.  A captured launch is an
// ordinary one: a graph's edges to copies, fills and other streams' nodes only exist in that form.
// in_order: the launch of such a kernel that starts when the one before it has completed.  For one that reads much through L1: an SM keeps
// the split of its memory between L1 and shared memory while blocks follow one another, and a product leaves 28 KB of L1.  For one of
// a few heavy blocks per SM: early ones pile up on the SMs that fall free first.  And for one that leaves SMs to another stream: early
// blocks would hold SMs of that stream for as long as the kernel before them runs, beyond the number left to this one (of two
// products of 40 blocks, 330 us each, the second's blocks were there 50 to 80 us after the first's).
template <typename... P>
struct ChainedLaunch {
  void (*kernel)(P...);
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
  int cluster;
  bool early;
  template <typename... A>
  cudaError_t operator()(A&&... args) const {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusActive;
    const bool chain = early && cudaStreamIsCapturing(stream, &capture) == cudaSuccess && capture == cudaStreamCaptureStatusNone;
    cudaLaunchAttribute attr[2]{};
    unsigned n = 0;
    if (chain) {
      attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
      attr[n].id = cudaLaunchAttributeClusterDimension;
      attr[n].val.clusterDim.x = cluster;
      attr[n].val.clusterDim.y = 1;
      attr[n++].val.clusterDim.z = 1;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
  }
};
template <typename... P>
ChainedLaunch<P...> chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster = 1) {
  return {kernel, grid, block, smem, stream, cluster, true};
}
template <typename... P>
ChainedLaunch<P...> in_order(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
  return {kernel, grid, block, smem, stream, 1, false};
}

}  // namespace st
