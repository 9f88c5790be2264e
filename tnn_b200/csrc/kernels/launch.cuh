// Programmatic dependent launch for chains of kernels in one stream. A kernel launched with launch_dependent() may become
// resident while the kernel before it in the stream still runs; it sets itself up (barriers, tensor memory, descriptor
// prefetch) and calls grid_dep_wait(), which returns when the kernel before it has finished and its writes are visible.
// A kernel that calls grid_dep_launch() lets its successor become resident from then on.
//
// Rules that keep this equivalent to plain stream order:
//   * every kernel launched with launch_dependent() executes grid_dep_wait() in every thread before its first access to
//     global memory, on every path (so "finished" is transitive along the chain);
//   * grid_dep_launch() comes after the kernel holds everything it needs to finish, tensor memory above all: a successor
//     resident on the same SM could otherwise take the columns and wait for this kernel, which would wait for them;
//   * no pointer parameter of such a kernel is __restrict__. The kernel before it may still write what it reads, so the
//     promise would be false, and under it a load may take the read-only path or move above the wait. The work lies in a
//     device function with __restrict__ parameters that the kernel calls after grid_dep_wait(), when the promise holds
//     and the compiler can again move loads across stores;
//   * kernels that wait for other GPUs use neither.
// Both calls do nothing in a kernel that was launched the ordinary way.
//
// Where it pays: kernels launched one by one, between which the device idles while the next grid is set up (GPT-2 medium
// forward pass, 171 launches: 4439 -> 4346 us). Not in a captured graph, whose replay has the next kernel ready anyway and
// where early blocks only take slots from running ones (GPT-2 small step, 293 kernels: 11.27 -> 11.46 ms): a launch that is
// being captured becomes a plain one.
#pragma once
#include <cuda_runtime.h>

namespace tnnb {

__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// The same with clusters of `cluster` blocks (1: none).
template <typename... KArgs, typename... Args>
static inline cudaError_t launch_dependent_cluster(void (*kern)(KArgs...), int cluster, dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                                   const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  cfg.numAttrs = (cudaStreamIsCapturing(st, &capture) == cudaSuccess && capture == cudaStreamCaptureStatusNone) ? 1 : 0;
  if (cluster > 1) {
    cudaLaunchAttribute& c = attr[cfg.numAttrs++];
    c.id = cudaLaunchAttributeClusterDimension;
    c.val.clusterDim.x = cluster;
    c.val.clusterDim.y = c.val.clusterDim.z = 1;
  }
  return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}
template <typename... KArgs, typename... Args>
static inline cudaError_t launch_dependent(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, const Args&... args) {
  return launch_dependent_cluster(kern, 1, grid, block, smem, st, args...);
}

}  // namespace tnnb
