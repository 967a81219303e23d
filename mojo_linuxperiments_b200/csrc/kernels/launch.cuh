// Host-side launch helper: cudaLaunchKernelEx with the programmatic-stream-serialisation attribute (so consecutive
// kernels of this library overlap their prologues with their predecessors' tails, also inside captured CUDA graphs)
// and, optionally, a thread-block cluster dimension.  B200RT_PDL=0 turns the attribute off (A/B measurements).
#pragma once
#include <cuda_runtime.h>
#include <cstdlib>
#include "trace.cuh"
#include "debug_check.cuh"

namespace b200 {

inline bool pdl_enabled() {
  static int v = -1;
  if (v < 0) {
    const char* e = std::getenv("B200RT_PDL");
    v = (e && e[0] == '0') ? 0 : 1;
  }
  return v != 0;
}

// internal linkage on purpose: the trace refresh below is per translation unit
// cluster.x 0: no cluster; programmatic: the kernel may start before its predecessor in the stream has completed (pdl_wait)
template <typename... KArgs, typename... Args>
static inline cudaError_t launch_with(bool programmatic, dim3 cluster, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                                      cudaStream_t stream, Args&&... args) {
  trace_refresh();
  debug_refresh();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  unsigned n = 0;
  if (programmatic && pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  if (cluster.x > 0) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = cluster.x;
    attr[n].val.clusterDim.y = cluster.y;
    attr[n].val.clusterDim.z = cluster.z;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

template <typename... KArgs, typename... Args>
static inline cudaError_t launch_ex(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster_x,
                             Args&&... args) {
  return launch_with(true, dim3(cluster_x > 0 ? cluster_x : 0, 1, 1), kernel, grid, block, smem, stream, static_cast<Args&&>(args)...);
}

// the same with a full cluster shape
template <typename... KArgs, typename... Args>
static inline cudaError_t launch_ex_cluster(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                            dim3 cluster, Args&&... args) {
  return launch_with(true, cluster, kernel, grid, block, smem, stream, static_cast<Args&&>(args)...);
}

// First kernel of a step: starts when everything before it in the stream has completed.  Kernels of the step read what was settled
// before it (lengths, positions, page table) ahead of their own dependency wait, which orders them behind their predecessor alone, and
// that one behind its own; this launch is what orders the whole chain behind the end of the step before (decode_advance,
// or copies and torch kernels, which release their dependents when they end without a promise that their writes are visible).
// In a captured step it is the first node, so it costs nothing there.
template <typename... KArgs, typename... Args>
static inline cudaError_t launch_first(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  return launch_with(false, dim3(0, 1, 1), kernel, grid, block, smem, stream, static_cast<Args&&>(args)...);
}

}  // namespace b200
