// Programmatic dependent launch: a kernel of a chain may be launched while the one in front of it
// is still running, do its set-up, and wait (pdl_wait) for that kernel's results before it touches
// them. Every kernel launched with `pdl` set executes pdl_wait before its first access to memory
// that another kernel writes; outside such a launch the wait returns at once. pdl_trigger lets the
// next kernel start; it comes after pdl_wait, so that whatever runs ahead of its own pdl_wait can
// rely on everything two kernels back.
#pragma once

#include <cuda_runtime.h>

namespace lb {

#ifdef __CUDACC__
__device__ __forceinline__ void pdl_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void pdl_trigger() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
#endif

// Set by the block runners around a chain of launches of one call (host thread local): kernels
// that support it are then launched with the programmatic attribute.
bool pdl_enabled();
struct PdlScope {
  explicit PdlScope(bool on);
  ~PdlScope();
  bool saved;
};

template <typename... KArgs, typename... Args>
inline int launch_pdl(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                      bool pdl, int cluster, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (cluster > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = cluster;
    attr[n].val.clusterDim.y = 1;
    attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (pdl) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kern, KArgs(args)...) == cudaSuccess ? 0 : -11;
}

}  // namespace lb
