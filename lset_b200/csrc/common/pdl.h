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
// The same for a kernel that streams `bytes` through registers. An early start costs it bandwidth: the SMs keep
// the division of their L1 that the GEMM in front runs with, nearly all of it shared memory, and loads on
// their way need lines of what is left. So above 96 MB such a kernel waits for the end of the one in front.
// Measured (us, early start / not, between its GEMMs): gated backward 22627 x 3072 144 / 111, 33280 x 12288
// 904 / 709 (alone 642, and 814 with the division set to shared memory); RMSNorm backward 22627 x 1024
// 49 / 42, 33280 x 4096 258 / 206 (with four CTAs an SM); RMSNorm 40280 x 1024 60 / 50; rotation of 40280 x 24
// heads 107 / 93. Steps
// with the line at 12 / 48 / 96 / 10^6 MB: 24 texts of 256 tokens encoded 5.68 / 5.62 / 5.55 / 5.55 ms,
// 64 texts 13.72 / 13.74 / 13.71 / 13.78; 12 pairs trained on 22.2 / 22.05 / 21.9 / 22.1, 6 pairs 15.0 /
// 14.8 / 14.8 / 14.8.
constexpr long long kPdlMaxBytes = 96 * 1000 * 1000;
bool pdl_enabled(long long bytes);
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
