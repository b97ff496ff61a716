// Shared definitions of the varlen attention kernels.
//
// Tiling. Queries of the G = Hq / Hk heads that share one KV head are stacked along the M
// dimension of the MMA: a 128-row tile holds G heads x QT tokens (QT = 128 / G), so short
// sequences still fill the tensor-core tile and K/V tiles are loaded once per group. Row r of a
// tile is head g = r / QT, token tok0 + r % QT.
//
// Plan. Sequence lengths live on the device; a one-block planning kernel turns cu_seqlens into a
// list of (sequence, tile) pairs that every layer's forward and backward launch reuses.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace lb {

constexpr int kAttnKvBlock = 64;   // KV rows per inner step of the forward and dQ kernels
constexpr int kLog2e = 0;          // (placeholder to keep the namespace non-empty for constexprs)
constexpr float kLog2eF = 1.4426950408889634f;
constexpr float kLn2F = 0.6931471805599453f;

// plan[0] = number of tiles; then (sequence index, tile index within the sequence) pairs.
struct AttnPlanView {
  const int* data;
  __device__ __forceinline__ int count() const { return data[0]; }
  __device__ __forceinline__ int seq(int i) const { return data[1 + 2 * i]; }
  __device__ __forceinline__ int tile(int i) const { return data[2 + 2 * i]; }
};

// Rows of the stream behind the last sequence belong to no work item: every CTA clears a share of O's
// (`vec` = 16-byte pieces of a row).
__device__ __forceinline__ void clear_tail(const int* plan, int capacity, __nv_bfloat16* O,
                                           long long ldo, int T, int vec) {
  const int end = plan[1 + 2 * capacity + 1];
  if (end < 0) return;
  for (int row = end + int(blockIdx.x); row < T; row += gridDim.x)
    for (int v = threadIdx.x; v < vec; v += blockDim.x)
      *reinterpret_cast<uint4*>(O + 1LL * row * ldo + v * 8) = make_uint4(0u, 0u, 0u, 0u);
}

// Called by every CTA of a persistent kernel when it takes no more work: the last one puts the plan's
// work counter back to zero for the next layer's launch.
__device__ __forceinline__ void finish_grid(const int* plan, int capacity) {
  if (threadIdx.x != 0) return;
  unsigned* words = reinterpret_cast<unsigned*>(const_cast<int*>(plan)) + 1 + 2 * capacity;
  __threadfence();
  if (atomicAdd(&words[2], 1u) + 1u == gridDim.x) {
    words[0] = 0u;
    words[2] = 0u;
  }
}

}  // namespace lb
