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

// The plan's word on the rows of the stream that belong to no sequence: one past the last token of the
// last one, and whether there are others in front of it (padding).
constexpr int kPlanGaps = 1 << 30;

// Clears the rows of P (`vec` 16-byte pieces each) that belong to no sequence, and so to no work item;
// every CTA takes a share. The sequences lie in ascending order; the padding in front of one is cleared
// with its first tile.
__device__ __forceinline__ void clear_outside(const int* plan, int capacity, const int* seq_start,
                                              const int* seq_end, __nv_bfloat16* P, long long ld, int T,
                                              int vec) {
  const int word = plan[1 + 2 * capacity + 1];
  if (word < 0) return;
  auto clear = [&](int row) {
    for (int v = threadIdx.x; v < vec; v += blockDim.x)
      *reinterpret_cast<uint4*>(P + 1LL * row * ld + v * 8) = make_uint4(0u, 0u, 0u, 0u);
  };
  for (int row = (word & ~kPlanGaps) + int(blockIdx.x); row < T; row += gridDim.x) clear(row);
  if ((word & kPlanGaps) == 0) return;
  const AttnPlanView view{plan};
  const int n = view.count();
  const int per = int(gridDim.x) > n && n > 0 ? int(gridDim.x) / n : 1;   // CTAs per tile
  for (int w = blockIdx.x; w < n * per; w += gridDim.x) {
    const int i = w % n;
    if (view.tile(i) != 0) continue;
    int lo = view.seq(i);
    const int end = seq_start[lo];
    while (lo > 0 && seq_end[lo - 1] <= seq_start[lo - 1]) --lo;   // (sequences without tokens have no tile)
    for (int row = (lo > 0 ? seq_end[lo - 1] : 0) + w / n; row < end; row += per) clear(row);
  }
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
