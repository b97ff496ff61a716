// Label matrix of the contrastive losses -> what the streaming loss kernels read: int8 labels padded
// to a multiple of 32 columns (padding = -1, ignored) and the rows' statistics. One pass over the
// labels, which bounds it; as separate conversions, reductions and elementwise ops it was a dozen
// launches and four passes (1009 x 4036 fp32 labels: 62 us, here 9).
#include <stdint.h>

#include "../common/row.cuh"

namespace lb {
namespace {

constexpr int kLabelThreads = 256;

// lab8[r, c] = label (converted as a cast does); row_scale[r] = 1 / max(sum of the positive labels, 1);
// row_w[r] = 1 / (number of kept rows) for rows with a positive and a column that is not ignored,
// 0 for the others. Every CTA takes rows; the last one to finish turns the marks in row_w into weights.
template <typename T>
__global__ void __launch_bounds__(kLabelThreads)
    label_prep_kernel(const T* __restrict__ labels, long long ld, int Q, int K, int Kp,
                      signed char* __restrict__ lab8, float* __restrict__ row_scale,
                      float* row_w, int* counters /* kept rows, CTAs done; zero on entry */) {
  __shared__ int s_sum[kLabelThreads / 32], s_max[kLabelThreads / 32];
  __shared__ bool s_last;
  int kept = 0;
  for (int r = blockIdx.x; r < Q; r += gridDim.x) {
    const T* src = labels + r * ld;
    signed char* dst = lab8 + 1LL * r * Kp;
    int sum = 0, mx = -128;
    for (int c0 = threadIdx.x * 4; c0 < Kp; c0 += kLabelThreads * 4) {
      char4 v;
      signed char* e = reinterpret_cast<signed char*>(&v);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        int x = -1;
        if (c0 + i < K) {
          x = static_cast<signed char>(static_cast<int>(src[c0 + i]));
          sum += x > 0 ? x : 0;
          mx = max(mx, x);
        }
        e[i] = static_cast<signed char>(x);
      }
      *reinterpret_cast<char4*>(dst + c0) = v;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sum += __shfl_xor_sync(0xffffffffu, sum, o);
      mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if ((threadIdx.x & 31) == 0) {
      s_sum[threadIdx.x >> 5] = sum;
      s_max[threadIdx.x >> 5] = mx;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < kLabelThreads / 32; ++w) {
        sum += s_sum[w];
        mx = max(mx, s_max[w]);
      }
      const bool keep = sum > 0 && mx >= 0;
      row_scale[r] = 1.f / float(sum > 1 ? sum : 1);
      row_w[r] = keep ? 1.f : 0.f;
      kept += keep;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    atomicAdd(&counters[0], kept);
    __threadfence();
    s_last = atomicAdd(&counters[1], 1) + 1 == int(gridDim.x);
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const int n = *reinterpret_cast<volatile int*>(&counters[0]);
  const float w = 1.f / float(n > 1 ? n : 1);
  for (int r = threadIdx.x; r < Q; r += kLabelThreads)
    row_w[r] = *reinterpret_cast<volatile float*>(row_w + r) != 0.f ? w : 0.f;
}

}  // namespace
}  // namespace lb

using namespace lb;

// labels [Q, K], rows ld elements apart; kind: 0 = fp32, 1 = int64, 2 = int32, 3 = int8 / bool. Kp: K
// rounded up to a multiple of 32. counters: two ints.
extern "C" int lb_label_prep(const void* labels, int kind, long long ld, int Q, int K, int Kp,
                             void* lab8, float* row_scale, float* row_w, int* counters,
                             void* stream) {
  if (Q <= 0) return 0;
  if (K <= 0 || (Kp & 31) || Kp < K) return -3;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(counters, 0, 2 * sizeof(int), st) != cudaSuccess) return -12;
  const int cap = row_num_sms() * 8;
  const int grid = Q < cap ? Q : cap;
  signed char* out = static_cast<signed char*>(lab8);
#define LB_LABELS(T)                                                                         \
  label_prep_kernel<T><<<grid, kLabelThreads, 0, st>>>(static_cast<const T*>(labels), ld, Q, K, Kp, \
                                                       out, row_scale, row_w, counters)
  if (kind == 0) LB_LABELS(float);
  else if (kind == 1) LB_LABELS(long long);
  else if (kind == 2) LB_LABELS(int);
  else if (kind == 3) LB_LABELS(signed char);
  else return -3;
#undef LB_LABELS
  return launch_rc();
}
