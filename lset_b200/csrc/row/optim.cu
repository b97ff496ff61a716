// Optimiser kernels over flat fp32 buffers: sum of squares (for the global gradient norm), the clip
// coefficient, and a fused AdamW step that also writes the bf16 compute copy of the parameters and
// clears the gradient. The clip coefficient stays on the device, so a step needs no host sync. A step
// takes all buffers of a model (one per layer) in a launch each: as launches per buffer, 29 layers of
// 16 M parameters spent 0.3 ms of 3.7 between them, and a small model's host most of the step on them.
// Replaces torch.optim.AdamW(fused=True) and clip_grad_norm_ (lset/train/engine.py:258-264,399-406).
#include "optim.h"

#include "../common/row.cuh"

namespace lb {
namespace {

using bf16 = __nv_bfloat16;

constexpr int kBatch = 40;       // buffers of one launch (its arguments hold the list)
constexpr int kChunk = 4096;     // elements of one CTA at a time

struct Groups {
  LbOptGroup g[kBatch];
  long long first[kBatch + 1];   // chunks in front of each buffer
  int n;
};

// Buffer and chunk within it of the c-th chunk of the list; `at` remembers the buffer (c only grows).
__device__ __forceinline__ long long find_chunk(const Groups& a, long long c, int& at) {
  while (at + 1 < a.n && c >= a.first[at + 1]) ++at;
  return c - a.first[at];
}

__global__ void __launch_bounds__(256)
    sumsq_partial_kernel(const __grid_constant__ Groups a, float* __restrict__ partial) {
  __shared__ float sred[8];
  float s[2] = {0.f, 0.f};
  int at = 0;
  for (long long c = blockIdx.x; c < a.first[a.n]; c += gridDim.x) {
    const long long e0 = find_chunk(a, c, at) * kChunk;
    const LbOptGroup& g = a.g[at];
    const float* x = g.g + e0;
    const int n = int(g.n - e0 < kChunk ? g.n - e0 : kChunk);
    float t = 0.f;
    if (n == kChunk) {
      float4 v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = reinterpret_cast<const float4*>(x)[i * 256 + threadIdx.x];
#pragma unroll
      for (int i = 0; i < 4; ++i) t += v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
    } else {
      for (int i = threadIdx.x; i < n; i += 256) t += x[i] * x[i];
    }
    s[0] += g.slot == 0 ? t : 0.f;
    s[1] += g.slot == 0 ? 0.f : t;
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const float t = row_sum<256>(s[k], sred);
    if (threadIdx.x == 0) partial[2 * blockIdx.x + k] = t;
    __syncthreads();
  }
}

// out[k] = sum of the partial sums of slot k.
__global__ void __launch_bounds__(256)
    sumsq_final_kernel(const float* __restrict__ partial, int P, float* __restrict__ out) {
  __shared__ float sred[8];
  float s[2] = {0.f, 0.f};
  for (int i = threadIdx.x; i < P; i += blockDim.x) {
    s[0] += partial[2 * i];
    s[1] += partial[2 * i + 1];
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const float t = row_sum<256>(s[k], sred);
    if (threadIdx.x == 0) out[k] = t;
    __syncthreads();
  }
}

// coef_out[0] = min(1, max_norm / (norm + 1e-6)); coef_out[1] = norm. max_norm <= 0 disables.
// coef_out[2] = 1 when this step must not be applied: `fault` (nullable device float, e.g. the
// status words of all ranks summed) is non-zero, i.e. some kernel of the step gave up a bounded
// wait and the gradients cannot be trusted. The AdamW kernels return at once when they see it,
// so a faulted step leaves parameters and moments untouched without the host having to look.
// With `parts` (of a single rank) sumsq[0] is first formed as the sum of its two words and sumsq[1] from
// the status word.
__global__ void clip_coef_kernel(float* sumsq, float max_norm, float* __restrict__ coef_out,
                                 const float* fault, const float* __restrict__ parts,
                                 const int* __restrict__ status) {
  if (parts != nullptr) {
    sumsq[0] = parts[0] + parts[1];
    sumsq[1] = float(*status);
  }
  const float norm = sqrtf(sumsq[0]);
  coef_out[1] = norm;
  coef_out[0] = (max_norm > 0.f) ? fminf(1.f, max_norm / (norm + 1e-6f)) : 1.f;
  coef_out[2] = (fault != nullptr && fault[0] != 0.f) ? 1.f : 0.f;
}

struct AdamArgs {
  float lr, beta1, beta2, eps, wd, bc1, bc2_sqrt, grad_scale;
  const float* coef;  // nullable: [0] clip coefficient, [2] non-zero = skip this step
  int zero_grad;
};

__global__ void __launch_bounds__(256) adamw_kernel(const __grid_constant__ Groups groups, AdamArgs a) {
  if (a.coef != nullptr && a.coef[2] != 0.f) return;
  const float gs = a.grad_scale * (a.coef != nullptr ? a.coef[0] : 1.f);
  const float step = a.lr / a.bc1;
  const float decay = 1.f - a.lr * a.wd;
  auto update = [&](float& p, float gj, float& m, float& v) {
    gj *= gs;
    m = a.beta1 * m + (1.f - a.beta1) * gj;
    v = a.beta2 * v + (1.f - a.beta2) * gj * gj;
    const float denom = sqrtf(v) / a.bc2_sqrt + a.eps;
    p = p * decay - step * m / denom;
  };
  int at = 0;
  for (long long c = blockIdx.x; c < groups.first[groups.n]; c += gridDim.x) {
    const long long e0 = find_chunk(groups, c, at) * kChunk;
    const LbOptGroup& t = groups.g[at];
    const long long left = t.n - e0;
    const int n4 = int((left < kChunk ? left : kChunk) / 4);
#pragma unroll 1
    for (int k = threadIdx.x; k < n4; k += 256) {
      const long long i = e0 / 4 + k;
      float4 p = reinterpret_cast<float4*>(t.p)[i];
      float4 g = reinterpret_cast<float4*>(t.g)[i];
      float4 m = reinterpret_cast<float4*>(t.m)[i];
      float4 v = reinterpret_cast<float4*>(t.v)[i];
      float* pp = &p.x;
      float* gp = &g.x;
      float* mp = &m.x;
      float* vp = &v.x;
#pragma unroll
      for (int j = 0; j < 4; ++j) update(pp[j], gp[j], mp[j], vp[j]);
      reinterpret_cast<float4*>(t.p)[i] = p;
      reinterpret_cast<float4*>(t.m)[i] = m;
      reinterpret_cast<float4*>(t.v)[i] = v;
      if (a.zero_grad) reinterpret_cast<float4*>(t.g)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (t.p_bf16 != nullptr) {
        __nv_bfloat162 lo = __floats2bfloat162_rn(p.x, p.y);
        __nv_bfloat162 hi = __floats2bfloat162_rn(p.z, p.w);
        uint2 o;
        o.x = *reinterpret_cast<uint32_t*>(&lo);
        o.y = *reinterpret_cast<uint32_t*>(&hi);
        reinterpret_cast<uint2*>(t.p_bf16)[i] = o;
      }
    }
    if (left < kChunk) {   // the last elements of a buffer that is no multiple of four
      for (long long i = e0 + 4 * n4 + threadIdx.x; i < t.n; i += 256) {
        float p = t.p[i], m = t.m[i], v = t.v[i];
        update(p, t.g[i], m, v);
        t.p[i] = p;
        t.m[i] = m;
        t.v[i] = v;
        if (a.zero_grad) t.g[i] = 0.f;
        if (t.p_bf16 != nullptr) static_cast<bf16*>(t.p_bf16)[i] = __float2bfloat16_rn(p);
      }
    }
  }
}

// The next buffers of a list that one launch takes.
int take_groups(const LbOptGroup* groups, int count, int from, Groups* a) {
  *a = Groups{};
  long long chunks = 0;
  int i = from;
  for (; i < count && a->n < kBatch; ++i) {
    if (groups[i].n <= 0) continue;
    a->first[a->n] = chunks;
    a->g[a->n++] = groups[i];
    chunks += (groups[i].n + kChunk - 1) / kChunk;
  }
  a->first[a->n] = chunks;
  return i;
}

bool aligned(const void* p, uintptr_t mask) { return (reinterpret_cast<uintptr_t>(p) & mask) == 0; }

}  // namespace
}  // namespace lb

using namespace lb;

// Floats of scratch for the sum of squares over `count` buffers.
extern "C" int lb_sumsq_scratch_floats(int count) {
  const int launches = (count + kBatch - 1) / kBatch;
  return 2 * row_num_sms() * 4 * (launches > 0 ? launches : 1);
}

// out[k] = sum(g^2) over the buffers of slot k (0, 1).
extern "C" int lb_sumsq_groups(const LbOptGroup* groups, int count, float* scratch, float* out,
                               void* stream) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int cap = row_num_sms() * 4;
  int rows = 0;
  for (int i = 0; i < count; ++i)
    if (!aligned(groups[i].g, 15u)) return -3;
  for (int from = 0; from < count;) {
    Groups a;
    from = take_groups(groups, count, from, &a);
    if (a.n == 0) break;
    const int grid = int(a.first[a.n] < cap ? a.first[a.n] : cap);
    sumsq_partial_kernel<<<grid, 256, 0, st>>>(a, scratch + 2 * rows);
    rows += grid;
  }
  sumsq_final_kernel<<<1, 256, 0, st>>>(scratch, rows, out);
  return launch_rc();
}

// coef_out: 3 floats (see clip_coef_kernel); fault: nullable device float.
extern "C" int lb_clip_coef(float* sumsq, float max_norm, float* coef_out, const float* fault,
                            void* stream) {
  clip_coef_kernel<<<1, 1, 0, reinterpret_cast<cudaStream_t>(stream)>>>(sumsq, max_norm, coef_out,
                                                                        fault, nullptr, nullptr);
  return launch_rc();
}

// The same for a single rank: sumsq (2 floats) is written out of the two sums and the status word.
extern "C" int lb_clip_coef_local(const float* parts, const int* status, float max_norm, float* sumsq,
                                  float* coef_out, void* stream) {
  clip_coef_kernel<<<1, 1, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      sumsq, max_norm, coef_out, sumsq + 1, parts, status);
  return launch_rc();
}

extern "C" int lb_adamw_groups(const LbOptGroup* groups, int count, float lr, float beta1, float beta2,
                               float eps, float wd, float bc1, float bc2_sqrt, float grad_scale,
                               const float* coef, int zero_grad, void* stream) {
  for (int i = 0; i < count; ++i) {
    const LbOptGroup& g = groups[i];
    if (!aligned(g.p, 15u) || !aligned(g.g, 15u) || !aligned(g.m, 15u) || !aligned(g.v, 15u) ||
        !aligned(g.p_bf16, 7u))
      return -3;
  }
  const AdamArgs a{lr, beta1, beta2, eps, wd, bc1, bc2_sqrt, grad_scale, coef, zero_grad};
  const long long cap = 1LL * row_num_sms() * 16;
  for (int from = 0; from < count;) {
    Groups list;
    from = take_groups(groups, count, from, &list);
    if (list.n == 0) break;
    const long long chunks = list.first[list.n];
    adamw_kernel<<<int(chunks < cap ? chunks : cap), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        list, a);
  }
  return launch_rc();
}
