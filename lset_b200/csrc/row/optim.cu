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

// Buffers of one launch, and the work items in front of each: chunks of the update, CTAs of the sums.
struct Groups {
  LbOptGroup g[kBatch];
  long long first[kBatch + 1];
  int n;
};

// Buffer and chunk within it of the c-th chunk of the list; `at` remembers the buffer (c only grows).
__device__ __forceinline__ long long find_chunk(const Groups& a, long long c, int& at) {
  while (at + 1 < a.n && c >= a.first[at + 1]) ++at;
  return c - a.first[at];
}

// The sums of squares have one order, which depends on the sizes of the buffers alone and on no other
// buffer in front: within a buffer a walk of its own, then its CTAs, then the buffers one after the other. The
// clip coefficient multiplies every gradient, and a model of many layers turns one weight that is rounded to
// another bf16 value for its sake into a loss of the next step that differs by up to some per cent in small
// batches. (One walk over all buffers, in which a thread's sum runs from one to the next, has other last bits
// with every other list.)
//
// Bound by memory: four loads of a thread are requested together.
__global__ void __launch_bounds__(256)
    sumsq_partial_kernel(const __grid_constant__ Groups a, float* __restrict__ partial) {
  __shared__ float sred[8];
  int at = 0;
  const long long cta = find_chunk(a, blockIdx.x, at);
  const long long ctas = a.first[at + 1] - a.first[at];
  const float* x = a.g[at].g;
  const long long n = a.g[at].n, n4 = n / 4, step = ctas * 256;
  const float4* x4 = reinterpret_cast<const float4*>(x);
  float s = 0.f;
  auto add = [&](const float4& v) { s += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w; };
  long long i = cta * 256 + threadIdx.x;
  for (; i + 3 * step < n4; i += 4 * step) {
    float4 v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = x4[i + j * step];
#pragma unroll
    for (int j = 0; j < 4; ++j) add(v[j]);
  }
  for (; i < n4; i += step) add(x4[i]);
  if (cta == 0) {
    for (long long j = n4 * 4 + threadIdx.x; j < n; j += 256) s += x[j] * x[j];
  }
  s = row_sum<256>(s, sred);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
}

// sums[b], a CTA for each buffer: its sum in the component of its slot.
__global__ void __launch_bounds__(256)
    sumsq_buffer_kernel(const __grid_constant__ Groups a, const float* __restrict__ partial,
                        float2* __restrict__ sums) {
  __shared__ float sred[8];
  const int b = blockIdx.x;
  float s = 0.f;
  for (long long i = a.first[b] + threadIdx.x; i < a.first[b + 1]; i += 256) s += partial[i];
  s = row_sum<256>(s, sred);
  if (threadIdx.x == 0) sums[b] = a.g[b].slot == 0 ? make_float2(s, 0.f) : make_float2(0.f, s);
}

// out[k] = sum of the buffers' sums of slot k, one after the other.
__global__ void sumsq_final_kernel(const float2* __restrict__ sums, int n, float* __restrict__ out) {
  float2 t = make_float2(0.f, 0.f);
  for (int b0 = 0; b0 < n; b0 += 32) {
    const float2 v = b0 + int(threadIdx.x) < n ? sums[b0 + threadIdx.x] : make_float2(0.f, 0.f);
#pragma unroll
    for (int l = 0; l < 32; ++l) {
      t.x += __shfl_sync(0xffffffffu, v.x, l);
      t.y += __shfl_sync(0xffffffffu, v.y, l);
    }
  }
  if (threadIdx.x == 0) {
    out[0] = t.x;
    out[1] = t.y;
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

// The next buffers of a list that one launch takes; `items`: work items of a buffer of n elements.
template <typename Items>
int take_groups(const LbOptGroup* groups, int count, int from, Groups* a, Items items) {
  *a = Groups{};
  long long total = 0;
  int i = from;
  for (; i < count && a->n < kBatch; ++i) {
    if (groups[i].n <= 0) continue;
    a->first[a->n] = total;
    a->g[a->n++] = groups[i];
    total += items(groups[i].n);
  }
  a->first[a->n] = total;
  return i;
}

// CTAs that a buffer's sum of squares is cut into.
int sumsq_ctas(long long n) {
  const long long need = (n / 4 + 255) / 256, cap = 4LL * row_num_sms();
  return int(need < 1 ? 1 : (need > cap ? cap : need));
}

bool aligned(const void* p, uintptr_t mask) { return (reinterpret_cast<uintptr_t>(p) & mask) == 0; }

}  // namespace
}  // namespace lb

using namespace lb;

// Floats of scratch for the sums of squares of `count` buffers: two of each, then its CTAs' partial sums.
extern "C" int lb_sumsq_scratch_floats(int count) {
  return (count > 0 ? count : 1) * (2 + 4 * row_num_sms());
}

// out[k] = sum(g^2) over the buffers of slot k (0, 1). scratch: 8-byte aligned.
extern "C" int lb_sumsq_groups(const LbOptGroup* groups, int count, float* scratch, float* out,
                               void* stream) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (!aligned(scratch, 7u)) return -3;
  float2* sums = reinterpret_cast<float2*>(scratch);
  float* partial = scratch + 2LL * (count > 0 ? count : 1);
  int buffers = 0;
  for (int i = 0; i < count; ++i)
    if (!aligned(groups[i].g, 15u)) return -3;
  for (int from = 0; from < count;) {
    Groups a;
    from = take_groups(groups, count, from, &a, sumsq_ctas);
    if (a.n == 0) break;
    sumsq_partial_kernel<<<unsigned(a.first[a.n]), 256, 0, st>>>(a, partial);
    sumsq_buffer_kernel<<<a.n, 256, 0, st>>>(a, partial, sums + buffers);
    partial += a.first[a.n];
    buffers += a.n;
  }
  sumsq_final_kernel<<<1, 32, 0, st>>>(sums, buffers, out);
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
    from = take_groups(groups, count, from, &list, [](long long n) { return (n + kChunk - 1) / kChunk; });
    if (list.n == 0) break;
    const long long chunks = list.first[list.n];
    adamw_kernel<<<int(chunks < cap ? chunks : cap), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        list, a);
  }
  return launch_rc();
}
