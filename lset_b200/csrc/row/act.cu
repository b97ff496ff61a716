// Gated activations and GELU, forward and backward, as flat 16-byte-vector kernels.
//
//   swiglu: out = silu(gate) * up          geglu: out = gelu_tanh(gate) * up       gelu: exact (erf)
// gate and up may be the two halves of one fused gate_up projection output (explicit row strides),
// and the backward writes d_gate and d_up side by side so a fused projection gets one dgrad GEMM.
// Counterparts: lset/kernels/swiglu.py:21-74, lset/kernels/geglu.py:22-86, aten GELU in
// lset/models/encoder/bert/model.py:107.
#include "../common/pdl.h"
#include "../common/row.cuh"

namespace lb {
namespace {

using bf16 = __nv_bfloat16;

enum { kSwiglu = 0, kGeglu = 1 };

__device__ __forceinline__ float sigmoidf_(float x) { return __frcp_rn(1.f + __expf(-x)); }

__device__ __forceinline__ float gelu_tanh_(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  return 0.5f * x * (1.f + tanhf(k0 * (x + k1 * x * x * x)));
}
__device__ __forceinline__ float gelu_tanh_grad_(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  const float t = tanhf(k0 * (x + k1 * x * x * x));
  return 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * k0 * (1.f + 3.f * k1 * x * x);
}

// A walk over the vectors of a [T, 8 * vec_per_row] matrix, grid * block apart. (A 64-bit division for
// every vector was a third of the forward's instructions.)
struct VecWalk {
  long long row, rows;
  int vec, d_vec, vec_per_row;
  long long d_row;
  __device__ VecWalk(long long T, int vpr) : rows(T), vec_per_row(vpr) {
    const long long first = 1LL * blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned stride = gridDim.x * blockDim.x;
    row = first / vpr;
    vec = int(first - row * vpr);
    d_row = stride / unsigned(vpr);
    d_vec = int(stride - unsigned(d_row) * unsigned(vpr));
  }
  __device__ bool more() const { return row < rows; }
  __device__ void step() {
    row += d_row;
    vec += d_vec;
    if (vec >= vec_per_row) {
      vec -= vec_per_row;
      ++row;
    }
  }
};

// Both directions are bound by memory, and close to the issue of instructions (78 % of the cycles before, at
// a clock that the GEMMs around them lower): an exponential and a reciprocal for each element, everything
// else two elements at a time. More threads hide more than more loads a thread do: 32 registers, eight CTAs a SM
// (two vectors a thread and half the threads: 490 us for the 418 / 391 below).
// Measured before / now (us, L2 flushed): 33280 x 12288 forward 418 / 391, backward 653 / 641; 22627 x 3072
// 80 / 78 and 117 / 114.
template <int KIND>
__device__ __forceinline__ uint4 glu_fwd8(const uint4& gq, const uint4& uq) {
  f2 g[4], u[4], o[4];
  unpack8(gq, g);
  unpack8(uq, u);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 x = f2_get(g[j]);
    const f2 a = KIND == kSwiglu ? f2_mul(g[j], f2_of(sigmoidf_(x.x), sigmoidf_(x.y)))
                                 : f2_of(gelu_tanh_(x.x), gelu_tanh_(x.y));
    o[j] = f2_mul(a, u[j]);
  }
  return pack8(o);
}

template <int KIND>
__global__ void __launch_bounds__(256, 8)
    glu_fwd_kernel(const bf16* __restrict__ gate, const bf16* __restrict__ up, long long ld_in,
                   bf16* __restrict__ out, long long ld_out, long long T, int I) {
  pdl_wait();
  pdl_trigger();
  for (VecWalk w(T, I / 8); w.more(); w.step()) {
    const int c = w.vec * 8;
    st16(out + w.row * ld_out + c,
         glu_fwd8<KIND>(ld16(gate + w.row * ld_in + c), ld16(up + w.row * ld_in + c)));
  }
}

template <int KIND>
__global__ void __launch_bounds__(256, 8)
    glu_bwd_kernel(const bf16* __restrict__ dout, long long ld_dout, const bf16* __restrict__ gate,
                   const bf16* __restrict__ up, long long ld_in, bf16* __restrict__ dgate,
                   bf16* __restrict__ dup, long long ld_d, long long T, int I) {
  pdl_wait();
  pdl_trigger();
  const f2 one = f2_of(1.f, 1.f), minus_one = f2_of(-1.f, -1.f);
  for (VecWalk w(T, I / 8); w.more(); w.step()) {
    const int c = w.vec * 8;
    f2 g[4], u[4], d[4], dg[4], du[4];
    unpack8(ld16(gate + w.row * ld_in + c), g);
    unpack8(ld16(up + w.row * ld_in + c), u);
    unpack8(ld16(dout + w.row * ld_dout + c), d);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 x = f2_get(g[j]);
      f2 act, dact;
      if (KIND == kSwiglu) {
        const f2 s = f2_of(sigmoidf_(x.x), sigmoidf_(x.y));
        act = f2_mul(g[j], s);
        dact = f2_mul(s, f2_fma(g[j], f2_fma(s, minus_one, one), one));
      } else {
        act = f2_of(gelu_tanh_(x.x), gelu_tanh_(x.y));
        dact = f2_of(gelu_tanh_grad_(x.x), gelu_tanh_grad_(x.y));
      }
      du[j] = f2_mul(d[j], act);
      dg[j] = f2_mul(f2_mul(d[j], u[j]), dact);
    }
    st16(dgate + w.row * ld_d + c, pack8(dg));
    st16(dup + w.row * ld_d + c, pack8(du));
  }
}

__global__ void __launch_bounds__(256)
    gelu_fwd_kernel(const bf16* __restrict__ x, bf16* __restrict__ y, long long n8) {
  pdl_wait();
  pdl_trigger();
  for (long long i = 1LL * blockIdx.x * blockDim.x + threadIdx.x; i < n8;
       i += 1LL * gridDim.x * blockDim.x) {
    float v[8];
    unpack8(ld16(x + i * 8), v);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = 0.5f * v[j] * (1.f + erff(v[j] * 0.7071067811865476f));
    st16(y + i * 8, pack8(v));
  }
}

__global__ void __launch_bounds__(256)
    gelu_bwd_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x, bf16* __restrict__ dx,
                    long long n8) {
  pdl_wait();
  pdl_trigger();
  for (long long i = 1LL * blockIdx.x * blockDim.x + threadIdx.x; i < n8;
       i += 1LL * gridDim.x * blockDim.x) {
    float v[8], g[8];
    unpack8(ld16(x + i * 8), v);
    unpack8(ld16(dy + i * 8), g);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float cdf = 0.5f * (1.f + erff(v[j] * 0.7071067811865476f));
      const float pdf = 0.3989422804014327f * __expf(-0.5f * v[j] * v[j]);
      g[j] *= cdf + v[j] * pdf;
    }
    st16(dx + i * 8, pack8(g));
  }
}

// x += y, in bf16.
__global__ void __launch_bounds__(256) add_bf16_kernel(bf16* x, const bf16* __restrict__ y, long long n8) {
  pdl_wait();
  pdl_trigger();
  for (long long i = 1LL * blockIdx.x * blockDim.x + threadIdx.x; i < n8;
       i += 1LL * gridDim.x * blockDim.x) {
    float a[8], b[8];
    unpack8(ld16(x + i * 8), a);
    unpack8(ld16(y + i * 8), b);
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] += b[j];
    st16(x + i * 8, pack8(a));
  }
}

// Column sums of dy [T, n0 + n1 + n2] added to up to three fp32 vectors: the bias gradients of
// linears that share an input. Bound by the read of dy. A CTA sums 64 columns (128 bytes of a row,
// eight lanes of 16) over a chunk of the rows, 32 rows at a time and DEPTH of those in flight; one
// chunk up to 4096 rows, more as the CTAs of a cluster, whose sums the first one adds up in their order:
// the result does not depend on timing.
// Measured at 700 rows (us): 768 columns 17.5 and 3072 columns 18.9 as a cast, a torch sum and two
// more passes each; 3.4 and 3.9 here. Four rows in flight / eight (some 14 us of each the measurement's
// own): 300 rows x 2304 16.2 / 20.0, 4096 x 3072 39.8 / 31.4, 40000 x 2304 64.0 / 54.6.
constexpr int kBiasCols = 64;

__device__ __forceinline__ void bias_cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float ld_cluster(const float* p, int rank) {
  uint32_t at;
  float v;
  asm("mapa.shared::cluster.u32 %0, %1, %2;"
      : "=r"(at)
      : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
  return v;
}

template <int DEPTH>
__global__ void __launch_bounds__(256)
    bias_grad_kernel(const bf16* __restrict__ dy, long long ld, int T, int n0, int n1, int n2,
                     float* g0, float* g1, float* g2) {
  __shared__ float part[32][kBiasCols + 1];
  __shared__ float total[kBiasCols];
  pdl_wait();
  pdl_trigger();
  const int cg = (threadIdx.x & 7) * 8, rl = threadIdx.x >> 3;
  const int col = blockIdx.y * kBiasCols + cg;
  const int N = n0 + n1 + n2;
  const int chunks = int(gridDim.x);
  const int chunk = (T + chunks - 1) / chunks;
  const int r0 = int(blockIdx.x) * chunk, r1 = min(T, r0 + chunk);
  float s[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) s[i] = 0.f;
  if (col < N) {
    for (int r = r0 + rl; r < r1; r += 32 * DEPTH) {
      uint4 q[DEPTH];
      const bf16* src = dy + r * ld + col;
      if (r + 32 * (DEPTH - 1) < r1) {   // (loads behind conditions of their own are not batched)
#pragma unroll
        for (int k = 0; k < DEPTH; ++k) q[k] = ld16(src + 32 * k * ld);
      } else {
#pragma unroll
        for (int k = 0; k < DEPTH; ++k)
          q[k] = r + 32 * k < r1 ? ld16(src + 32 * k * ld) : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int k = 0; k < DEPTH; ++k) {
        float f[8];
        unpack8(q[k], f);
#pragma unroll
        for (int i = 0; i < 8; ++i) s[i] += f[i];
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) part[rl][cg + i] = s[i];
  __syncthreads();
  float t = 0.f;
  if (threadIdx.x < kBiasCols) {
#pragma unroll
    for (int k = 0; k < 32; ++k) t += part[k][threadIdx.x];
    total[threadIdx.x] = t;
  }
  if (chunks > 1) bias_cluster_sync();
  if (blockIdx.x == 0 && threadIdx.x < kBiasCols) {
    for (int k = 1; k < chunks; ++k) t += ld_cluster(total + threadIdx.x, k);
    const int c = blockIdx.y * kBiasCols + threadIdx.x;
    if (c < N) {
      float* g = c < n0 ? g0 : (c < n0 + n1 ? g1 : g2);
      const int at = c < n0 ? c : (c < n0 + n1 ? c - n0 : c - n0 - n1);
      if (g != nullptr) g[at] += t;
    }
  }
  if (chunks > 1) bias_cluster_sync();   // nobody's sums go before they are read
}

int flat_grid(long long work_items, int per_sm = 16) {
  long long g = (work_items + 255) / 256;
  const long long cap = 1LL * row_num_sms() * per_sm;
  if (g > cap) g = cap;
  return int(g > 0 ? g : 1);
}

// CTAs of the gated kernels: with many vectors eight waves, whose ends overlap the next one's starts
// (22627 x 3072, forward / backward: 80 / 119 us with two waves, 78 / 114 with eight); with few, two
// (3000 x 3072: 23 us, 25 with a wave for every vector).
int glu_grid(long long vectors) {
  return flat_grid(vectors, vectors > 64LL * 256 * row_num_sms() ? 64 : 16);
}

}  // namespace
}  // namespace lb

using namespace lb;

// kind: 0 = SwiGLU, 1 = GeGLU (tanh). gate/up rows are ld_in apart; I must be a multiple of 8.
extern "C" int lb_glu_fwd(int kind, const void* gate, const void* up, long long ld_in, void* out,
                          long long ld_out, long long T, int I, void* stream) {
  if (T <= 0 || I <= 0) return 0;
  if ((I & 7) || (ld_in & 7) || (ld_out & 7)) return -3;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  return launch_pdl(kind == kSwiglu ? glu_fwd_kernel<kSwiglu> : glu_fwd_kernel<kGeglu>,
                    dim3(glu_grid(T * (I / 8))), dim3(256), 0, st, pdl_enabled(6 * T * I), 1,
                    (const bf16*)gate, (const bf16*)up, ld_in, (bf16*)out, ld_out, T, I);
}

extern "C" int lb_glu_bwd(int kind, const void* dout, long long ld_dout, const void* gate,
                          const void* up, long long ld_in, void* dgate, void* dup, long long ld_d,
                          long long T, int I, void* stream) {
  if (T <= 0 || I <= 0) return 0;
  if ((I & 7) || (ld_in & 7) || (ld_dout & 7) || (ld_d & 7)) return -3;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  return launch_pdl(kind == kSwiglu ? glu_bwd_kernel<kSwiglu> : glu_bwd_kernel<kGeglu>,
                    dim3(glu_grid(T * (I / 8))), dim3(256), 0, st, pdl_enabled(10 * T * I), 1,
                    (const bf16*)dout, ld_dout, (const bf16*)gate, (const bf16*)up, ld_in,
                    (bf16*)dgate, (bf16*)dup, ld_d, T, I);
}

extern "C" int lb_gelu_fwd(const void* x, void* y, long long n, void* stream) {
  if (n <= 0) return 0;
  if (n & 7) return -3;
  return launch_pdl(gelu_fwd_kernel, dim3(flat_grid(n / 8)), dim3(256), 0,
                    reinterpret_cast<cudaStream_t>(stream), pdl_enabled(4 * n), 1, (const bf16*)x,
                    (bf16*)y, n / 8);
}

extern "C" int lb_gelu_bwd(const void* dy, const void* x, void* dx, long long n, void* stream) {
  if (n <= 0) return 0;
  if (n & 7) return -3;
  return launch_pdl(gelu_bwd_kernel, dim3(flat_grid(n / 8)), dim3(256), 0,
                    reinterpret_cast<cudaStream_t>(stream), pdl_enabled(6 * n), 1, (const bf16*)dy,
                    (const bf16*)x, (bf16*)dx, n / 8);
}

extern "C" int lb_add_bf16(void* x, const void* y, long long n, void* stream) {
  if (n <= 0) return 0;
  if (n & 7) return -3;
  return launch_pdl(add_bf16_kernel, dim3(flat_grid(n / 8)), dim3(256), 0,
                    reinterpret_cast<cudaStream_t>(stream), pdl_enabled(6 * n), 1, (bf16*)x,
                    (const bf16*)y, n / 8);
}

// dy: [T, n0 + n1 + n2] bf16, rows ld apart; g0, g1, g2 (null: skipped) += its column sums.
extern "C" int lb_bias_grad(const void* dy, long long ld, int T, int n0, int n1, int n2, float* g0,
                            float* g1, float* g2, void* stream) {
  const int N = n0 + n1 + n2;
  if (T <= 0 || N <= 0) return 0;
  if ((ld & 7) || (n0 & 7) || (n1 & 7) || (n2 & 7)) return -3;
  const int chunks = T <= 4096 ? 1 : (T / 2048 < 8 ? T / 2048 : 8);   // of a cluster, one of 8 at most
  return launch_pdl(T / chunks >= 1024 ? bias_grad_kernel<8> : bias_grad_kernel<4>,
                    dim3(chunks, (N + kBiasCols - 1) / kBiasCols), dim3(256), 0,
                    reinterpret_cast<cudaStream_t>(stream), pdl_enabled(2LL * T * N), chunks, (const bf16*)dy, ld,
                    T, n0, n1, n2, g0, g1, g2);
}
