// RMSNorm and LayerNorm, forward and backward, each with an optional fused residual add.
//
//   rms  : nr = bf16(r + a) (when a residual is given);  rstd = rsqrt(mean(nr^2) + eps);
//          y = bf16(nr * rstd) * (w + w_off)          (w_off = 1 for Gemma's "(1 + w)" weights)
//   ln   : same with mean subtraction and a bias.
// The normalised value is rounded to bf16 before the weight multiply, and the weight gradient
// accumulates dy * bf16(xhat) in fp32: the rounding points of the reference kernels
// (lset/kernels/rmsnorm.py:68-73,99-114; lset/kernels/residual_rmsnorm.py:58-77;
// lset/kernels/layernorm.py:73-77; lset/kernels/residual_layernorm.py:46-139).
//
// Backward runs on a persistent grid; every CTA writes one fp32 partial row of dW (and dB) to a
// caller-provided scratch buffer, and a second small kernel sums the partials.
#include "../common/api.h"
#include "../common/pdl.h"
#include "../common/row.cuh"

namespace lb {
namespace {

using bf16 = __nv_bfloat16;

// Eight weights of a slice that does not start at a 16-byte boundary.
__device__ __forceinline__ uint4 ld8_unaligned(const bf16* p) {
  float f[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) f[i] = __bfloat162float(p[i]);
  return pack8(f);
}

template <int TPR, int NV, bool W_ALIGNED>
__global__ void __launch_bounds__(kRowThreads)
    rms_fwd_kernel(const bf16* __restrict__ x, const bf16* __restrict__ res_in,
                   const bf16* __restrict__ w, bf16* __restrict__ y, bf16* __restrict__ res_out,
                   float* __restrict__ rstd_out, int N, int H, float eps, float w_off) {
  __shared__ float sred[8];
  constexpr int ROWS = kRowThreads / TPR;
  const int t = threadIdx.x % TPR;
  const int r = threadIdx.x / TPR;
  const long long row = 1LL * blockIdx.x * ROWS + r;
  const bool valid = row < N;
  // Every load of the row is requested before the first is used, the weights (in L1 / L2 after the
  // first rows) among them; the row stays packed in between, so that more CTAs fit per SM.
  uint4 xq[NV], rq[NV], wq[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int idx = (v * TPR + t) * 8;
    if (valid && idx < H) wq[v] = W_ALIGNED ? ld16(w + idx) : ld8_unaligned(w + idx);
  }
  pdl_wait();
  pdl_trigger();
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int idx = (v * TPR + t) * 8;
    if (valid && idx < H) {
      xq[v] = ld16(x + row * H + idx);
      if (res_in != nullptr) rq[v] = ld16(res_in + row * H + idx);
    }
  }
  float ss = 0.f;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int idx = (v * TPR + t) * 8;
    if (valid && idx < H) {
      float f[8];
      unpack8(xq[v], f);
      if (res_in != nullptr) {
        float rv[8];
        unpack8(rq[v], rv);
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] += rv[i];
        xq[v] = pack8(f);
        unpack8(xq[v], f);
        st16(res_out + row * H + idx, xq[v]);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) ss += f[i] * f[i];
    }
  }
  ss = row_sum<TPR>(ss, sred);
  const float rstd = rsqrtf(ss / float(H) + eps);
  if (valid && t == 0 && rstd_out != nullptr) rstd_out[row] = rstd;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int idx = (v * TPR + t) * 8;
    if (valid && idx < H) {
      float f[8], wl[8];
      unpack8(xq[v], f);
      unpack8(wq[v], wl);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = bf16_round(f[i] * rstd) * (wl[i] + w_off);
      st16(y + row * H + idx, pack8(f));
    }
  }
}

// Gemma's post-norm pair in one pass: z = bf16(bf16(a·rstd1)·w1); nr = bf16(residual + z);
// y = bf16(nr·rstd2)·w2. The row stays in registers between the two norms; a, rstd1, nr and rstd2
// are what the two backward launches need.
template <int TPR, int NV>
__global__ void __launch_bounds__(kRowThreads)
    rms_double_fwd_kernel(const bf16* __restrict__ a, const bf16* __restrict__ res_in,
                          const bf16* __restrict__ w1, const bf16* __restrict__ w2,
                          bf16* __restrict__ y, bf16* __restrict__ res_out,
                          float* __restrict__ rstd1_out, float* __restrict__ rstd2_out, int N, int H,
                          float eps, float w_off) {
  __shared__ float sred[8];
  extern __shared__ float sw[];  // [H] first weights, [H] second weights (+ offset)
  const int t = threadIdx.x % TPR;
  const int r = threadIdx.x / TPR;
  constexpr int ROWS = kRowThreads / TPR;
  for (int i = threadIdx.x; i < H; i += kRowThreads) {
    sw[i] = __bfloat162float(w1[i]) + w_off;
    sw[H + i] = __bfloat162float(w2[i]) + w_off;
  }
  __syncthreads();
  for (long long row0 = 1LL * blockIdx.x * ROWS; row0 < N; row0 += 1LL * gridDim.x * ROWS) {
    const long long row = row0 + r;
    const bool valid = row < N;
    float xv[NV][8];
    uint4 rq[NV];
    float ss = 0.f;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int idx = (v * TPR + t) * 8;
      if (valid && idx < H) {
        unpack8(ld16(a + row * H + idx), xv[v]);
        rq[v] = ld16(res_in + row * H + idx);
#pragma unroll
        for (int i = 0; i < 8; ++i) ss += xv[v][i] * xv[v][i];
      }
    }
    ss = row_sum<TPR>(ss, sred);
    const float rstd1 = rsqrtf(ss / float(H) + eps);
    float ss2 = 0.f;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int idx = (v * TPR + t) * 8;
      if (valid && idx < H) {
        float rv[8];
        unpack8(rq[v], rv);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float z = bf16_round(bf16_round(xv[v][i] * rstd1) * sw[idx + i]);
          xv[v][i] = bf16_round(rv[i] + z);
          ss2 += xv[v][i] * xv[v][i];
        }
        st16(res_out + row * H + idx, pack8(xv[v]));
      }
    }
    ss2 = row_sum<TPR>(ss2, sred);
    const float rstd2 = rsqrtf(ss2 / float(H) + eps);
    if (valid && t == 0) {
      rstd1_out[row] = rstd1;
      rstd2_out[row] = rstd2;
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int idx = (v * TPR + t) * 8;
      if (valid && idx < H) {
        float o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = bf16_round(xv[v][i] * rstd2) * sw[H + idx + i];
        st16(y + row * H + idx, pack8(o));
      }
    }
  }
}

// Sum over the TPR threads of a row, one barrier a call among those threads only: `sred` alternates between
// two slots from call to call. The values and the order of row_sum.
template <int TPR>
__device__ __forceinline__ float row_sum_alt(float v, float (&sred)[2][8], int slot) {
#pragma unroll
  for (int o = (TPR < 32 ? TPR : 32) / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if constexpr (TPR > 32) {
    const int warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) sred[slot][warp] = v;
    asm volatile("bar.sync %0, %1;" ::"r"(1 + int(threadIdx.x) / TPR), "n"(TPR) : "memory");
    constexpr int W = TPR / 32;
    const int w0 = (warp / W) * W;
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < W; ++i) t += sred[slot][w0 + i];
    v = t;
  }
  return v;
}

// Bound by memory where enough rows are in flight. x and dy stay packed in registers (unpacked twice) and
// the weights in shared memory, so that only the dW accumulators live as long as the CTA: three CTAs a SM (two
// above 4096 columns). Four columns of a thread are next to its neighbour's in shared memory (eight in
// a row cost every access twice its banks); two columns an instruction; one barrier a row.
// Measured before / now (us, L2 flushed): 22627 x 1024 53 / 49, 40280 x 1024 76 / 72, 33280 x 4096 201 / 197,
// 21000 x 2560 107 / 105, 5000 x 8192 104 / 92. (A warp a row, with no barrier, needs twice the
// registers: 59 at 22627 x 1024.) One wave of four CTAs a SM, which 64 registers allow, takes 45, 68, 179, 92 and
// 84, but cuts the sums of dW into other partial rows: the gradient norm then has other last bits, and every
// weight of a clipped step.
template <int TPR, int NV>
constexpr int rms_bwd_smem(int H) { return (H + 8 * TPR * NV) * int(sizeof(float)); }

template <int TPR, int NV>
__global__ void __launch_bounds__(kRowThreads, NV > 2 ? 2 : 3)
    rms_bwd_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ dres,
                   const bf16* __restrict__ xin, const bf16* __restrict__ w,
                   const float* __restrict__ rstd_in, bf16* __restrict__ dx,
                   float* __restrict__ dw_partial, int N, int H, float w_off) {
  __shared__ float sred[2][8];
  extern __shared__ float sdw[];  // [H] dW accumulator of the CTA, then [2 NV][TPR][4] weights
  float* sw = sdw + H;
  constexpr int ROWS = kRowThreads / TPR;
  const int t = threadIdx.x % TPR;
  const int r = threadIdx.x / TPR;
  f2 dwacc[NV][4];
#pragma unroll
  for (int v = 0; v < NV; ++v)
#pragma unroll
    for (int i = 0; i < 4; ++i) dwacc[v][i] = 0ull;
  for (int i = threadIdx.x; i < H; i += kRowThreads) {
    const int col = i % 8, at = i / 8;   // column `col` of thread at % TPR in vector at / TPR
    sdw[i] = 0.f;
    sw[((at / TPR * 2 + col / 4) * TPR + at % TPR) * 4 + col % 4] = __bfloat162float(w[i]) + w_off;
  }
  __syncthreads();
  pdl_wait();
  pdl_trigger();

  auto load_w = [&](int v, f2 (&wl)[4]) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const float4 q = *reinterpret_cast<const float4*>(sw + ((v * 2 + k) * TPR + t) * 4);
      wl[2 * k] = f2_of(q.x, q.y);
      wl[2 * k + 1] = f2_of(q.z, q.w);
    }
  };
  int slot = 0;
  for (long long row0 = 1LL * blockIdx.x * ROWS; row0 < N; row0 += 1LL * gridDim.x * ROWS) {
    const long long row = row0 + r;
    const bool valid = row < N;
    const float rstd = valid ? rstd_in[row] : 0.f;
    const f2 rstd2 = f2_of(rstd, rstd);
    uint4 xq[NV], gq[NV], rq[NV];
    float dot = 0.f;
    // every load of the row is requested before the first use
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int idx = (v * TPR + t) * 8;
      if (valid && idx < H) {
        xq[v] = ld16(xin + row * H + idx);
        gq[v] = ld16(dy + row * H + idx);
        if (dres != nullptr) rq[v] = ld16(dres + row * H + idx);
      }
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int idx = (v * TPR + t) * 8;
      if (valid && idx < H) {
        f2 g[4], xh[4];
        unpack8(xq[v], xh);
        unpack8(gq[v], g);
        f2 wl[4];
        load_w(v, wl);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          xh[i] = f2_mul(xh[i], rstd2);
          const float2 a = f2_get(f2_mul(g[i], wl[i])), b = f2_get(xh[i]);
          dot = fmaf(a.x, b.x, dot);
          dot = fmaf(a.y, b.y, dot);
          dwacc[v][i] = f2_fma(g[i], f2_bf16_round(xh[i]), dwacc[v][i]);
        }
      }
    }
    dot = row_sum_alt<TPR>(dot, sred, slot) / float(H);
    slot ^= 1;
    const f2 minus_dot = f2_of(-dot, -dot);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int idx = (v * TPR + t) * 8;
      if (valid && idx < H) {
        f2 g[4], o[4], wl[4];
        load_w(v, wl);
        unpack8(gq[v], g);
        unpack8(xq[v], o);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          o[i] = f2_mul(rstd2, f2_fma(g[i], wl[i], f2_mul(f2_mul(o[i], rstd2), minus_dot)));
        if (dres != nullptr) {
          f2 dr[4];
          unpack8(rq[v], dr);
#pragma unroll
          for (int i = 0; i < 4; ++i) o[i] = f2_add(o[i], dr[i]);
        }
        st16(dx + row * H + idx, pack8(o));
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int idx = (v * TPR + t) * 8;
    if (idx < H) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 a = f2_get(dwacc[v][i]);
        atomicAdd(&sdw[idx + 2 * i], a.x);
        atomicAdd(&sdw[idx + 2 * i + 1], a.y);
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < H; i += kRowThreads) dw_partial[1LL * blockIdx.x * H + i] = sdw[i];
}

template <int TPR, int NV>
__global__ void __launch_bounds__(kRowThreads)
    ln_fwd_kernel(const bf16* __restrict__ x, const bf16* __restrict__ res_in,
                  const bf16* __restrict__ w, const bf16* __restrict__ b, bf16* __restrict__ y,
                  bf16* __restrict__ res_out, float* __restrict__ mean_out,
                  float* __restrict__ rstd_out, int N, int H, float eps) {
  __shared__ float sred[8];
  constexpr int ROWS = kRowThreads / TPR;
  const int t = threadIdx.x % TPR;
  const int r = threadIdx.x / TPR;
  float wv[NV][8], bv[NV][8];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int idx = (v * TPR + t) * 8;
    if (idx < H) {
      unpack8(ld16(w + idx), wv[v]);
      if (b != nullptr) {
        unpack8(ld16(b + idx), bv[v]);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) bv[v][i] = 0.f;
      }
    }
  }
  pdl_wait();
  pdl_trigger();
  for (long long row0 = 1LL * blockIdx.x * ROWS; row0 < N; row0 += 1LL * gridDim.x * ROWS) {
    const long long row = row0 + r;
    const bool valid = row < N;
    float xv[NV][8];
    float s = 0.f;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int idx = (v * TPR + t) * 8;
      if (valid && idx < H) {
        unpack8(ld16(x + row * H + idx), xv[v]);
        if (res_in != nullptr) {
          float rv[8];
          unpack8(ld16(res_in + row * H + idx), rv);
#pragma unroll
          for (int i = 0; i < 8; ++i) xv[v][i] = bf16_round(xv[v][i] + rv[i]);
          st16(res_out + row * H + idx, pack8(xv[v]));
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) s += xv[v][i];
      }
    }
    const float mean = row_sum<TPR>(s, sred) / float(H);
    float ss = 0.f;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int idx = (v * TPR + t) * 8;
      if (valid && idx < H) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float d = xv[v][i] - mean;
          ss += d * d;
        }
      }
    }
    const float rstd = rsqrtf(row_sum<TPR>(ss, sred) / float(H) + eps);
    if (valid && t == 0) {
      if (mean_out != nullptr) mean_out[row] = mean;
      if (rstd_out != nullptr) rstd_out[row] = rstd;
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int idx = (v * TPR + t) * 8;
      if (valid && idx < H) {
        float o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
          o[i] = bf16_round((xv[v][i] - mean) * rstd) * wv[v][i] + bv[v][i];
        st16(y + row * H + idx, pack8(o));
      }
    }
  }
}

template <int TPR, int NV>
__global__ void __launch_bounds__(kRowThreads)
    ln_bwd_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ dres,
                  const bf16* __restrict__ xin, const bf16* __restrict__ w,
                  const float* __restrict__ mean_in, const float* __restrict__ rstd_in,
                  bf16* __restrict__ dx, float* __restrict__ dwb_partial, int N, int H) {
  __shared__ float sred[8];
  extern __shared__ float sdw[];  // [2, H]: dW then dB
  constexpr int ROWS = kRowThreads / TPR;
  const int t = threadIdx.x % TPR;
  const int r = threadIdx.x / TPR;
  float wv[NV][8], dwacc[NV][8], dbacc[NV][8];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int idx = (v * TPR + t) * 8;
#pragma unroll
    for (int i = 0; i < 8; ++i) dwacc[v][i] = dbacc[v][i] = 0.f;
    if (idx < H) unpack8(ld16(w + idx), wv[v]);
  }
  for (int i = threadIdx.x; i < 2 * H; i += kRowThreads) sdw[i] = 0.f;
  pdl_wait();
  pdl_trigger();

  for (long long row0 = 1LL * blockIdx.x * ROWS; row0 < N; row0 += 1LL * gridDim.x * ROWS) {
    const long long row = row0 + r;
    const bool valid = row < N;
    const float rstd = valid ? rstd_in[row] : 0.f;
    const float mean = valid ? mean_in[row] : 0.f;
    float xh[NV][8], m[NV][8];
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int idx = (v * TPR + t) * 8;
      if (valid && idx < H) {
        float g[8];
        unpack8(ld16(xin + row * H + idx), xh[v]);
        unpack8(ld16(dy + row * H + idx), g);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          xh[v][i] = (xh[v][i] - mean) * rstd;
          m[v][i] = g[i] * wv[v][i];
          s1 += m[v][i];
          s2 += m[v][i] * xh[v][i];
          dwacc[v][i] += g[i] * bf16_round(xh[v][i]);
          dbacc[v][i] += g[i];
        }
      }
    }
    s1 = row_sum<TPR>(s1, sred) / float(H);
    s2 = row_sum<TPR>(s2, sred) / float(H);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int idx = (v * TPR + t) * 8;
      if (valid && idx < H) {
        float o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = rstd * (m[v][i] - s1 - xh[v][i] * s2);
        if (dres != nullptr) {
          float dr[8];
          unpack8(ld16(dres + row * H + idx), dr);
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] += dr[i];
        }
        st16(dx + row * H + idx, pack8(o));
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int idx = (v * TPR + t) * 8;
    if (idx < H) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        atomicAdd(&sdw[idx + i], dwacc[v][i]);
        atomicAdd(&sdw[H + idx + i], dbacc[v][i]);
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * H; i += kRowThreads)
    dwb_partial[1LL * blockIdx.x * 2 * H + i] = sdw[i];
}

// out[c] (+)= sum_p partial[p, c]. A CTA owns 32 columns; its 32 warps each sum a slice of the
// partial rows (coalesced 128-byte reads), then the slices are combined in shared memory. Several sums of
// one block's backward are one launch.
struct ColsumJobs {
  LbColsum job[kMaxColsums];
  int first[kMaxColsums + 1];   // CTAs
};

__global__ void __launch_bounds__(1024) colsum_kernel(ColsumJobs jobs, int out_fp32, int accumulate) {
  __shared__ float sm[32][33];
  int j = 0;
  while (j + 1 < kMaxColsums && int(blockIdx.x) >= jobs.first[j + 1]) ++j;
  const LbColsum& job = jobs.job[j];
  const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5;
  const int c = (int(blockIdx.x) - jobs.first[j]) * 32 + lane;
  const int P = job.rows, C = job.cols;
  const float* partial = job.partial;
  float s = 0.f;
  pdl_wait();
  pdl_trigger();
  if (c < C)
    for (int p = grp; p < P; p += 32) s += partial[1LL * p * C + c];
  sm[grp][lane] = s;
  __syncthreads();
  if (grp == 0 && c < C) {
    float tot = 0.f;
#pragma unroll
    for (int g2 = 0; g2 < 32; ++g2) tot += sm[g2][lane];
    const bool upper = job.split > 0 && c >= job.split;
    void* out = upper ? job.out2 : job.out;
    const int at = upper ? c - job.split : c;
    if (out == nullptr) return;
    if (out_fp32) {
      float* o = reinterpret_cast<float*>(out);
      o[at] = accumulate ? o[at] + tot : tot;
    } else {
      bf16* o = reinterpret_cast<bf16*>(out);
      o[at] = __float2bfloat16_rn(accumulate ? __bfloat162float(o[at]) + tot : tot);
    }
  }
}

int launch_colsums(const LbColsum* jobs, int n, int out_fp32, int accumulate, cudaStream_t st) {
  ColsumJobs a = {};
  int ctas = 0, k = 0;
  for (int i = 0; i < n; ++i) {
    if (jobs[i].cols <= 0) continue;
    a.job[k] = jobs[i];
    a.first[k++] = ctas;
    ctas += (jobs[i].cols + 31) / 32;
  }
  for (; k <= kMaxColsums; ++k) a.first[k] = ctas;
  if (ctas == 0) return 0;
  return launch_pdl(colsum_kernel, dim3(ctas), dim3(1024), 0, st, pdl_enabled(), 1, a, out_fp32,
                    accumulate);
}

int launch_colsum(const float* partial, int P, int C, void* out, int out_fp32, int accumulate,
                  cudaStream_t st) {
  const LbColsum job = {partial, P, C, out, nullptr, 0};
  return launch_colsums(&job, 1, out_fp32, accumulate, st);
}

// CTAs of the backward kernels for each SM, and so the partial rows that their weight gradients are cut into: part of
// the bits of a training step.
constexpr int kBwdPerSm = 6;

int bwd_grid(int N, int rows_per_cta) {
  const int need = (N + rows_per_cta - 1) / rows_per_cta;
  const int cap = row_num_sms() * kBwdPerSm;
  return need < cap ? (need > 0 ? need : 1) : cap;
}

}  // namespace
}  // namespace lb

using namespace lb;

// Number of fp32 partial rows that the backward kernels may write (scratch = rows * H floats for
// RMSNorm, rows * 2H for LayerNorm).
extern "C" int lb_norm_bwd_partial_rows() { return row_num_sms() * 8; }

extern "C" int lb_rms_norm_fwd(const void* x, const void* res_in, const void* w, void* y,
                               void* res_out, float* rstd, int N, int H, float eps, float w_off,
                               void* stream) {
  if (N <= 0) return 0;
  if (H & 7) return -3;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  LB_ROW_DISPATCH(H, {
    constexpr int ROWS = kRowThreads / TPR;
    const int grid = (N + ROWS - 1) / ROWS;
    const bool aligned = (reinterpret_cast<uintptr_t>(w) & 15u) == 0;
    return launch_pdl(aligned ? rms_fwd_kernel<TPR, NV, true> : rms_fwd_kernel<TPR, NV, false>,
                      dim3(grid), dim3(kRowThreads), 0, st, pdl_enabled((res_in != nullptr ? 8LL : 4LL) * N * H), 1, (const bf16*)x,
                      (const bf16*)res_in, (const bf16*)w, (bf16*)y, (bf16*)res_out, rstd, N, H, eps,
                      w_off);
  });
}

// Fused forward of rmsnorm(a)·w1 → + residual → rmsnorm(·)·w2. Outputs y, res_out (the new
// residual stream), rstd1 (of a) and rstd2 (of res_out).
extern "C" int lb_rms_norm_double_fwd(const void* a, const void* res_in, const void* w1,
                                      const void* w2, void* y, void* res_out, float* rstd1,
                                      float* rstd2, int N, int H, float eps, float w_off,
                                      void* stream) {
  if (N <= 0) return 0;
  if ((H & 7) || 2 * H * sizeof(float) > 48 * 1024) return -3;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  LB_ROW_DISPATCH(H, {
    constexpr int ROWS = kRowThreads / TPR;
    const int grid = (N + ROWS - 1) / ROWS;
    rms_double_fwd_kernel<TPR, NV><<<grid, kRowThreads, 2 * H * sizeof(float), st>>>(
        (const bf16*)a, (const bf16*)res_in, (const bf16*)w1, (const bf16*)w2, (bf16*)y,
        (bf16*)res_out, rstd1, rstd2, N, H, eps, w_off);
  });
  return launch_rc();
}

// dw_out: [H] fp32 or bf16; scratch: lb_norm_bwd_partial_rows() * H floats.
extern "C" int lb_rms_norm_bwd(const void* dy, const void* dres, const void* xin, const void* w,
                               const float* rstd, void* dx, float* scratch, void* dw_out,
                               int dw_fp32, int dw_accumulate, int N, int H, float w_off,
                               void* stream) {
  if (N <= 0) return 0;
  if (H & 7) return -3;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  int grid = 1;
  LB_ROW_DISPATCH_NARROW(H, {
    constexpr int ROWS = kRowThreads / TPR;
    grid = bwd_grid(N, ROWS);
    constexpr auto smem = rms_bwd_smem<TPR, NV>;
    if (smem(H) > 48 * 1024)  // wide rows: opt in above the 48 KB default
      cudaFuncSetAttribute(rms_bwd_kernel<TPR, NV>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           smem(8 * TPR * NV));
    const int rc = launch_pdl(rms_bwd_kernel<TPR, NV>, dim3(grid), dim3(kRowThreads), smem(H), st,
                              pdl_enabled((dres != nullptr ? 8LL : 6LL) * N * H), 1, (const bf16*)dy,
                              (const bf16*)dres, (const bf16*)xin, (const bf16*)w, rstd, (bf16*)dx,
                              scratch, N, H, w_off);
    if (rc) return rc;
  });
  if (dw_out != nullptr)
    return launch_colsum(scratch, grid, H, dw_out, dw_fp32, dw_accumulate, st);
  return launch_rc();
}

// Partial rows that either norm's backward leaves in its scratch for N rows of width H.
extern "C" int lb_norm_bwd_rows(int N, int H) {
  if (N <= 0 || H <= 0) return 0;
  LB_ROW_DISPATCH_NARROW(H, { return bwd_grid(N, kRowThreads / TPR); });
  return 0;
}

extern "C" int lb_layer_norm_fwd(const void* x, const void* res_in, const void* w, const void* b,
                                 void* y, void* res_out, float* mean, float* rstd, int N, int H,
                                 float eps, void* stream) {
  if (N <= 0) return 0;
  if (H & 7) return -3;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  LB_ROW_DISPATCH(H, {
    constexpr int ROWS = kRowThreads / TPR;
    const int grid = (N + ROWS - 1) / ROWS;
    return launch_pdl(ln_fwd_kernel<TPR, NV>, dim3(grid), dim3(kRowThreads), 0, st, pdl_enabled((res_in != nullptr ? 8LL : 4LL) * N * H),
                      1, (const bf16*)x, (const bf16*)res_in, (const bf16*)w, (const bf16*)b,
                      (bf16*)y, (bf16*)res_out, mean, rstd, N, H, eps);
  });
}

// dwb_out: [2, H] (dW then dB), fp32 or bf16; scratch: lb_norm_bwd_partial_rows() * 2H floats.
extern "C" int lb_layer_norm_bwd(const void* dy, const void* dres, const void* xin, const void* w,
                                 const float* mean, const float* rstd, void* dx, float* scratch,
                                 void* dwb_out, int dw_fp32, int dw_accumulate, int N, int H,
                                 void* stream) {
  if (N <= 0) return 0;
  if (H & 7) return -3;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  int grid = 1;
  LB_ROW_DISPATCH_NARROW(H, {
    constexpr int ROWS = kRowThreads / TPR;
    grid = bwd_grid(N, ROWS);
    if (2 * H * sizeof(float) > 48 * 1024)
      cudaFuncSetAttribute(ln_bwd_kernel<TPR, NV>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           2 * H * (int)sizeof(float));
    const int rc = launch_pdl(ln_bwd_kernel<TPR, NV>, dim3(grid), dim3(kRowThreads), 2 * H * sizeof(float),
                              st, pdl_enabled((dres != nullptr ? 8LL : 6LL) * N * H), 1, (const bf16*)dy,
                              (const bf16*)dres, (const bf16*)xin, (const bf16*)w, mean, rstd, (bf16*)dx,
                              scratch, N, H);
    if (rc) return rc;
  });
  if (dwb_out != nullptr)
    return launch_colsum(scratch, grid, 2 * H, dwb_out, dw_fp32, dw_accumulate, st);
  return launch_rc();
}

extern "C" int lb_colsum(const float* partial, int P, int C, void* out, int out_fp32,
                         int accumulate, void* stream) {
  if (C <= 0) return 0;
  return launch_colsum(partial, P, C, out, out_fp32, accumulate, reinterpret_cast<cudaStream_t>(stream));
}

// How many of the n sums from the first on may run side by side: none of them adds to another's output.
static int colsum_batch(const LbColsum* jobs, int n) {
  int k = 0;
  for (; k < n && k < kMaxColsums; ++k)
    for (int j = 0; j < k; ++j)
      for (const void* a : {jobs[k].out, jobs[k].out2})
        if (a != nullptr && (a == jobs[j].out || a == jobs[j].out2)) return k;
  return k;
}

// Up to kMaxColsums sums of fp32 partial rows, added to fp32 outputs. They are one launch as long as each has
// outputs of its own: a weight that two norms share is added to by one launch after the other.
extern "C" int lb_colsums(const LbColsum* jobs, int n, void* stream) {
  if (n < 0 || n > kMaxColsums) return -3;
  LbColsum each[2 * kMaxColsums];
  int k = 0;
  for (int i = 0; i < n; ++i) {
    each[k++] = jobs[i];
    if (jobs[i].split > 0 && jobs[i].out != nullptr && jobs[i].out == jobs[i].out2) {
      each[k - 1].out2 = nullptr;
      each[k] = jobs[i];
      each[k++].out = nullptr;
    }
  }
  for (int from = 0; from < k;) {
    const int count = colsum_batch(each + from, k - from);
    if (int rc = launch_colsums(each + from, count, 1, 1, reinterpret_cast<cudaStream_t>(stream))) return rc;
    from += count;
  }
  return 0;
}

// ------------------------------------------------------------------------------------------------
// Allocation-free RMSNorm backward (see norm_noalloc.h): same kernels as lb_rms_norm_bwd, with the
// per-CTA partials in a fixed array that is part of the library image.
// ------------------------------------------------------------------------------------------------
#include <mutex>

#include "norm_noalloc.h"

namespace {

// One copy per device that loads the library. In host code this name is only a handle for
// cudaGetSymbolAddress; the kernels receive the looked-up device address.
static __device__ __align__(256) float g_noalloc_partials[LB_NOALLOC_MAX_PARTIAL_ROWS * LB_NOALLOC_MAX_H];

constexpr int kNoAllocMaxDevices = 64;
float* g_noalloc_ptr[kNoAllocMaxDevices] = {};
std::mutex g_noalloc_mutex;

// Device address of the array on the current device; looked up once per device.
int noalloc_scratch(float** out) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNoAllocMaxDevices)
    return LB_NOALLOC_ERR_DEVICE;
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (g_noalloc_ptr[dev] == nullptr) {
    float* p = nullptr;
    if (cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_noalloc_partials) != cudaSuccess ||
        p == nullptr) {
      cudaGetLastError();  // clear the sticky-free error state for the caller
      return LB_NOALLOC_ERR_SYMBOL;
    }
    g_noalloc_ptr[dev] = p;
  }
  *out = g_noalloc_ptr[dev];
  return 0;
}

}  // namespace

extern "C" const char* lb_noalloc_strerror(int code) {
  switch (code) {
    case 0: return "ok";
    case LB_NOALLOC_ERR_TOO_LARGE:
      return "row width H exceeds LB_NOALLOC_MAX_H (4096): the built-in scratch array is too small";
    case LB_NOALLOC_ERR_SYMBOL:
      return "cudaGetSymbolAddress failed for the built-in scratch array on the current device";
    case LB_NOALLOC_ERR_DEVICE: return "current device index is outside the library's device table";
    case -3: return "bad shape: H must be a positive multiple of 8";
    case -11: return "kernel launch failed";
    default: return "unknown error";
  }
}

extern "C" int lb_rms_norm_bwd_noalloc(const void* dy, const void* dres, const void* xin,
                                       const void* w, const float* rstd, void* dx, void* dw_out,
                                       int dw_fp32, int dw_accumulate, int N, int H, float w_off,
                                       void* stream) {
  if (N <= 0) return 0;
  if (H <= 0 || (H & 7)) return -3;
  if (H > LB_NOALLOC_MAX_H) return LB_NOALLOC_ERR_TOO_LARGE;
  float* scratch = nullptr;
  if (int rc = noalloc_scratch(&scratch)) return rc;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  int grid = 1;
  LB_ROW_DISPATCH_NARROW(H, {
    constexpr int ROWS = kRowThreads / TPR;
    grid = bwd_grid(N, ROWS);
    if (grid > LB_NOALLOC_MAX_PARTIAL_ROWS) grid = LB_NOALLOC_MAX_PARTIAL_ROWS;
    constexpr auto smem = rms_bwd_smem<TPR, NV>;
    if (smem(H) > 48 * 1024)  // wide rows: opt in above the 48 KB default
      cudaFuncSetAttribute(rms_bwd_kernel<TPR, NV>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           smem(8 * TPR * NV));
    rms_bwd_kernel<TPR, NV><<<grid, kRowThreads, smem(H), st>>>(
        (const bf16*)dy, (const bf16*)dres, (const bf16*)xin, (const bf16*)w, rstd, (bf16*)dx,
        scratch, N, H, w_off);
  });
  if (dw_out != nullptr)
    return launch_colsum(scratch, grid, H, dw_out, dw_fp32, dw_accumulate, st);
  return launch_rc();
}
