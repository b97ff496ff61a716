// Per-head RMSNorm fused with rotary position embedding for Q and K, forward and backward, plus
// the rope-only variant (do_norm = 0). One launch handles every (token, head) of both Q and K; the
// cos/sin rows are gathered by position id inside the kernel.
//
//   xn = bf16(x * rstd) * w            (per head, statistics over head_dim, when do_norm)
//   y[:h/2] = xn[:h/2] * cos - xn[h/2:] * sin ;  y[h/2:] = xn[h/2:] * cos + xn[:h/2] * sin
//
// Counterpart of the reference's Triton kernels (lset/kernels/qk_norm_rope.py:79-134,191-287 and
// lset/kernels/rope.py:12-75). Inputs may be slices of a fused QKV projection output (row strides
// are explicit), so no split/copy of the QKV tensor is needed.
#include "../common/api.h"
#include "../common/pdl.h"
#include "../common/row.cuh"

namespace lb {
namespace {

using bf16 = __nv_bfloat16;

struct RopeArgs {
  const bf16* q_in;
  const bf16* k_in;
  long long ldq_in, ldk_in;
  const bf16* qw;
  const bf16* kw;
  const float* cos;  // [P, hd/2]
  const float* sin;
  const void* pos;   // int32 or int64 [T]; nullptr -> token index modulo pos_mod
  int pos_i64;
  int pos_mod;
  bf16* q_out;
  bf16* k_out;
  long long ldq_out, ldk_out;
  float* q_rstd;  // [T, Hq]
  float* k_rstd;  // [T, Hk]
  int T, Hq, Hk;
  float eps, w_off;
  int do_norm;
  int parts, part_heads;  // lane groups per token, and the heads (of q and k together) each walks over
};

__device__ __forceinline__ int token_pos(const RopeArgs& a, long long tok) {
  if (a.pos == nullptr) return int(tok % a.pos_mod);
  return a.pos_i64 ? int(reinterpret_cast<const long long*>(a.pos)[tok])
                   : reinterpret_cast<const int*>(a.pos)[tok];
}

// A group of HD/16 lanes owns one token at a time (or, with few tokens, a part of its heads, see
// rope_parts) and walks over its heads UB at a time: the cos/sin
// row and the position are fetched once per token, and the 16-byte loads of the next UB heads are
// already in flight while the current UB heads are normalised, rotated and stored. A lane holds eight
// elements of either half of a head, the two partners of eight rotations, so that nothing but the sum of
// squares crosses lanes. (With a lane per eight neighbouring elements, every element came over once by
// shuffle, and the shuffles bound the kernel; the sum of squares is added up in the same order.)
// Measured (us, tokens x heads of 128, L2 flushed): 22627 x 24 72 -> 64, 40280 x 24 117 -> 94, 33280 x 40
// 156 -> 132 (65 % -> 81 % of copy bandwidth at 40280); 22627 x 40 heads of 64 59 -> 51.
template <int HD>
__global__ void __launch_bounds__(kRowThreads, 3) qk_rope_fwd_kernel(RopeArgs a) {
  constexpr int LPH = HD / 16;  // lanes per head
  constexpr int TPB = kRowThreads / LPH;
  constexpr int UB = 2;
  constexpr int HALF = HD / 2;
  __shared__ float swt[2 * HD];  // q then k norm weights (+ offset)
  const int l = threadIdx.x % LPH;
  const int g = threadIdx.x / LPH;
  const int e0 = l * 8;
  for (int i = threadIdx.x; i < 2 * HD; i += kRowThreads)
    swt[i] = a.do_norm ? __bfloat162float(i < HD ? a.qw[i] : a.kw[i - HD]) + a.w_off : 1.f;
  __syncthreads();
  pdl_wait();
  pdl_trigger();
  const unsigned total = unsigned(a.T) * a.parts;
  for (unsigned u0 = blockIdx.x * TPB; u0 < total; u0 += gridDim.x * TPB) {
    const unsigned tok_u = (u0 + g) / a.parts;
    const long long tok = tok_u;
    const bool valid = tok < a.T;
    const int h_first = int(u0 + g - tok_u * a.parts) * a.part_heads;
    const int heads = min(h_first + a.part_heads, a.Hq + a.Hk);
    const bf16* qrow = a.q_in + tok * a.ldq_in + e0;
    const bf16* krow = a.k_in + tok * a.ldk_in + e0;
    bf16* qdst = a.q_out + tok * a.ldq_out + e0;
    bf16* kdst = a.k_out + tok * a.ldk_out + e0;
    auto load_batch = [&](int h0, uint4 (&raw)[UB][2]) {
#pragma unroll
      for (int j = 0; j < UB; ++j) {
        const int h = h0 + j;
        raw[j][0] = raw[j][1] = make_uint4(0u, 0u, 0u, 0u);
        if (valid && h < heads) {
          const bf16* p = h < a.Hq ? qrow + h * HD : krow + (h - a.Hq) * HD;
          raw[j][0] = ld16(p);
          raw[j][1] = ld16(p + HALF);
        }
      }
    };
    uint4 cur[UB][2], nxt[UB][2];
    load_batch(h_first, cur);
    float c[8], s[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) c[i] = s[i] = 0.f;
    if (valid) {
      const int pos = token_pos(a, tok);
      const float4* cp = reinterpret_cast<const float4*>(a.cos + 1LL * pos * HALF + e0);
      const float4* sp = reinterpret_cast<const float4*>(a.sin + 1LL * pos * HALF + e0);
      *reinterpret_cast<float4*>(c) = cp[0];
      *reinterpret_cast<float4*>(c + 4) = cp[1];
      *reinterpret_cast<float4*>(s) = sp[0];
      *reinterpret_cast<float4*>(s + 4) = sp[1];
    }
    for (int b0 = 0; b0 < a.part_heads; b0 += UB) {   // uniform over the CTA
      const int h0 = h_first + b0;
      if (b0 + UB < a.part_heads) load_batch(h0 + UB, nxt);
#pragma unroll
      for (int j = 0; j < UB; ++j) {
        const int h = h0 + j;
        const bool live = valid && h < heads;
        const bool is_q = h < a.Hq;
        float x[2][8];
        unpack8(cur[j][0], x[0]);
        unpack8(cur[j][1], x[1]);
        if (a.do_norm) {
          float ss[2] = {0.f, 0.f};
#pragma unroll
          for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int i = 0; i < 8; ++i) ss[k] += x[k][i] * x[k][i];
          float sum = ss[0] + ss[1];
#pragma unroll
          for (int o = LPH / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
          const float rstd = rsqrtf(sum / float(HD) + a.eps);
          if (live && l == 0) {
            if (is_q) a.q_rstd[tok * a.Hq + h] = rstd;
            else a.k_rstd[tok * a.Hk + (h - a.Hq)] = rstd;
          }
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const float* wt = swt + (is_q ? 0 : HD) + k * HALF + e0;
            const float4 w0 = *reinterpret_cast<const float4*>(wt);
            const float4 w1 = *reinterpret_cast<const float4*>(wt + 4);
            const float wl[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) x[k][i] = bf16_round(x[k][i] * rstd) * wl[i];
          }
        }
        float y[2][8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          y[0][i] = x[0][i] * c[i] - x[1][i] * s[i];
          y[1][i] = x[1][i] * c[i] - x[0][i] * -s[i];
        }
        if (live) {
          bf16* p = is_q ? qdst + h * HD : kdst + (h - a.Hq) * HD;
          st16(p, pack8(y[0]));
          st16(p + HALF, pack8(y[1]));
        }
      }
#pragma unroll
      for (int j = 0; j < UB; ++j) {
        cur[j][0] = nxt[j][0];
        cur[j][1] = nxt[j][1];
      }
    }
  }
}

struct RopeBwdArgs {
  const bf16* dq;   // grads of rotated outputs
  const bf16* dk;
  long long lddq, lddk;
  const bf16* q_in;  // forward inputs (pre-norm)
  const bf16* k_in;
  long long ldq_in, ldk_in;
  const bf16* qw;
  const bf16* kw;
  const float* cos;
  const float* sin;
  const void* pos;
  int pos_i64;
  int pos_mod;
  const float* q_rstd;
  const float* k_rstd;
  bf16* dq_in;  // grads of the forward inputs
  bf16* dk_in;
  long long lddq_in, lddk_in;
  float* dw_partial;  // [grid, 2, HD]
  int T, Hq, Hk;
  float w_off;
  int do_norm;
  int parts, part_heads;
};

// Same token-per-lane-group walk as the forward kernel, UB heads at a time: the gradient rows, the forward
// inputs and the saved rstd of UB heads are requested before any of them is used. With few tokens a lane
// holds eight elements of either half of a head, as in the forward (HALVES 2): half the lanes a head, so
// half the CTAs, one wave of them. With many tokens registers bound the loads in flight, and eight
// neighbouring elements a lane, the partner's by shuffle (HALVES 1), are as fast or faster.
// Measured (us, tokens x 24 heads of 128, HALVES 1 / 2): 920 18.4 / 10.7, 2500 23 / 15, 6000 49 / 35,
// 22627 106 / 108, 40280 174 / 172; 22627 x 40 heads of 64 106 / 119.
template <int HD, int HALVES>
__global__ void __launch_bounds__(kRowThreads, 2) qk_rope_bwd_kernel(RopeBwdArgs a) {
  constexpr int LPH = HD / 8 / HALVES;
  constexpr int TPB = kRowThreads / LPH;
  constexpr int UB = 4 / HALVES;
  constexpr int HALF = HD / 2;
  __shared__ float sdw[2 * HD];
  __shared__ float swt[2 * HD];  // q then k norm weights (+ offset)
  const int l = threadIdx.x % LPH;
  const int g = threadIdx.x / LPH;
  const int e0 = l * 8;
  const int c0 = e0 % HALF;
  float dwq[HALVES][8], dwk[HALVES][8];
#pragma unroll
  for (int k = 0; k < HALVES; ++k)
#pragma unroll
    for (int i = 0; i < 8; ++i) dwq[k][i] = dwk[k][i] = 0.f;
  for (int i = threadIdx.x; i < 2 * HD; i += kRowThreads) {
    sdw[i] = 0.f;
    swt[i] = a.do_norm ? __bfloat162float(i < HD ? a.qw[i] : a.kw[i - HD]) + a.w_off : 1.f;
  }
  __syncthreads();
  RopeArgs pa;  // only the position fields are used by token_pos
  pa.pos = a.pos;
  pa.pos_i64 = a.pos_i64;
  pa.pos_mod = a.pos_mod;
  pdl_wait();
  pdl_trigger();

  const unsigned total = unsigned(a.T) * a.parts;
  for (unsigned u0 = blockIdx.x * TPB; u0 < total; u0 += gridDim.x * TPB) {
    const unsigned tok_u = (u0 + g) / a.parts;
    const long long tok = tok_u;
    const bool valid = tok < a.T;
    const int h_first = int(u0 + g - tok_u * a.parts) * a.part_heads;
    const int heads = min(h_first + a.part_heads, a.Hq + a.Hk);
    float c[8], s[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) c[i] = s[i] = 0.f;
    if (valid) {
      const int pos = token_pos(pa, tok);
      const float4* cp = reinterpret_cast<const float4*>(a.cos + 1LL * pos * HALF + c0);
      const float4* sp = reinterpret_cast<const float4*>(a.sin + 1LL * pos * HALF + c0);
      *reinterpret_cast<float4*>(c) = cp[0];
      *reinterpret_cast<float4*>(c + 4) = cp[1];
      *reinterpret_cast<float4*>(s) = sp[0];
      *reinterpret_cast<float4*>(s + 4) = sp[1];
    }
    if (e0 >= HALF) {   // (of a single half a lane: gn = g*c + partner*s in the first, - in the second)
#pragma unroll
      for (int i = 0; i < 8; ++i) s[i] = -s[i];
    }
    const bf16* gq = a.dq + tok * a.lddq + e0;
    const bf16* gk = a.dk + tok * a.lddk + e0;
    const bf16* xq = a.q_in + tok * a.ldq_in + e0;
    const bf16* xk = a.k_in + tok * a.ldk_in + e0;
    bf16* oq = a.dq_in + tok * a.lddq_in + e0;
    bf16* ok = a.dk_in + tok * a.lddk_in + e0;
    for (int b0 = 0; b0 < a.part_heads; b0 += UB) {
      const int h0 = h_first + b0;
      uint4 graw[UB][HALVES], xraw[UB][HALVES];
      float rs[UB];
#pragma unroll
      for (int j = 0; j < UB; ++j) {
        const int h = h0 + j;
#pragma unroll
        for (int k = 0; k < HALVES; ++k) graw[j][k] = xraw[j][k] = make_uint4(0u, 0u, 0u, 0u);
        rs[j] = 0.f;
        if (valid && h < heads) {
          const bool is_q = h < a.Hq;
          const bf16* gp = is_q ? gq + h * HD : gk + (h - a.Hq) * HD;
#pragma unroll
          for (int k = 0; k < HALVES; ++k) graw[j][k] = ld16(gp + k * HALF);
          if (a.do_norm) {
            const bf16* xp = is_q ? xq + h * HD : xk + (h - a.Hq) * HD;
#pragma unroll
            for (int k = 0; k < HALVES; ++k) xraw[j][k] = ld16(xp + k * HALF);
            rs[j] = is_q ? a.q_rstd[tok * a.Hq + h] : a.k_rstd[tok * a.Hk + (h - a.Hq)];
          }
        }
      }
#pragma unroll
      for (int j = 0; j < UB; ++j) {
        const int h = h0 + j;
        const bool live = valid && h < heads;   // (loads of the others are zero, and add nothing)
        const bool is_q = h < a.Hq;
        float gv[HALVES][8], gn[HALVES][8], o[HALVES][8];
#pragma unroll
        for (int k = 0; k < HALVES; ++k) unpack8(graw[j][k], gv[k]);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if constexpr (HALVES == 2) {
            gn[0][i] = gv[0][i] * c[i] + gv[1][i] * s[i];
            gn[1][i] = gv[1][i] * c[i] + gv[0][i] * -s[i];
          } else {
            const float p = __shfl_xor_sync(0xffffffffu, gv[0][i], LPH / 2);
            gn[0][i] = gv[0][i] * c[i] + p * s[i];
          }
        }
        if (a.do_norm) {
          float x[HALVES][8], m[HALVES][8], dots[HALVES] = {};
          const float rstd = rs[j];
#pragma unroll
          for (int k = 0; k < HALVES; ++k) {
            unpack8(xraw[j][k], x[k]);
            const float* wt = swt + (is_q ? 0 : HD) + k * HALF + e0;
            const float4 w0 = *reinterpret_cast<const float4*>(wt);
            const float4 w1 = *reinterpret_cast<const float4*>(wt + 4);
            const float wl[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              x[k][i] *= rstd;  // xhat
              m[k][i] = gn[k][i] * wl[i];
              dots[k] += m[k][i] * x[k][i];
              const float dwv = gn[k][i] * bf16_round(x[k][i]);
              if (is_q) dwq[k][i] += dwv;
              else dwk[k][i] += dwv;
            }
          }
          float dot = HALVES == 2 ? dots[0] + dots[HALVES - 1] : dots[0];
#pragma unroll
          for (int sh = LPH / 2; sh > 0; sh >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, sh);
          dot /= float(HD);
#pragma unroll
          for (int k = 0; k < HALVES; ++k)
#pragma unroll
            for (int i = 0; i < 8; ++i) o[k][i] = rstd * (m[k][i] - x[k][i] * dot);
        } else {
#pragma unroll
          for (int k = 0; k < HALVES; ++k)
#pragma unroll
            for (int i = 0; i < 8; ++i) o[k][i] = gn[k][i];
        }
        if (live) {
          bf16* p = is_q ? oq + h * HD : ok + (h - a.Hq) * HD;
#pragma unroll
          for (int k = 0; k < HALVES; ++k) st16(p + k * HALF, pack8(o[k]));
        }
      }
    }
  }
  if (a.do_norm && a.dw_partial != nullptr) {
    // the groups of a warp first: as many fewer additions to the same words of shared memory
#pragma unroll
    for (int k = 0; k < HALVES; ++k)
#pragma unroll
      for (int i = 0; i < 8; ++i) {
#pragma unroll
        for (int sh = 16; sh >= LPH; sh >>= 1) {
          dwq[k][i] += __shfl_xor_sync(0xffffffffu, dwq[k][i], sh);
          dwk[k][i] += __shfl_xor_sync(0xffffffffu, dwk[k][i], sh);
        }
        if ((threadIdx.x & 31) < LPH) {
          atomicAdd(&sdw[k * HALF + e0 + i], dwq[k][i]);
          atomicAdd(&sdw[HD + k * HALF + e0 + i], dwk[k][i]);
        }
      }
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * HD; i += kRowThreads)
      a.dw_partial[1LL * blockIdx.x * 2 * HD + i] = sdw[i];
  }
}

}  // namespace
}  // namespace lb

using namespace lb;

// Lane groups per token. One walks over all heads, the next loads in flight under the current heads'
// arithmetic, which is what the kernels are bound by with many tokens (a group for every four heads:
// 142 against 127 us at 40280 tokens of 16 + 8 heads of 128). With so few tokens that the groups
// are fewer than the SMs hold, the walk is a chain of latencies, and a group for every few heads is
// faster (32 tokens: 21 against 29 us, 1024: 20 against 27; about 10 us of each are the measurement's own).
static bool few_tokens(int T, int hd) {
  return 1LL * T < 3LL * row_num_sms() * (kRowThreads / (hd / 16)) / 2;
}
static void rope_parts(bool few, int heads, int unit, int* parts, int* part_heads) {
  const int all = (heads + unit - 1) / unit;
  *parts = few ? all : 1;
  *part_heads = few ? unit : all * unit;
}

extern "C" int lb_rope_bwd_partial_rows() { return row_num_sms() * 8; }

extern "C" int lb_qk_norm_rope_fwd(const void* q_in, long long ldq_in, const void* k_in,
                                   long long ldk_in, const void* qw, const void* kw,
                                   const float* cos, const float* sin, const void* pos, int pos_i64,
                                   int pos_mod, void* q_out, long long ldq_out, void* k_out,
                                   long long ldk_out, float* q_rstd, float* k_rstd, int T, int Hq,
                                   int Hk, int hd, float eps, float w_off, int do_norm,
                                   void* stream) {
  if (T <= 0) return 0;
  if ((ldq_in | ldk_in | ldq_out | ldk_out) & 7) return -3;
  if (1LL * T * (Hq + Hk) >= (1LL << 32)) return -3;
  RopeArgs a{(const bf16*)q_in, (const bf16*)k_in, ldq_in, ldk_in, (const bf16*)qw, (const bf16*)kw,
             cos, sin, pos, pos_i64, pos_mod > 0 ? pos_mod : 1, (bf16*)q_out, (bf16*)k_out, ldq_out,
             ldk_out, q_rstd, k_rstd, T, Hq, Hk, eps, w_off, do_norm, 1, 0};
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  auto run = [&](auto kern, int lph) {
    const int tpb = kRowThreads / lph;
    rope_parts(few_tokens(T, hd), Hq + Hk, 2, &a.parts, &a.part_heads);
    const long long g = (1LL * T * a.parts + tpb - 1) / tpb;
    const long long cap = 1LL * row_num_sms() * 3;  // one wave at three CTAs per SM
    return launch_pdl(kern, dim3(unsigned(g < cap ? g : cap)), dim3(kRowThreads), 0, st,
                      pdl_enabled(), 1, a);
  };
  if (hd == 128) return run(qk_rope_fwd_kernel<128>, 8);
  if (hd == 64) return run(qk_rope_fwd_kernel<64>, 4);
  if (hd == 256) return run(qk_rope_fwd_kernel<256>, 16);
  return -3;
}

// CTAs of the backward, each of which leaves a partial row in its scratch.
extern "C" int lb_rope_bwd_rows(int T, int Hq, int Hk, int hd) {
  if (T <= 0 || hd < 64) return 0;
  const bool few = few_tokens(T, hd);
  int parts, part_heads;
  rope_parts(few, Hq + Hk, few ? 2 : 4, &parts, &part_heads);
  const int tpb = kRowThreads / (hd / (few ? 16 : 8));
  const long long g = (1LL * T * parts + tpb - 1) / tpb;
  const long long cap = 1LL * row_num_sms() * (few ? 2 : 4);
  return int(g < cap ? g : cap);
}

// dw_out: [2, hd] (q weight grad then k weight grad); scratch: lb_rope_bwd_partial_rows()*2*hd floats.
extern "C" int lb_qk_norm_rope_bwd(const void* dq, long long lddq, const void* dk, long long lddk,
                                   const void* q_in, long long ldq_in, const void* k_in,
                                   long long ldk_in, const void* qw, const void* kw,
                                   const float* cos, const float* sin, const void* pos, int pos_i64,
                                   int pos_mod, const float* q_rstd, const float* k_rstd,
                                   void* dq_in, long long lddq_in, void* dk_in, long long lddk_in,
                                   float* scratch, void* dw_out, int dw_fp32, int dw_accumulate,
                                   int T, int Hq, int Hk, int hd, float w_off, int do_norm,
                                   void* stream) {
  if (T <= 0) return 0;
  if ((lddq | lddk | ldq_in | ldk_in | lddq_in | lddk_in) & 7) return -3;
  if (1LL * T * (Hq + Hk) >= (1LL << 32)) return -3;
  RopeBwdArgs a{(const bf16*)dq, (const bf16*)dk, lddq, lddk, (const bf16*)q_in, (const bf16*)k_in,
                ldq_in, ldk_in, (const bf16*)qw, (const bf16*)kw, cos, sin, pos, pos_i64,
                pos_mod > 0 ? pos_mod : 1, q_rstd, k_rstd, (bf16*)dq_in, (bf16*)dk_in, lddq_in,
                lddk_in, scratch, T, Hq, Hk, w_off, do_norm, 1, 0};
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int grid = lb_rope_bwd_rows(T, Hq, Hk, hd);
  const bool few = few_tokens(T, hd);
  rope_parts(few, Hq + Hk, few ? 2 : 4, &a.parts, &a.part_heads);
  auto run = [&](auto kern) {
    return launch_pdl(kern, dim3(grid), dim3(kRowThreads), 0, st, pdl_enabled(), 1, a);
  };
  int rc = -3;
  if (hd == 128) rc = few ? run(qk_rope_bwd_kernel<128, 2>) : run(qk_rope_bwd_kernel<128, 1>);
  else if (hd == 64) rc = few ? run(qk_rope_bwd_kernel<64, 2>) : run(qk_rope_bwd_kernel<64, 1>);
  else if (hd == 256) rc = few ? run(qk_rope_bwd_kernel<256, 2>) : run(qk_rope_bwd_kernel<256, 1>);
  if (rc) return rc;
  if (do_norm && dw_out != nullptr && scratch != nullptr) {
    return lb_colsum(scratch, grid, 2 * hd, dw_out, dw_fp32, dw_accumulate, stream);
  }
  return launch_rc();
}
