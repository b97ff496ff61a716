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
#include "rope.cuh"

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
  return a.pos == nullptr ? int(tok % a.pos_mod) : rope_pos(a.pos, a.pos_i64, tok);
}

// A group of HD/16 lanes owns one token at a time (or, with few tokens, a part of its heads, see
// rope_parts) and walks over its heads UB at a time: the cos/sin
// row and the position are fetched once per token, and the 16-byte loads of the next UB heads are
// already in flight while the current UB heads are normalised, rotated and stored. A lane holds eight
// elements of either half of a head, the two partners of eight rotations, so that nothing but the sum of
// squares crosses lanes. (With a lane per eight neighbouring elements, every element came over once by
// shuffle, and the shuffles bound the kernel; the sum of squares is added up in the same order.)
// Measured (us, tokens x heads of 128, L2 flushed): 22627 x 24 72 -> 62, 40280 x 24 117 -> 94, 33280 x 40
// 156 -> 132 (65 % -> 81 % of copy bandwidth at 40280); 22627 x 40 heads of 64 59 -> 55. Two elements an
// instruction, and weights without bank conflicts, change nothing there, but among GEMMs, which take the clock
// down: 40280 x 24 116 -> 108, 22627 x 24 77 -> 73.
template <int HD>
__global__ void __launch_bounds__(kRowThreads, 3) qk_rope_fwd_kernel(RopeArgs a) {
  constexpr int LPH = HD / 16;  // lanes per head
  constexpr int TPB = kRowThreads / LPH;
  constexpr int UB = 2;
  constexpr int HALF = HD / 2;
  __shared__ __align__(16) float swt[2 * HD];  // q then k norm weights (+ offset): [half][4 of 8][lane][4]
  const int l = threadIdx.x % LPH;
  const int g = threadIdx.x / LPH;
  const int e0 = l * 8;
  for (int i = threadIdx.x; i < 2 * HD; i += kRowThreads)
    swt[weight_at<HD>(i)] =
        a.do_norm ? __bfloat162float(i < HD ? a.qw[i] : a.kw[i - HD]) + a.w_off : 1.f;
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
    f2 c[4], s[4];
    load_angles<HALF>(a.cos, a.sin, valid ? token_pos(a, tok) : -1, e0, c, s);
    for (int b0 = 0; b0 < a.part_heads; b0 += UB) {   // uniform over the CTA
      const int h0 = h_first + b0;
      if (b0 + UB < a.part_heads) load_batch(h0 + UB, nxt);
#pragma unroll
      for (int j = 0; j < UB; ++j) {
        const int h = h0 + j;
        const bool live = valid && h < heads;
        const bool is_q = h < a.Hq;
        f2 y[2][4];
        rope_head<HD>(cur[j], a.do_norm, swt + (is_q ? 0 : HD) + l * 4, a.eps, c, s, y, [&](float rstd) {
          if (live && l == 0) {
            if (is_q) a.q_rstd[tok * a.Hq + h] = rstd;
            else a.k_rstd[tok * a.Hk + (h - a.Hq)] = rstd;
          }
        });
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
  int grid;               // partial rows of dW; a CTA of each for q's heads, then one for k's
  int parts, part_heads;  // as of the forward
};

// Threads of a CTA, and lane groups, each of which owns a token at a time.
constexpr int kRopeBwdThreads = 128;
constexpr int rope_bwd_groups(int hd) { return kRopeBwdThreads / (hd / 16); }

// Same token-per-lane-group walk as the forward kernel, UB heads at a time: the gradient rows, the forward
// inputs and the saved rstd of UB heads are requested before any of them is used, and registers bound how
// many those are. So a CTA walks over q's heads or over k's, with the weights of the one in registers and one
// set of dW accumulators, and a lane holds eight elements of either half of a head, as in the forward.
//
// dW has one order of summation, part of the bits of a training step (the gradient norm, and through the clip
// coefficient every weight): group g of row r of `grid` partial rows adds up its units' heads, in ascending order, of
// units r * TPB + g + i * grid * TPB (a unit: part_heads of q's and k's heads of a token), then the
// groups one after the other.
// Measured with both kinds a CTA, weights in shared memory and an element an instruction / now (us, tokens x
// 24 heads of 128, L2 flushed): 22627 105 / 84, 40280 174 / 135, 8000 52 / 37, 3000 31 / 25, 1200 24 / 16; 33280 x
// 40 225 / 178; 22627 x 40 heads of 64 107 / 77. Groups of two heads of one kind for few tokens take 20 at 3000 and
// 14 at 1200, in another order of summation. (Three CTAs a SM with a head at a time: 119 at 22627.)
template <int HD>
__global__ void __launch_bounds__(kRopeBwdThreads, 4) qk_rope_bwd_kernel(RopeBwdArgs a) {
  constexpr int LPH = HD / 16;
  constexpr int TPB = rope_bwd_groups(HD);
  constexpr int UB = 2;
  constexpr int HALF = HD / 2;
  __shared__ float sdw[TPB][HD];
  const int l = threadIdx.x % LPH;
  const int g = threadIdx.x / LPH;
  const int e0 = l * 8;
  const bool is_q = int(blockIdx.x) < a.grid;
  const unsigned cta = is_q ? blockIdx.x : blockIdx.x - a.grid;
  const int H = is_q ? a.Hq : a.Hk, h_from = is_q ? 0 : a.Hq;   // of the heads of both
  const int span = min(H, a.part_heads);
  f2 dw[2][4], wt[2][4];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    uint4 q = make_uint4(0u, 0u, 0u, 0u);
    if (a.do_norm) {
      float f[8];   // (a weight may start at any element)
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = __bfloat162float((is_q ? a.qw : a.kw)[k * HALF + e0 + i]) + a.w_off;
#pragma unroll
      for (int i = 0; i < 4; ++i) wt[k][i] = f2_of(f[2 * i], f[2 * i + 1]);
    } else {
      unpack8(q, wt[k]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) dw[k][i] = 0ull;
  }
  RopeArgs pa;  // only the position fields are used by token_pos
  pa.pos = a.pos;
  pa.pos_i64 = a.pos_i64;
  pa.pos_mod = a.pos_mod;
  const bf16* gp = (is_q ? a.dq : a.dk) + e0;
  const bf16* xp = (is_q ? a.q_in : a.k_in) + e0;
  bf16* op = (is_q ? a.dq_in : a.dk_in) + e0;
  const float* rp = is_q ? a.q_rstd : a.k_rstd;
  const long long ldg = is_q ? a.lddq : a.lddk, ldx = is_q ? a.ldq_in : a.ldk_in;
  const long long ldo = is_q ? a.lddq_in : a.lddk_in;
  pdl_wait();
  pdl_trigger();

  const unsigned total = unsigned(a.T) * a.parts;
  for (unsigned u0 = cta * TPB; u0 < total; u0 += a.grid * TPB) {
    const unsigned tok_u = (u0 + g) / a.parts;
    const long long tok = tok_u;
    const int first = int(u0 + g - tok_u * a.parts) * a.part_heads - h_from;
    const int h_first = max(first, 0), heads = min(first + a.part_heads, H);
    const bool valid = tok < a.T && h_first < heads;
    if (__all_sync(0xffffffffu, !valid)) continue;   // (the warp's parts are heads of the other kind)
    f2 c[4], s[4];
    load_angles<HALF>(a.cos, a.sin, valid ? token_pos(pa, tok) : -1, e0, c, s);
    for (int b0 = 0; b0 < span; b0 += UB) {
      const int h0 = h_first + b0;
      uint4 graw[UB][2], xraw[UB][2];
      float rs[UB];
#pragma unroll
      for (int j = 0; j < UB; ++j) {
        const int h = h0 + j;
#pragma unroll
        for (int k = 0; k < 2; ++k) graw[j][k] = xraw[j][k] = make_uint4(0u, 0u, 0u, 0u);
        rs[j] = 0.f;
        if (valid && h < heads) {
#pragma unroll
          for (int k = 0; k < 2; ++k) graw[j][k] = ld16(gp + tok * ldg + h * HD + k * HALF);
          if (a.do_norm) {
#pragma unroll
            for (int k = 0; k < 2; ++k) xraw[j][k] = ld16(xp + tok * ldx + h * HD + k * HALF);
            rs[j] = rp[tok * H + h];
          }
        }
      }
#pragma unroll
      for (int j = 0; j < UB; ++j) {
        const int h = h0 + j;
        const bool live = valid && h < heads;   // (loads of the others are zero, and add nothing)
        f2 gv[2][4], gn[2][4];
        unpack8(graw[j][0], gv[0]);
        unpack8(graw[j][1], gv[1]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          gn[0][i] = f2_fma(gv[0][i], c[i], f2_mul(gv[1][i], s[i]));
          gn[1][i] = f2_fma(gv[1][i], c[i], f2_neg(f2_mul(gv[0][i], s[i])));
        }
        if (a.do_norm) {
          f2 x[2][4];
          float dots[2] = {0.f, 0.f};
          const f2 r2 = f2_of(rs[j], rs[j]);
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            unpack8(xraw[j][k], x[k]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              x[k][i] = f2_mul(x[k][i], r2);  // xhat
              dw[k][i] = f2_fma(gn[k][i], f2_bf16_round(x[k][i]), dw[k][i]);
              gn[k][i] = f2_mul(gn[k][i], wt[k][i]);
              const float2 m = f2_get(gn[k][i]), xh = f2_get(x[k][i]);
              dots[k] = fmaf(m.x, xh.x, dots[k]);
              dots[k] = fmaf(m.y, xh.y, dots[k]);
            }
          }
          float dot = dots[0] + dots[1];
#pragma unroll
          for (int sh = LPH / 2; sh > 0; sh >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, sh);
          dot /= float(HD);
          const f2 minus_dot = f2_of(-dot, -dot);
#pragma unroll
          for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int i = 0; i < 4; ++i)
              gn[k][i] = f2_mul(r2, f2_fma(x[k][i], minus_dot, gn[k][i]));
        }
        if (live) {
#pragma unroll
          for (int k = 0; k < 2; ++k) st16(op + tok * ldo + h * HD + k * HALF, pack8(gn[k]));
        }
      }
    }
  }
  if (a.do_norm && a.dw_partial != nullptr) {
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 v = f2_get(dw[k][i]);
        sdw[g][k * HALF + e0 + 2 * i] = v.x;
        sdw[g][k * HALF + e0 + 2 * i + 1] = v.y;
      }
    __syncthreads();
    for (int i = threadIdx.x; i < HD; i += kRopeBwdThreads) {
      float t = 0.f;
#pragma unroll
      for (int j = 0; j < TPB; ++j) t += sdw[j][i];
      a.dw_partial[(2LL * cta + (is_q ? 0 : 1)) * HD + i] = t;
    }
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
static void rope_parts(int T, int tokens_per_cta, int heads, int unit, int* parts, int* part_heads) {
  const bool few = 1LL * T < 3LL * row_num_sms() * tokens_per_cta / 2;
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
    rope_parts(T, tpb, Hq + Hk, 2, &a.parts, &a.part_heads);
    const long long g = (1LL * T * a.parts + tpb - 1) / tpb;
    const long long cap = 1LL * row_num_sms() * 3;  // one wave at three CTAs per SM
    return launch_pdl(kern, dim3(unsigned(g < cap ? g : cap)), dim3(kRowThreads), 0, st,
                      pdl_enabled(4LL * T * (Hq + Hk) * hd), 1, a);
  };
  if (hd == 128) return run(qk_rope_fwd_kernel<128>, 8);
  if (hd == 64) return run(qk_rope_fwd_kernel<64>, 4);
  if (hd == 256) return run(qk_rope_fwd_kernel<256>, 16);
  return -3;
}

// Partial rows of dW that the backward leaves in its scratch: with the parts, its order of summation.
static int rope_bwd_plan(int T, int heads, int hd, int* parts, int* part_heads) {
  const int groups = rope_bwd_groups(hd);
  rope_parts(T, groups, heads, 4, parts, part_heads);
  const long long need = (1LL * T * *parts + groups - 1) / groups, cap = 4LL * row_num_sms();
  return int(need < cap ? need : cap);
}
extern "C" int lb_rope_bwd_rows(int T, int Hq, int Hk, int hd) {
  if (T <= 0 || hd < 64) return 0;
  int parts, part_heads;
  return rope_bwd_plan(T, Hq + Hk, hd, &parts, &part_heads);
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
                lddk_in, scratch, T, Hq, Hk, w_off, do_norm};
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (hd != 64 && hd != 128 && hd != 256) return -3;
  a.grid = rope_bwd_plan(T, Hq + Hk, hd, &a.parts, &a.part_heads);
  auto run = [&](auto kern) {
    return launch_pdl(kern, dim3(2 * a.grid), dim3(kRopeBwdThreads), 0, st,
                      pdl_enabled(6LL * T * (Hq + Hk) * hd), 1, a);
  };
  int rc = -3;
  if (hd == 128) rc = run(qk_rope_bwd_kernel<128>);
  else if (hd == 64) rc = run(qk_rope_bwd_kernel<64>);
  else if (hd == 256) rc = run(qk_rope_bwd_kernel<256>);
  if (rc) return rc;
  if (do_norm && dw_out != nullptr && scratch != nullptr) {
    return lb_colsum(scratch, a.grid, 2 * hd, dw_out, dw_fp32, dw_accumulate, stream);
  }
  return launch_rc();
}
