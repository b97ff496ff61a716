// Decoder-block runner: see block.h. Host code only, except for one small scaling kernel; every
// heavy launch goes through the library's own launchers (declared in common/api.h).
#include "block.h"

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../common/api.h"
#include "../common/pdl.h"
#include "../gemm/gemm_small.h"

namespace {

constexpr size_t kAlign = 256;

inline size_t up(size_t x) { return (x + kAlign - 1) / kAlign * kAlign; }

inline int tp_tokens(const LbTpCtx* tp) { return tp->world * tp->rows; }

// Carves 256-byte aligned slices out of one arena. With a null base it only measures.
struct Arena {
  char* base;
  size_t off = 0;
  explicit Arena(void* b) : base(static_cast<char*>(b)) {}
  void* take(size_t bytes) {
    void* p = base ? base + off : nullptr;
    off += up(bytes);
    return p;
  }
  __nv_bfloat16* bf(size_t n) { return static_cast<__nv_bfloat16*>(take(n * 2)); }
  float* f32(size_t n) { return static_cast<float*>(take(n * 4)); }
};

__global__ void scale_bf16_kernel(__nv_bfloat16* x, long long n, float s) {
  lb::pdl_wait();
  lb::pdl_trigger();
  long long i = blockIdx.x * 1LL * blockDim.x + threadIdx.x;
  const long long step = 1LL * gridDim.x * blockDim.x;
  for (; i < n; i += step) x[i] = __float2bfloat16_rn(__bfloat162float(x[i]) * s);
}

int scale_bf16(__nv_bfloat16* x, long long n, float s, cudaStream_t st) {
  if (n <= 0) return 0;
  long long g = (n + 255) / 256;
  if (g > 1184) g = 1184;
  return lb::launch_pdl(scale_bf16_kernel, dim3(unsigned(g)), dim3(256), 0, st, lb::pdl_enabled(), 1, x,
                        n, s);
}

struct Saved {
  __nv_bfloat16 *x1, *res1, *qkv, *qr, *kr, *o, *x2, *gu, *h;
  float *rstd1, *rstd2, *q_rstd, *k_rstd, *lse;
  __nv_bfloat16* ts[8];  // LoRA: s · x · Aᵀ per linear (qkv parts 0-2, o 3, gate_up parts 4-5, down 6)
};

const LbLinear* linear_at(const LbBlockDesc* d, int i) {
  switch (i) {
    case 0: case 1: case 2: return i < d->qkv.n ? &d->qkv.part[i] : nullptr;
    case 3: return &d->o_proj;
    case 4: case 5: return i - 4 < d->gate_up.n ? &d->gate_up.part[i - 4] : nullptr;
    case 6: return &d->down;
    default: return nullptr;
  }
}

// `T` rows for everything the projections and the attention see; `R` rows for what lives on the
// token-sharded stream (R == T when the stream is not sharded).
Saved carve_saved(const LbBlockDesc* d, int T, int R, int has_residual, Arena& a) {
  Saved s{};
  const size_t t = (size_t)T, r = (size_t)R;
  s.x1 = a.bf(t * d->H);
  s.res1 = has_residual ? a.bf(r * d->H) : nullptr;
  s.rstd1 = a.f32(r);
  s.qkv = a.bf(t * d->qkv.width);
  s.qr = a.bf(t * d->Hq * d->hd);
  s.kr = a.bf(t * d->Hk * d->hd);
  s.q_rstd = d->qk_norm ? a.f32(t * d->Hq) : nullptr;
  s.k_rstd = d->qk_norm ? a.f32(t * d->Hk) : nullptr;
  s.o = a.bf(t * d->Hq * d->hd);
  s.lse = a.f32(t * d->Hq);
  s.rstd2 = a.f32(r);
  s.x2 = a.bf(t * d->H);
  s.gu = a.bf(t * d->gate_up.width);
  s.h = a.bf(t * d->I);
  for (int i = 0; i < 7; ++i) {
    const LbLinear* l = linear_at(d, i);
    s.ts[i] = (l != nullptr && l->lora_r > 0) ? a.bf(t * l->lora_r) : nullptr;
  }
  return s;
}

struct Work {
  __nv_bfloat16 *dres2, *dh, *dgu, *dx2, *dO, *dqr, *dkr, *dqkv, *dx1, *us;
  __nv_bfloat16 *dy_all, *dres_all;  // token-sharded stream: gathered output gradients
  float* delta;
};

Work carve_work(const LbBlockDesc* d, int T, int R, bool sharded, Arena& a) {
  Work w{};
  const size_t t = (size_t)T, r = (size_t)R;
  w.dres2 = sharded ? nullptr : a.bf(r * d->H);  // sharded: lives in the publication area
  int rmax = 0;
  for (int i = 0; i < 7; ++i) {
    const LbLinear* l = linear_at(d, i);
    if (l != nullptr && l->lora_r > rmax) rmax = l->lora_r;
  }
  w.us = rmax > 0 ? a.bf(t * rmax) : nullptr;
  // The MLP half of the backward is finished before the attention half starts: both overlay
  // the same region.
  const size_t mark = a.off;
  w.dy_all = sharded ? a.bf(t * d->H) : nullptr;
  w.dh = a.bf(t * d->I);
  w.dgu = a.bf(t * d->gate_up.width);
  w.dx2 = a.bf(r * d->H);
  const size_t end_mlp = a.off;
  a.off = mark;
  w.dres_all = sharded ? a.bf(t * d->H) : nullptr;
  w.dO = a.bf(t * d->Hq * d->hd);
  w.dqr = a.bf(t * d->Hq * d->hd);
  w.dkr = a.bf(t * d->Hk * d->hd);
  w.dqkv = a.bf(t * d->qkv.width);
  w.dx1 = a.bf(r * d->H);
  w.delta = a.f32(t * d->Hq);
  if (a.off < end_mlp) a.off = end_mlp;
  return w;
}

#define LB_TRY(expr)          \
  do {                        \
    const int rc_ = (expr);   \
    if (rc_ != 0) return rc_; \
  } while (0)

thread_local int t_fewer = 0;  // launches saved by the current call

// Fills in the tile width and split of `g`: whether it is modelled to take less than `alternative`.
bool small_wins(LbSmallGemm* g, double alternative) {
  if (!lb_gemm_use_2cta(-1)) return false;
  const double cost = lb_gemm_small_plan(g, &g->bn, &g->splits);
  return cost >= 0.0 && cost < alternative;
}

LbSmallGemm small_linear(const LbLinear& l, const __nv_bfloat16* x, long long ldx, __nv_bfloat16* y,
                         long long ldy, int T, const LbStreamCtx* c, const void* bias) {
  LbSmallGemm g = {};
  g.A = x;
  g.B[0] = l.w;
  g.C[0] = y;
  g.lda = ldx;
  g.ldb[0] = l.ldw;
  g.ldc[0] = ldy;
  g.M = T;
  g.N = g.ext[0] = l.n_out;
  g.K = l.k_in;
  g.nparts = 1;
  g.mode = kParallelN;
  g.b_ready = 1;
  g.may_split = c->may_split;
  g.bias[0] = bias;
  g.status = c->status;
  g.stream = c->stream;
  return g;
}

// Adapters: ts_i = s · x · A_iᵀ [T, r] of linears that share their input. One launch reads x for all of them
// (33280 x 4096, rank 16, for q, k and v: 3 x 66 us and a launch for each scale apart, 98 together; gate and up
// 74).
int lora_fwd_products(const LbLinear* l, int n, const __nv_bfloat16* x, long long ldx, int T,
                      __nv_bfloat16* const* ts, const LbStreamCtx* c) {
  bool any = false;
  for (int i = 0; i < n; ++i) any = any || l[i].lora_r > 0;
  if (!any) return 0;
  LbSmallGemm g = small_linear(l[0], x, ldx, nullptr, 0, T, c, nullptr);
  double apart = 0.0;
  bool same = true;
  g.N = 0;
  for (int i = 0; i < n; ++i) {
    g.B[i] = l[i].lora_a;
    g.ldb[i] = l[i].k_in;
    g.C[i] = ts[i];
    g.ldc[i] = g.ext[i] = l[i].lora_r;
    g.N += l[i].lora_r;
    apart += lb_gemm_tile_cost(T, l[i].lora_r, l[i].k_in, 0, 0) + 3.5;
    same = same && l[i].lora_r > 0 && l[i].k_in == l[0].k_in && l[i].lora_scale == l[0].lora_scale;
  }
  g.nparts = n;
  if (same && l[0].lora_scale != 0.f && small_wins(&g, apart)) {
    t_fewer += 2 * n - 1;
    return lb_gemm_small_scaled(&g, l[0].lora_scale);
  }
  for (int i = 0; i < n; ++i) {
    if (l[i].lora_r == 0) continue;
    if (n > 1) {
      LB_TRY(lora_fwd_products(l + i, 1, x, ldx, T, ts + i, c));
      continue;
    }
    LB_TRY(lb_gemm_bf16(x, l[i].lora_a, ts[i], T, l[i].lora_r, l[i].k_in, ldx, l[i].k_in, l[i].lora_r, 0, 0, 0,
                        0, nullptr, 1, 0, c->status, c->stream));
    LB_TRY(scale_bf16(ts[i], 1LL * T * l[i].lora_r, l[i].lora_scale,
                      reinterpret_cast<cudaStream_t>(c->stream)));
  }
  return 0;
}

// y[:, :n_out] (row stride ldy) = x · Wᵀ (+ LoRA). `ts` receives s · x · Aᵀ when the linear has adapters.
int lin_fwd(const LbLinear& l, const __nv_bfloat16* x, long long ldx, __nv_bfloat16* y,
            long long ldy, int T, __nv_bfloat16* ts, const LbStreamCtx* c,
            const void* bias = nullptr, bool ts_ready = false) {
  if (l.lora_r > 0) {
    if (!ts_ready) LB_TRY(lora_fwd_products(&l, 1, x, ldx, T, &ts, c));
    return lb_gemm_bf16_ext(x, l.w, ts, l.lora_b, y, T, l.n_out, l.k_in, l.lora_r, ldx, l.ldw,
                            l.lora_r, l.lora_r, ldy, 0, nullptr, c->status, c->stream);
  }
  if (c->may_split) {
    LbSmallGemm g = small_linear(l, x, ldx, y, ldy, T, c, bias);
    if (small_wins(&g, lb_gemm_tile_cost(T, l.n_out, l.k_in, 0, bias != nullptr)))
      return lb_gemm_small(&g);
  }
  return lb_gemm_bf16(x, l.w, y, T, l.n_out, l.k_in, ldx, l.ldw, ldy, 0, 0, 0, 0, bias, 1, 0,
                      c->status, c->stream);
}

// g = GELU(u), u = x · Wᵀ + bias, both [T, n_out] contiguous; u is left unwritten where one launch does both
// and it is not to be kept.
int lin_gelu_fwd(const LbLinear& l, const __nv_bfloat16* x, long long ldx, __nv_bfloat16* u, bool keep_u,
                 __nv_bfloat16* gelu, int I, int T, const LbStreamCtx* c, const void* bias) {
  if (l.lora_r == 0) {
    LbSmallGemm g = small_linear(l, x, ldx, keep_u ? u : nullptr, I, T, c, bias);
    g.glu_h = gelu;
    g.ld_h = I;
    g.glu_kind = 2;
    // (beside it the activation: a launch, two passes at 5 TB/s)
    if (small_wins(&g, lb_gemm_tile_cost(T, l.n_out, l.k_in, 0, bias != nullptr) + 2.5 + 4.0 * T * I / 5e6)) {
      ++t_fewer;
      return lb_gemm_small(&g);
    }
  }
  LB_TRY(lin_fwd(l, x, ldx, u, I, T, nullptr, c, bias));
  return lb_gelu_fwd(u, gelu, 1LL * T * I, c->stream);
}

// dx[T, k_in] (contiguous) = or += dy · W (+ s · (dy · B) · A). `us` is scratch for s · dy · B and is
// left filled for the weight-gradient step that follows.
int lin_dgrad(const LbLinear& l, const __nv_bfloat16* dy, long long lddy, __nv_bfloat16* dx, int T,
              bool accumulate, __nv_bfloat16* us, const LbStreamCtx* c) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(c->stream);
  const void* peers[1] = {dx};
  if (l.lora_r > 0) {
    LbSmallGemm g = small_linear(l, dy, lddy, us, l.lora_r, T, c, nullptr);
    g.B[0] = l.lora_b;
    g.ldb[0] = g.N = g.ext[0] = l.lora_r;
    g.K = l.n_out;
    g.b_mn = 1;
    if (l.lora_scale != 0.f && small_wins(&g, lb_gemm_tile_cost(T, l.lora_r, l.n_out, 0, 0) + 3.5)) {
      ++t_fewer;
      LB_TRY(lb_gemm_small_scaled(&g, l.lora_scale));
    } else {
      LB_TRY(lb_gemm_bf16(dy, l.lora_b, us, T, l.lora_r, l.n_out, lddy, l.lora_r, l.lora_r, 0, 1, 0, 0,
                          nullptr, 1, 0, c->status, c->stream));
      LB_TRY(scale_bf16(us, 1LL * T * l.lora_r, l.lora_scale, st));
    }
    if (!accumulate)
      return lb_gemm_bf16_ext(dy, l.w, us, l.lora_a, dx, T, l.k_in, l.n_out, l.lora_r, lddy, l.ldw,
                              l.lora_r, l.k_in, l.k_in, 1, nullptr, c->status, c->stream);
    LB_TRY(lb_gemm_bf16_scatter16(dy, l.w, peers, 1, T, T, l.k_in, l.n_out, lddy, l.ldw, l.k_in, 0,
                                  1, 0, c->status, c->stream));
    return lb_gemm_bf16_scatter16(us, l.lora_a, peers, 1, T, T, l.k_in, l.lora_r, l.lora_r, l.k_in,
                                  l.k_in, 0, 1, 0, c->status, c->stream);
  }
  if (!accumulate)
    return lb_gemm_bf16(dy, l.w, dx, T, l.k_in, l.n_out, lddy, l.ldw, l.k_in, 0, 1, 0, 0, nullptr, 1,
                        0, c->status, c->stream);
  return lb_gemm_bf16_scatter16(dy, l.w, peers, 1, T, T, l.k_in, l.n_out, lddy, l.ldw, l.k_in, 0, 1,
                                0, c->status, c->stream);
}

// dW += dyᵀ · x; adapters: dA += usᵀ · x, dB += dyᵀ · ts. Frozen tensors (null accumulators) are skipped.
int lin_wgrad(const LbLinear& l, const __nv_bfloat16* dy, long long lddy, const __nv_bfloat16* x,
              long long ldx, int T, const __nv_bfloat16* ts, const __nv_bfloat16* us,
              const LbStreamCtx* c) {
  if (l.wgrad != nullptr)
    LB_TRY(lb_gemm_bf16(dy, x, l.wgrad, l.n_out, l.k_in, T, lddy, ldx, l.k_in, 1, 1, 1, 1, nullptr,
                        0 /*auto*/, 0, c->status, c->stream));
  if (l.lora_r > 0) {
    if (l.lora_a_grad != nullptr)
      LB_TRY(lb_gemm_bf16(us, x, l.lora_a_grad, l.lora_r, l.k_in, T, l.lora_r, ldx, l.k_in, 1, 1, 1,
                          1, nullptr, 0, 0, c->status, c->stream));
    if (l.lora_b_grad != nullptr)
      LB_TRY(lb_gemm_bf16(dy, ts, l.lora_b_grad, l.n_out, l.lora_r, T, lddy, l.lora_r, l.lora_r, 1,
                          1, 1, 1, nullptr, 0, 0, c->status,
                          c->stream));
  }
  return 0;
}

// ---- projections with several linears in one launch -----------------------------------------------
// A product with few tokens goes to lb_gemm_small, and there all linears of a projection are one
// launch. `alternative` is the modelled time of the launches it replaces.
bool plain(const LbProjection& p) {
  for (int i = 0; i < p.n; ++i)
    if (p.part[i].lora_r > 0) return false;
  return true;
}

// Only where nothing is computed a second time: the tile kernels' results differ in their roundings.
bool short_attn(const LbStreamCtx* c, int Hq, int Hk, int hd, int rotation) {
  return c->may_split && c->plan_q == nullptr &&
         lb_attn_short_ok(c->n_seq, c->max_len, Hq, Hk, hd, rotation);
}

LbSmallGemm small_gemm(const LbProjection& p, int mode, const LbStreamCtx* c) {
  LbSmallGemm g = {};
  g.nparts = p.n;
  g.mode = mode;
  for (int i = 0; i < p.n; ++i) {
    g.B[i] = p.part[i].w;
    g.ldb[i] = p.part[i].ldw;
    g.ext[i] = p.part[i].n_out;
  }
  g.may_split = c->may_split;
  g.status = c->status;
  g.stream = c->stream;
  return g;
}

// y [T, p.width] = x · [W_0; W_1; ..]ᵀ
int proj_fwd(const LbProjection& p, const __nv_bfloat16* x, long long ldx, __nv_bfloat16* y, int T,
             __nv_bfloat16* const* ts, const LbStreamCtx* c, const void* const* bias = nullptr) {
  if (p.n > 1 && plain(p)) {
    LbSmallGemm g = small_gemm(p, kParallelN, c);
    double apart = 0.0;
    __nv_bfloat16* col = y;
    for (int i = 0; i < p.n; ++i) {
      g.C[i] = col;
      g.bias[i] = bias != nullptr ? bias[i] : nullptr;
      g.ldc[i] = p.width;
      col += p.part[i].n_out;
      apart += lb_gemm_tile_cost(T, p.part[i].n_out, p.part[i].k_in, 0, bias != nullptr);
    }
    g.A = x;
    g.lda = ldx;
    g.M = T;
    g.N = p.width;
    g.K = p.part[0].k_in;
    g.b_ready = 1;
    if (small_wins(&g, apart)) {
      t_fewer += p.n - 1;
      return lb_gemm_small(&g);
    }
  }
  LB_TRY(lora_fwd_products(p.part, p.n, x, ldx, T, ts, c));
  for (int i = 0; i < p.n; ++i) {
    LB_TRY(lin_fwd(p.part[i], x, ldx, y, p.width, T, ts[i], c, bias != nullptr ? bias[i] : nullptr, true));
    y += p.part[i].n_out;
  }
  return 0;
}

// h [T, I] = act(x · W_gateᵀ) * (x · W_upᵀ), with the two products in gu [T, 2I] (the one-launch form
// leaves gu unwritten unless it is to be kept).
int glu_proj_fwd(const LbBlockDesc* d, const __nv_bfloat16* x, __nv_bfloat16* gu, bool keep_gu,
                 __nv_bfloat16* h, int T, __nv_bfloat16* const* ts, const LbStreamCtx* c) {
  const LbProjection& p = d->gate_up;
  const int I = d->I;
  if (plain(p)) {
    LbSmallGemm g = small_gemm(p, kParallelN, c);
    if (p.n == 1) {  // one fused weight: its two halves
      g.nparts = 2;
      g.B[1] = static_cast<const __nv_bfloat16*>(p.part[0].w) + I * p.part[0].ldw;
      g.ldb[1] = p.part[0].ldw;
    }
    g.ext[0] = g.ext[1] = I;
    if (keep_gu) {
      g.C[0] = gu;
      g.C[1] = gu + I;
      g.ldc[0] = g.ldc[1] = 2 * I;
    }
    g.glu_h = h;
    g.ld_h = I;
    g.glu_kind = d->act_kind;
    g.A = x;
    g.lda = d->H;
    g.M = T;
    g.N = 2 * I;
    g.K = d->H;
    g.b_ready = 1;
    // On the CTA-pair kernel the activation costs the epilogue (6 us of the model) and saves a launch and
    // its passes over memory. With one fused weight and the products kept that is even up to some
    // thousand tokens (2048: 46.8 against 45.3 us, 4100: 71 against 68, 22627: 257 against 266).
    const bool pair = T >= 256 && I >= 256 && g.ldb[0] == g.ldb[1] && lb_gemm_use_2cta(-1) &&
                      (p.n == 2 || !keep_gu || T >= 8192);
    double other = 6.0;
    if (pair) {
      other += lb_gemm_tile_cost(T, 2 * I, d->H, 0, 0);
    } else {
      other += 6.0 * T * I / 5e6;   // the activation: a launch, three passes at 5 TB/s
      for (int i = 0; i < p.n; ++i) other += lb_gemm_tile_cost(T, p.part[i].n_out, d->H, 0, 0);
    }
    // (measured, small / pair: 520 x 3072 x 1024 25 / 29 us, 800 x 9728 x 2560 175 / 121, 1500 x 1152 x 768
    // 21 / 25, 6000 x 1152 x 768 48 / 39)
    if (small_wins(&g, other)) {
      t_fewer += p.n;
      return lb_gemm_small(&g);
    }
    if (pair) {
      t_fewer += p.n;
      return lb_gemm_glu_2cta(x, g.B[0], g.B[1], g.C[0], g.C[1], h, T, I, d->H, d->H, g.ldb[0], 2 * I,
                              I, d->act_kind, c->status, c->stream);
    }
  }
  LB_TRY(proj_fwd(p, x, d->H, gu, T, ts, c));
  return lb_glu_fwd(d->act_kind, gu, gu + I, 2 * I, h, I, T, I, c->stream);
}

// dx [T, k_in] = dy · [W_0; W_1; ..] (the parts' products added up in bf16) and dW_i += dy_iᵀ · x.
int proj_bwd(const LbProjection& p, const __nv_bfloat16* dy, const __nv_bfloat16* x,
             __nv_bfloat16* dx, int T, __nv_bfloat16* const* ts, __nv_bfloat16* us,
             const LbStreamCtx* c) {
  const int K = p.part[0].k_in;
  bool dx_done = false, dw_done = false;
  if (p.n > 1 && plain(p)) {
    double apart = 0.0, apart_w = 0.0;
    bool all_w = true;
    for (int i = 0; i < p.n; ++i) {
      apart += lb_gemm_tile_cost(T, K, p.part[i].n_out, 0, 0);
      apart_w += lb_gemm_tile_cost(p.part[i].n_out, K, T, 1, 0);
      all_w = all_w && p.part[i].wgrad != nullptr;
    }
    LbSmallGemm g = small_gemm(p, kParallelK, c);
    g.A = dy;
    g.lda = p.width;
    g.C[0] = dx;
    g.ldc[0] = K;
    g.M = T;
    g.N = K;
    g.K = p.width;
    g.b_mn = 1;
    g.b_ready = 1;
    if (small_wins(&g, apart)) {
      LB_TRY(lb_gemm_small(&g));
      t_fewer += p.n - 1;
      dx_done = true;
    }
    if (all_w) {
      LbSmallGemm w = small_gemm(p, kParallelM, c);
      w.A = dy;
      w.lda = p.width;
      w.B[0] = x;
      w.ldb[0] = K;
      for (int i = 0; i < p.n; ++i) {
        w.C[i] = p.part[i].wgrad;
        w.ldc[i] = K;
      }
      w.M = p.width;
      w.N = K;
      w.K = T;
      w.a_mn = w.b_mn = w.out_fp32 = 1;
      if (small_wins(&w, apart_w)) {
        LB_TRY(lb_gemm_small(&w));
        t_fewer += p.n - 1;
        dw_done = true;
      }
    }
  }
  for (int i = 0, col = 0; i < p.n; ++i) {
    const LbLinear& l = p.part[i];
    if (!dx_done) LB_TRY(lin_dgrad(l, dy + col, p.width, dx, T, i > 0, us, c));
    if (!dw_done) LB_TRY(lin_wgrad(l, dy + col, p.width, x, K, T, ts[i], us, c));
    col += l.n_out;
  }
  return 0;
}

int lin_fwd_launches(const LbLinear& l) { return l.lora_r > 0 ? 3 : 1; }

int lin_bwd_launches(const LbLinear& l, bool accumulate) {
  int n = l.wgrad != nullptr ? 1 : 0;
  if (l.lora_r > 0)
    n += 3 + (accumulate ? 1 : 0) + (l.lora_a_grad != nullptr) + (l.lora_b_grad != nullptr);
  else
    n += 1;
  return n;
}

// ---- token-sharded stream (tensor parallelism with sequence parallelism) ------------------------
// Running counters of one call. The double-buffering rule of the symmetric areas: use e touches
// half e & 1 and contains exactly one barrier; a half is rewritten two uses later, after the
// barrier of the use in between, which every peer joins only after its GEMM of use e is complete
// in stream order. A reduce-scatter half is read (its slots summed) right after the barrier of
// its use and rewritten two uses later under the same rule.
struct TpRun {
  const LbTpCtx* t;
  unsigned ag_epoch, ag_calls, rs_epoch, bar_epoch;
  explicit TpRun(const LbTpCtx* tp)
      : t(tp), ag_epoch(tp->ag_epoch), ag_calls(tp->ag_calls), rs_epoch(tp->rs_epoch),
        bar_epoch(tp->bar_epoch) {}
  // half of the publication area the next gathered GEMM uses: the producer of the shard may
  // write straight into it
  __nv_bfloat16* next_slot() const {
    return static_cast<__nv_bfloat16*>(t->ag_local[(ag_epoch + 1) & 1]);
  }
};

int tp_barrier(TpRun& r, const LbStreamCtx* c) {
  ++r.bar_epoch;
  return lb_device_barrier(r.t->pads, r.t->world, r.t->rank, r.bar_epoch, r.t->bar_limit_ns,
                           c->status, c->stream);
}

// y[Tp, N] (row stride ldy) = all_gather(shard)[Tp, K] · op(w); `x_all` [Tp, K] receives the
// gathered rows (own rows by a local copy, the peers' rows by the pull warps of the GEMM).
// op(w) = wᵀ for w [N, K] (b_mn 0) or w for w [K, N] (b_mn 1).
int tp_ag_gemm(TpRun& r, const __nv_bfloat16* shard, __nv_bfloat16* x_all, const LbLinear& l,
               int b_mn, __nv_bfloat16* y, long long ldy, int N, int K, const LbStreamCtx* c) {
  const LbTpCtx* t = r.t;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(c->stream);
  ++r.ag_epoch;
  ++r.ag_calls;
  const int half = r.ag_epoch & 1;
  __nv_bfloat16* slot = static_cast<__nv_bfloat16*>(t->ag_local[half]);
  const size_t bytes = (size_t)t->rows * K * 2;
  if (shard != slot &&
      cudaMemcpyAsync(slot, shard, bytes, cudaMemcpyDeviceToDevice, st) != cudaSuccess)
    return -11;
  if (cudaMemcpyAsync(x_all + (size_t)t->rank * t->rows * K, shard, bytes,
                      cudaMemcpyDeviceToDevice, st) != cudaSuccess)
    return -11;
  LB_TRY(tp_barrier(r, c));  // every shard is published
  return lb_gemm_bf16_ag(t->ag_peers[half], x_all, l.w, y, t->rows, t->world, t->rank, N, K, K,
                         l.ldw, ldy, b_mn, nullptr, t->ag_flags, t->ag_counter, r.ag_calls,
                         c->status, c->stream);
}

// out[rows, N] = reduce_scatter(a[Tp, K] · op(w)): every rank stores its partial rows into its
// own slot of the owner's area from the GEMM epilogue; the owner sums its slots after the barrier.
int tp_gemm_rs(TpRun& r, const __nv_bfloat16* a, long long lda, const LbLinear& l, int b_mn,
               __nv_bfloat16* out, int N, int K, const LbStreamCtx* c) {
  const LbTpCtx* t = r.t;
  ++r.rs_epoch;
  const int half = r.rs_epoch & 1;
  LB_TRY(lb_gemm_bf16_push16(a, l.w, t->rs_peers[half], t->world, t->rows, tp_tokens(t), N, K, lda,
                             l.ldw, N, 0, b_mn, 0, c->status, c->stream));
  LB_TRY(tp_barrier(r, c));  // every contribution has landed
  return lb_take_sum(t->rs_local[half], out, (long long)t->rows * N, t->world, c->stream);
}

bool tp_shape_ok(const LbBlockDesc* d, const LbStreamCtx* c, const LbTpCtx* t) {
  if (t->world < 2 || t->world > 8 || t->rank < 0 || t->rank >= t->world || t->rows <= 0)
    return false;
  if (c->T > tp_tokens(t) || !c->packed) return false;
  if (d->qkv.n != 1 || d->gate_up.n != 1) return false;
  for (int i = 0; i < 7; ++i) {
    const LbLinear* l = linear_at(d, i);
    if (l != nullptr && l->lora_r > 0) return false;
  }
  return true;
}

int block_fwd_tp(const LbBlockDesc* d, const LbStreamCtx* c, const LbBlockIO* io) {
  const LbTpCtx* t = io->tp;
  if (!tp_shape_ok(d, c, t)) return -3;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(c->stream);
  const int T = c->T, R = t->rows, Tp = tp_tokens(t);
  Arena arena(io->saved);
  const Saved s = carve_saved(d, Tp, R, io->residual != nullptr, arena);
  const int H = d->H, hd = d->hd, Nq = d->Hq * hd, Nk = d->Hk * hd, W = d->qkv.width, I = d->I;
  const __nv_bfloat16* branch = static_cast<const __nv_bfloat16*>(io->branch);
  const __nv_bfloat16* stream_in = io->residual != nullptr ? s.res1 : branch;
  __nv_bfloat16* out = static_cast<__nv_bfloat16*>(io->out);
  TpRun r(t);

  __nv_bfloat16* x1s = r.next_slot();
  LB_TRY(lb_rms_norm_fwd(branch, io->residual, d->ln1_w, x1s, s.res1, s.rstd1, R, H, d->eps,
                         d->w_off, c->stream));
  LB_TRY(tp_ag_gemm(r, x1s, s.x1, d->qkv.part[0], 0, s.qkv, W, W, H, c));
  LB_TRY(lb_qk_norm_rope_fwd(s.qkv, W, s.qkv + Nq, W, d->qk_norm ? d->qn_w : nullptr,
                             d->qk_norm ? d->kn_w : nullptr, c->cos, c->sin, c->pos, c->pos_i64, 1,
                             s.qr, Nq, s.kr, Nk, s.q_rstd, s.k_rstd, T, d->Hq, d->Hk, hd, d->eps,
                             d->w_off, d->qk_norm, c->stream));
  if (Tp > T &&  // rows that pad the stream to a multiple of the group size
      cudaMemsetAsync(s.o + (size_t)T * Nq, 0, (size_t)(Tp - T) * Nq * 2, st) != cudaSuccess)
    return -11;
  LB_TRY(lb_attn_fwd(s.qr, Nq, s.kr, Nk, s.qkv + Nq + Nk, W, c->seq_start, c->seq_end, c->plan_f,
                     c->cap_f, c->tile_f, s.o, Nq, s.lse, T, d->Hq, d->Hk, hd, d->softmax_scale,
                     d->causal, c->status, c->stream));
  LB_TRY(tp_gemm_rs(r, s.o, Nq, d->o_proj, 0, out, H, Nq, c));
  __nv_bfloat16* x2s = r.next_slot();
  LB_TRY(lb_rms_norm_fwd(out, stream_in, d->ln2_w, x2s, io->res_out, s.rstd2, R, H, d->eps,
                         d->w_off, c->stream));
  LB_TRY(tp_ag_gemm(r, x2s, s.x2, d->gate_up.part[0], 0, s.gu, 2 * I, 2 * I, H, c));
  LB_TRY(lb_glu_fwd(d->act_kind, s.gu, s.gu + I, 2 * I, s.h, I, Tp, I, c->stream));
  return tp_gemm_rs(r, s.h, I, d->down, 0, out, H, I, c);
}

int block_bwd_tp(const LbBlockDesc* d, const LbStreamCtx* c, const LbBlockIO* io) {
  const LbTpCtx* t = io->tp;
  if (!tp_shape_ok(d, c, t)) return -3;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(c->stream);
  const int T = c->T, R = t->rows, Tp = tp_tokens(t);
  const bool has_res = io->residual != nullptr;
  Arena sa(io->saved);
  const Saved s = carve_saved(d, Tp, R, has_res, sa);
  Arena wa(io->work);
  const Work w = carve_work(d, Tp, R, true, wa);
  const int H = d->H, hd = d->hd, Nq = d->Hq * hd, Nk = d->Hk * hd, W = d->qkv.width, I = d->I;
  const __nv_bfloat16* d_out = static_cast<const __nv_bfloat16*>(io->d_out);
  const __nv_bfloat16* stream_in =
      has_res ? s.res1 : static_cast<const __nv_bfloat16*>(io->branch);
  TpRun r(t);

  // ---- MLP: down is row-parallel (its output gradient is gathered), gate-up column-parallel
  // (its input gradient is reduced and scattered)
  LB_TRY(tp_ag_gemm(r, d_out, w.dy_all, d->down, 1, w.dh, I, I, H, c));
  LB_TRY(lin_wgrad(d->down, w.dy_all, H, s.h, I, Tp, nullptr, nullptr, c));
  LB_TRY(lb_glu_bwd(d->act_kind, w.dh, I, s.gu, s.gu + I, 2 * I, w.dgu, w.dgu + I, 2 * I, Tp, I,
                    c->stream));
  LB_TRY(tp_gemm_rs(r, w.dgu, 2 * I, d->gate_up.part[0], 1, w.dx2, H, 2 * I, c));
  LB_TRY(lin_wgrad(d->gate_up.part[0], w.dgu, 2 * I, s.x2, H, Tp, nullptr, nullptr, c));
  // the gradient of the stream after the attention branch: written where the next gathered GEMM
  // publishes from, and read again by the first norm's backward at the end of this call
  __nv_bfloat16* dres2 = r.next_slot();
  LB_TRY(lb_rms_norm_bwd(w.dx2, io->d_res_out, io->res_out, d->ln2_w, s.rstd2, dres2,
                         c->norm_scratch, d->ln2_wgrad, 1, 1, R, H, d->w_off, c->stream));
  // ---- attention
  LB_TRY(tp_ag_gemm(r, dres2, w.dres_all, d->o_proj, 1, w.dO, Nq, Nq, H, c));
  LB_TRY(lin_wgrad(d->o_proj, w.dres_all, H, s.o, Nq, Tp, nullptr, nullptr, c));
  if (Tp > T &&
      cudaMemsetAsync(w.dqkv + (size_t)T * W, 0, (size_t)(Tp - T) * W * 2, st) != cudaSuccess)
    return -11;
  LB_TRY(lb_attn_bwd(w.dO, Nq, s.qr, Nq, s.kr, Nk, s.qkv + Nq + Nk, W, s.o, Nq, s.lse, w.delta,
                     c->seq_start, c->seq_end, c->plan_q, c->cap_q, c->plan_kv, c->cap_kv, w.dqr, Nq,
                     w.dkr, Nk, w.dqkv + Nq + Nk, W, T, d->Hq, d->Hk, hd, d->softmax_scale,
                     d->causal, c->status, c->stream));
  {
    const bool want_dw = d->qk_norm && d->qn_wgrad != nullptr && d->kn_wgrad != nullptr;
    const bool direct = want_dw && d->kn_wgrad == d->qn_wgrad + hd;
    void* dw_out = !want_dw ? nullptr : (direct ? (void*)d->qn_wgrad : (void*)c->wg_tmp);
    LB_TRY(lb_qk_norm_rope_bwd(w.dqr, Nq, w.dkr, Nk, s.qkv, W, s.qkv + Nq, W,
                               d->qk_norm ? d->qn_w : nullptr, d->qk_norm ? d->kn_w : nullptr,
                               c->cos, c->sin, c->pos, c->pos_i64, 1, s.q_rstd, s.k_rstd, w.dqkv, W,
                               w.dqkv + Nq, W, d->qk_norm ? c->rope_scratch : nullptr, dw_out, 1,
                               direct ? 1 : 0, T, d->Hq, d->Hk, hd, d->w_off, d->qk_norm,
                               c->stream));
    if (want_dw && !direct) {
      LB_TRY(lb_colsum(c->wg_tmp, 1, hd, d->qn_wgrad, 1, 1, c->stream));
      LB_TRY(lb_colsum(c->wg_tmp + hd, 1, hd, d->kn_wgrad, 1, 1, c->stream));
    }
  }
  LB_TRY(tp_gemm_rs(r, w.dqkv, W, d->qkv.part[0], 1, w.dx1, H, W, c));
  LB_TRY(lin_wgrad(d->qkv.part[0], w.dqkv, W, s.x1, H, Tp, nullptr, nullptr, c));
  return lb_rms_norm_bwd(w.dx1, dres2, stream_in, d->ln1_w, s.rstd1, io->dx, c->norm_scratch,
                         d->ln1_wgrad, 1, 1, R, H, d->w_off, c->stream);
}

}  // namespace

extern "C" size_t lb_block_saved_bytes(const LbBlockDesc* d, int T, int has_residual,
                                       const LbTpCtx* tp) {
  Arena a(nullptr);
  if (tp != nullptr)
    carve_saved(d, tp_tokens(tp), tp->rows, has_residual, a);
  else
    carve_saved(d, T, T, has_residual, a);
  return a.off;
}

extern "C" size_t lb_block_work_bytes(const LbBlockDesc* d, int T, const LbTpCtx* tp) {
  Arena a(nullptr);
  if (tp != nullptr)
    carve_work(d, tp_tokens(tp), tp->rows, true, a);
  else
    carve_work(d, T, T, false, a);
  return a.off;
}

extern "C" int lb_block_fwd_launches(const LbBlockDesc* d, const LbStreamCtx* c, int has_residual,
                                     const LbTpCtx* tp) {
  (void)has_residual;
  if (tp != nullptr)  // two norms, rope, attention, glu; 2 gathered GEMMs (own-row copy, barrier,
    return 5 + 2 * 3 + 2 * 3;  // GEMM) and 2 reduced GEMMs (GEMM, barrier, take-and-clear)
  int n = 5;  // two norms, rope, attention, glu
  for (int i = 0; i < 7; ++i) {
    const LbLinear* l = linear_at(d, i);
    if (l != nullptr) n += lin_fwd_launches(*l);
  }
  (void)c;
  return n;
}

extern "C" int lb_block_bwd_launches(const LbBlockDesc* d, const LbStreamCtx* c,
                                     const LbTpCtx* tp) {
  (void)c;
  int n = 1 + 3 + 1 + 2;  // glu, attention (delta, dq, dkv), rope, norms
  const bool qk_sums = d->qk_norm && d->qn_wgrad != nullptr && d->kn_wgrad != nullptr;
  if (tp != nullptr) {
    n += (d->ln1_wgrad != nullptr) + (d->ln2_wgrad != nullptr);
    if (qk_sums) n += d->kn_wgrad == d->qn_wgrad + d->hd ? 1 : 3;
    n += 2 * 3 + 1 + 2 * 3;  // as in the forward, plus the copy of d_out into the publication area
    for (int i = 0; i < 7; ++i) {
      const LbLinear* l = linear_at(d, i);
      if (l != nullptr && l->wgrad != nullptr) n += 1;
    }
    return n;
  }
  n += d->ln1_wgrad != nullptr || d->ln2_wgrad != nullptr || qk_sums;   // sums of the partial rows
  for (int i = 0; i < 7; ++i) {
    const LbLinear* l = linear_at(d, i);
    if (l != nullptr) n += lin_bwd_launches(*l, (i == 1 || i == 2 || i == 5));
  }
  return n;
}

static int block_fwd(const LbBlockDesc* d, const LbStreamCtx* c, const LbBlockIO* io) {
  const int T = c->T;
  if (T <= 0) return 0;
  if (io->tp != nullptr) return block_fwd_tp(d, c, io);
  if (d->qkv.n < 1 || d->qkv.n > 3 || d->gate_up.n < 1 || d->gate_up.n > 2) return -3;
  if (d->qkv.width != (d->Hq + 2 * d->Hk) * d->hd || d->gate_up.width != 2 * d->I) return -3;
  Arena arena(io->saved);
  const Saved s = carve_saved(d, T, T, io->residual != nullptr, arena);
  const int H = d->H, hd = d->hd, Nq = d->Hq * hd, Nk = d->Hk * hd, W = d->qkv.width;
  const __nv_bfloat16* branch = static_cast<const __nv_bfloat16*>(io->branch);
  const __nv_bfloat16* stream_in = io->residual != nullptr ? s.res1 : branch;
  __nv_bfloat16* out = static_cast<__nv_bfloat16*>(io->out);

  // The first launch of a pass is ordered behind everything before it on the stream, weight updates
  // and events of other streams included; the others may start while the one in front of them runs
  // and read weights meanwhile.
  {
    const lb::PdlScope first(io->chained != 0);
    LB_TRY(lb_rms_norm_fwd(branch, io->residual, d->ln1_w, s.x1, s.res1, s.rstd1, T, H, d->eps,
                           d->w_off, c->stream));
  }
  const lb::PdlScope pdl(true);
  LB_TRY(proj_fwd(d->qkv, s.x1, H, s.qkv, T, s.ts, c));
  if (short_attn(c, d->Hq, d->Hk, hd, 1)) {
    ++t_fewer;
    LB_TRY(lb_attn_short(s.qkv, s.qkv + Nq, s.qkv + Nq + Nk, W, d->qk_norm ? d->qn_w : nullptr,
                         d->qk_norm ? d->kn_w : nullptr, c->cos, c->sin, c->pos, c->pos_i64, c->seq_start,
                         c->seq_end, c->plan_f, c->cap_f, s.o, Nq, T, c->n_seq, c->max_len, d->Hq, d->Hk, hd,
                         d->eps, d->w_off, d->softmax_scale, d->causal, c->stream));
  } else {
    LB_TRY(lb_qk_norm_rope_fwd(s.qkv, W, s.qkv + Nq, W, d->qk_norm ? d->qn_w : nullptr,
                               d->qk_norm ? d->kn_w : nullptr, c->cos, c->sin, c->pos, c->pos_i64, 1,
                               s.qr, Nq, s.kr, Nk, s.q_rstd, s.k_rstd, T, d->Hq, d->Hk, hd, d->eps,
                               d->w_off, d->qk_norm, c->stream));
    LB_TRY(lb_attn_fwd(s.qr, Nq, s.kr, Nk, s.qkv + Nq + Nk, W, c->seq_start, c->seq_end, c->plan_f,
                       c->cap_f, c->tile_f, s.o, Nq, s.lse, T, d->Hq, d->Hk, hd, d->softmax_scale,
                       d->causal, c->status, c->stream));
  }
  // attention branch output: staged in `out`, consumed by the second norm before the MLP writes there
  LB_TRY(lin_fwd(d->o_proj, s.o, Nq, out, H, T, s.ts[3], c));
  LB_TRY(lb_rms_norm_fwd(out, stream_in, d->ln2_w, s.x2, io->res_out, s.rstd2, T, H, d->eps,
                         d->w_off, c->stream));
  // without gradients nothing reads the two products again
  LB_TRY(glu_proj_fwd(d, s.x2, s.gu, c->plan_q != nullptr, s.h, T, s.ts + 4, c));
  return lin_fwd(d->down, s.h, d->I, out, H, T, s.ts[6], c);
}

static int block_bwd(const LbBlockDesc* d, const LbStreamCtx* c, const LbBlockIO* io) {
  const int T = c->T;
  if (T <= 0) return 0;
  if (io->tp != nullptr) return block_bwd_tp(d, c, io);
  const bool has_res = io->residual != nullptr;
  Arena sa(io->saved);
  const Saved s = carve_saved(d, T, T, has_res, sa);
  Arena wa(io->work);
  const Work w = carve_work(d, T, T, false, wa);
  const int H = d->H, hd = d->hd, Nq = d->Hq * hd, Nk = d->Hk * hd, W = d->qkv.width, I = d->I;
  const __nv_bfloat16* d_out = static_cast<const __nv_bfloat16*>(io->d_out);
  const __nv_bfloat16* stream_in =
      has_res ? s.res1 : static_cast<const __nv_bfloat16*>(io->branch);

  // ---- MLP
  LB_TRY(lin_dgrad(d->down, d_out, H, w.dh, T, false, w.us, c));
  // From the second launch on, as in the forward: 2 us less from launch to launch, which is what a step of
  // few tokens consists of (8 padded pairs on 28 layers of width 1024: 21.5 -> 19.4 ms together with
  // padding cleared by the attention kernels and the norms' sums at the end of the call, 1915 -> 1551
  // launches).
  const lb::PdlScope pdl(true);
  LB_TRY(lin_wgrad(d->down, d_out, H, s.h, I, T, s.ts[6], w.us, c));
  LB_TRY(lb_glu_bwd(d->act_kind, w.dh, I, s.gu, s.gu + I, 2 * I, w.dgu, w.dgu + I, 2 * I, T, I,
                    c->stream));
  LB_TRY(proj_bwd(d->gate_up, w.dgu, s.x2, w.dx2, T, s.ts + 4, w.us, c));
  // second norm: the gradient of its input is both the attention branch's and the stream's
  float* sums1 = c->norm_scratch + (size_t)lb_norm_bwd_partial_rows() * H;
  LB_TRY(lb_rms_norm_bwd(w.dx2, io->d_res_out, io->res_out, d->ln2_w, s.rstd2, w.dres2,
                         c->norm_scratch, nullptr, 1, 1, T, H, d->w_off, c->stream));
  // ---- attention
  LB_TRY(lin_dgrad(d->o_proj, w.dres2, H, w.dO, T, false, w.us, c));
  LB_TRY(lin_wgrad(d->o_proj, w.dres2, H, s.o, Nq, T, s.ts[3], w.us, c));
  LB_TRY(lb_attn_bwd(w.dO, Nq, s.qr, Nq, s.kr, Nk, s.qkv + Nq + Nk, W, s.o, Nq, s.lse, w.delta,
                     c->seq_start, c->seq_end, c->plan_q, c->cap_q, c->plan_kv, c->cap_kv, w.dqr, Nq,
                     w.dkr, Nk, w.dqkv + Nq + Nk, W, T, d->Hq, d->Hk, hd, d->softmax_scale,
                     d->causal, c->status, c->stream));
  const bool want_dw = d->qk_norm && d->qn_wgrad != nullptr && d->kn_wgrad != nullptr;
  LB_TRY(lb_qk_norm_rope_bwd(w.dqr, Nq, w.dkr, Nk, s.qkv, W, s.qkv + Nq, W,
                             d->qk_norm ? d->qn_w : nullptr, d->qk_norm ? d->kn_w : nullptr, c->cos,
                             c->sin, c->pos, c->pos_i64, 1, s.q_rstd, s.k_rstd, w.dqkv, W,
                             w.dqkv + Nq, W, d->qk_norm ? c->rope_scratch : nullptr, nullptr, 1, 0, T,
                             d->Hq, d->Hk, hd, d->w_off, d->qk_norm, c->stream));
  LB_TRY(proj_bwd(d->qkv, w.dqkv, s.x1, w.dx1, T, s.ts, w.us, c));
  LB_TRY(lb_rms_norm_bwd(w.dx1, w.dres2, stream_in, d->ln1_w, s.rstd1, io->dx, sums1, nullptr, 1, 1, T,
                         H, d->w_off, c->stream));
  // the norms' weight gradients out of their kernels' partial sums: one launch for all of them
  LbColsum sums[kMaxColsums];
  int n = 0;
  const int rows = lb_norm_bwd_rows(T, H);
  if (d->ln2_wgrad != nullptr) sums[n++] = {c->norm_scratch, rows, H, d->ln2_wgrad, nullptr, 0};
  if (d->ln1_wgrad != nullptr) sums[n++] = {sums1, rows, H, d->ln1_wgrad, nullptr, 0};
  if (want_dw)
    sums[n++] = {c->rope_scratch, lb_rope_bwd_rows(T, d->Hq, d->Hk, hd), 2 * hd, d->qn_wgrad,
                 d->kn_wgrad, hd};
  return lb_colsums(sums, n, c->stream);
}

extern "C" int lb_block_fwd(const LbBlockDesc* d, const LbStreamCtx* c, LbBlockIO* io) {
  t_fewer = 0;
  const int rc = block_fwd(d, c, io);
  io->fewer_launches = t_fewer;
  return rc;
}

extern "C" int lb_block_bwd(const LbBlockDesc* d, const LbStreamCtx* c, LbBlockIO* io) {
  t_fewer = 0;
  const int rc = block_bwd(d, c, io);
  io->fewer_launches = t_fewer;
  return rc;
}

// ---- encoder block ---------------------------------------------------------------------------
namespace {

struct EncSaved {
  __nv_bfloat16 *qkv, *o, *nr1, *y1, *u, *g, *nr2, *tmp;
  float *lse, *mean1, *rstd1, *mean2, *rstd2;
};

EncSaved carve_enc_saved(const LbEncoderDesc* d, int T, Arena& a) {
  EncSaved s{};
  const size_t t = (size_t)T;
  s.qkv = a.bf(t * d->qkv.width);
  s.o = a.bf(t * d->H);
  s.lse = a.f32(t * d->heads);
  s.nr1 = a.bf(t * d->H);
  s.y1 = a.bf(t * d->H);
  s.mean1 = a.f32(t);
  s.rstd1 = a.f32(t);
  s.u = a.bf(t * d->I);
  s.g = a.bf(t * d->I);
  s.nr2 = a.bf(t * d->H);
  s.mean2 = a.f32(t);
  s.rstd2 = a.f32(t);
  s.tmp = a.bf(t * d->H);
  return s;
}

struct EncWork {
  __nv_bfloat16 *dnr2, *dg, *du, *dy1, *dnr1, *dO, *dqkv;
  float* delta;
};

EncWork carve_enc_work(const LbEncoderDesc* d, int T, Arena& a) {
  EncWork w{};
  const size_t t = (size_t)T;
  w.dnr2 = a.bf(t * d->H);
  w.dy1 = a.bf(t * d->H);
  w.dnr1 = a.bf(t * d->H);
  const size_t mark = a.off;  // the MLP half is finished before the attention half starts
  w.dg = a.bf(t * d->I);
  w.du = a.bf(t * d->I);
  const size_t end = a.off;
  a.off = mark;
  w.dO = a.bf(t * d->H);
  w.dqkv = a.bf(t * d->qkv.width);
  w.delta = a.f32(t * d->heads);
  if (a.off < end) a.off = end;
  return w;
}

int enc_linear_bwd(const LbLinear& l, float* bgrad, const __nv_bfloat16* dy, const __nv_bfloat16* x,
                   __nv_bfloat16* dx, int T, const LbStreamCtx* c, int* n) {
  LB_TRY(lin_dgrad(l, dy, l.n_out, dx, T, false, nullptr, c));
  LB_TRY(lin_wgrad(l, dy, l.n_out, x, l.k_in, T, nullptr, nullptr, c));
  *n += 1 + (l.wgrad != nullptr);
  if (bgrad != nullptr) {
    LB_TRY(lb_bias_grad(dy, l.n_out, T, l.n_out, 0, 0, bgrad, nullptr, nullptr, c->stream));
    ++*n;
  }
  return 0;
}

bool enc_ok(const LbEncoderDesc* d) {
  return (d->qkv.n == 1 || d->qkv.n == 3) && d->qkv.width == 3 * d->H && d->heads * d->hd == d->H;
}

}  // namespace

extern "C" size_t lb_encoder_saved_bytes(const LbEncoderDesc* d, int T) {
  Arena a(nullptr);
  carve_enc_saved(d, T, a);
  return a.off;
}

extern "C" size_t lb_encoder_work_bytes(const LbEncoderDesc* d, int T) {
  Arena a(nullptr);
  carve_enc_work(d, T, a);
  return a.off;
}

extern "C" int lb_encoder_fwd(const LbEncoderDesc* d, const LbStreamCtx* c, LbBlockIO* io) {
  const int T = c->T, H = d->H, I = d->I, W = d->qkv.width;
  io->launches = 0;
  if (T <= 0) return 0;
  if (!enc_ok(d)) return -3;
  t_fewer = 0;
  Arena arena(io->saved);
  const EncSaved s = carve_enc_saved(d, T, arena);
  const __nv_bfloat16* x = static_cast<const __nv_bfloat16*>(io->branch);
  __nv_bfloat16* no_ts[3] = {nullptr, nullptr, nullptr};
  {  // as in block_fwd
    const lb::PdlScope first(io->chained != 0);
    LB_TRY(proj_fwd(d->qkv, x, H, s.qkv, T, no_ts, c, d->bias));
  }
  const lb::PdlScope pdl(true);
  if (short_attn(c, d->heads, d->heads, d->hd, 0)) {
    LB_TRY(lb_attn_short(s.qkv, s.qkv + H, s.qkv + 2 * H, W, nullptr, nullptr, nullptr, nullptr, nullptr, 0,
                         c->seq_start, c->seq_end, c->plan_f, c->cap_f, s.o, H, T, c->n_seq, c->max_len,
                         d->heads, d->heads, d->hd, 0.f, 0.f, d->softmax_scale, 0, c->stream));
  } else {
    LB_TRY(lb_attn_fwd(s.qkv, W, s.qkv + H, W, s.qkv + 2 * H, W, c->seq_start, c->seq_end, c->plan_f,
                       c->cap_f, c->tile_f, s.o, H, s.lse, T, d->heads, d->heads, d->hd,
                       d->softmax_scale, 0, c->status, c->stream));
  }
  LB_TRY(lin_fwd(d->o_proj, s.o, H, s.tmp, H, T, nullptr, c, d->bias[3]));
  LB_TRY(lb_layer_norm_fwd(s.tmp, x, d->ln1_w, d->ln1_b, s.y1, s.nr1, s.mean1, s.rstd1, T, H, d->eps,
                           c->stream));
  LB_TRY(lin_gelu_fwd(d->in, s.y1, H, s.u, c->plan_q != nullptr, s.g, I, T, c, d->bias[4]));
  LB_TRY(lin_fwd(d->out, s.g, I, s.tmp, H, T, nullptr, c, d->bias[5]));
  LB_TRY(lb_layer_norm_fwd(s.tmp, s.y1, d->ln2_w, d->ln2_b, io->out, s.nr2, s.mean2, s.rstd2, T, H,
                           d->eps, c->stream));
  io->launches += 7 + d->qkv.n - t_fewer;
  return 0;
}

extern "C" int lb_encoder_bwd(const LbEncoderDesc* d, const LbStreamCtx* c, LbBlockIO* io) {
  const int T = c->T, H = d->H, W = d->qkv.width;
  io->launches = 0;
  if (T <= 0) return 0;
  if (!enc_ok(d)) return -3;
  t_fewer = 0;
  int n = 0;
  Arena sa(io->saved), wa(io->work);
  const EncSaved s = carve_enc_saved(d, T, sa);
  const EncWork w = carve_enc_work(d, T, wa);
  const __nv_bfloat16* x = static_cast<const __nv_bfloat16*>(io->branch);
  const __nv_bfloat16* dy = static_cast<const __nv_bfloat16*>(io->d_out);
  __nv_bfloat16* dx = static_cast<__nv_bfloat16*>(io->dx);
  __nv_bfloat16* no_ts[3] = {nullptr, nullptr, nullptr};
  float* sums1 = c->norm_scratch + (size_t)lb_norm_bwd_partial_rows() * 2 * H;
  LB_TRY(lb_layer_norm_bwd(dy, nullptr, s.nr2, d->ln2_w, s.mean2, s.rstd2, w.dnr2, c->norm_scratch,
                           nullptr, 1, 1, T, H, c->stream));
  const lb::PdlScope pdl(true);
  LB_TRY(enc_linear_bwd(d->out, d->bias_grad[5], w.dnr2, s.g, w.dg, T, c, &n));
  LB_TRY(lb_gelu_bwd(w.dg, s.u, w.du, 1LL * T * d->I, c->stream));
  LB_TRY(enc_linear_bwd(d->in, d->bias_grad[4], w.du, s.y1, w.dy1, T, c, &n));
  LB_TRY(lb_add_bf16(w.dy1, w.dnr2, 1LL * T * H, c->stream));
  LB_TRY(lb_layer_norm_bwd(w.dy1, nullptr, s.nr1, d->ln1_w, s.mean1, s.rstd1, w.dnr1, sums1, nullptr, 1,
                           1, T, H, c->stream));
  LB_TRY(enc_linear_bwd(d->o_proj, d->bias_grad[3], w.dnr1, s.o, w.dO, T, c, &n));
  LB_TRY(lb_attn_bwd(w.dO, H, s.qkv, W, s.qkv + H, W, s.qkv + 2 * H, W, s.o, H, s.lse, w.delta,
                     c->seq_start, c->seq_end, c->plan_q, c->cap_q, c->plan_kv, c->cap_kv, w.dqkv, W,
                     w.dqkv + H, W, w.dqkv + 2 * H, W, T, d->heads, d->heads, d->hd,
                     d->softmax_scale, 0, c->status, c->stream));
  LB_TRY(proj_bwd(d->qkv, w.dqkv, x, dx, T, no_ts, nullptr, c));
  float* const* bg = d->bias_grad;
  if (bg[0] != nullptr || bg[1] != nullptr || bg[2] != nullptr) {
    const int parts = d->qkv.n;
    LB_TRY(lb_bias_grad(w.dqkv, W, T, d->qkv.part[0].n_out, parts == 3 ? H : 0, parts == 3 ? H : 0,
                        bg[0], bg[1], bg[2], c->stream));
    ++n;
  }
  LB_TRY(lb_add_bf16(dx, w.dnr1, 1LL * T * H, c->stream));
  // both norms' weight and bias gradients out of their kernels' partial sums
  LbColsum sums[2];
  int k = 0;
  const int rows = lb_norm_bwd_rows(T, H);
  if (d->ln2_wgrad != nullptr || d->ln2_bgrad != nullptr)
    sums[k++] = {c->norm_scratch, rows, 2 * H, d->ln2_wgrad, d->ln2_bgrad, H};
  if (d->ln1_wgrad != nullptr || d->ln1_bgrad != nullptr)
    sums[k++] = {sums1, rows, 2 * H, d->ln1_wgrad, d->ln1_bgrad, H};
  LB_TRY(lb_colsums(sums, k, c->stream));
  // norms; gelu, two additions; attention; input gradients of the projections
  n += 2 + (k > 0) + 3 + 3 + d->qkv.n;
  for (int i = 0; i < d->qkv.n; ++i) n += d->qkv.part[i].wgrad != nullptr;
  io->launches = n - t_fewer;
  return 0;
}
