// Varlen flash attention backward on tcgen05, without atomics: three launches.
//
//   delta     delta[h, t] = sum_d dO[t,h,d] * O[t,h,d]
//   dQ        one 256-thread CTA per (sequence, query tile, KV head), two CTAs per SM, walking KV
//             blocks of 64:
//               S = Q·Kᵀ, dP = dO·Vᵀ (TMEM) -> dS = P∘(dP − delta)·scale (bf16, written over the V
//               block in smem) -> dQ += dS·K
//   dK/dV     work item = (sequence, 128-row KV tile, KV head), walking (query block,
//             head) pairs through a 3-deep TMA ring, with Sᵀ/dPᵀ double-buffered in TMEM so the
//             score products of step i+1 run while step i is in the softmax-gradient math:
//               Sᵀ = K·Qᵀ, dPᵀ = V·dOᵀ (TMEM) -> Pᵀ, dSᵀ (bf16, smem) -> dV += Pᵀ·dO, dK += dSᵀ·Q
//             Sixteen warps do the math, one requests the loads, one issues the products; the grid
//             is persistent, and an item's loads run under the end of the one before it.
// Thread t owns accumulator row t % 128 and a half (dQ kernel, 256 threads) or a quarter (dK/dV
// kernel, 512 threads) of the 64 columns of a score block.
// The Q / dO / K / V tiles are loaded once by TMA and serve both as K-major operands (contraction
// over head_dim) and as MN-major operands (contraction over tokens); nothing is transposed in
// memory. Probabilities are recomputed from the forward's LSE.
//
// Counterpart of the flash_attn / varlen_attn backward used by the reference through autograd
// (lset/models/decoder/qwen3/attention.py:203-234).
#include "../common/api.h"
#include "../common/pdl.h"
#include "../common/ptx.cuh"
#include "../common/row.cuh"
#include "../common/tma_desc.h"
#include "attn_common.cuh"

namespace lb {
namespace {

using bf16 = __nv_bfloat16;

struct AttnBwdArgs {
  const int* seq_start;  // first token of each sequence
  const int* seq_end;    // one past its last token
  const int* plan;
  const float* lse;    // [Hq, T]
  const float* delta;  // [Hq, T]
  bf16* dQ;
  long long lddq;
  bf16* dK;
  long long lddk;
  bf16* dV;
  long long lddv;
  int T, Hq, Hk;
  float scale;       // softmax scale
  float scale_log2;  // scale * log2(e)
  int causal;
  int* status;
  int capacity;      // of the plan
  unsigned* counter; // its work counter (persistent kernel; see finish_grid)
};

// ------------------------------------------------------------------------------------ delta
template <int HD>
__global__ void __launch_bounds__(256)
    attn_delta_kernel(const bf16* __restrict__ dO, long long lddo, const bf16* __restrict__ O,
                      long long ldo, float* __restrict__ delta, AttnBwdArgs a) {
  const int T = a.T, Hq = a.Hq;
  pdl_wait();
  pdl_trigger();
  // the gradient rows of tokens outside every sequence are written by no other kernel
  clear_outside(a.plan, a.capacity, a.seq_start, a.seq_end, a.dQ, a.lddq, T, Hq * HD / 8);
  clear_outside(a.plan, a.capacity, a.seq_start, a.seq_end, a.dK, a.lddk, T, a.Hk * HD / 8);
  clear_outside(a.plan, a.capacity, a.seq_start, a.seq_end, a.dV, a.lddv, T, a.Hk * HD / 8);
  constexpr int LPH = HD / 8;
  constexpr int UPB = 256 / LPH;
  const int l = threadIdx.x % LPH;
  const long long units = 1LL * T * Hq;
  for (long long u0 = 1LL * blockIdx.x * UPB; u0 < units; u0 += 1LL * gridDim.x * UPB) {
    const long long u = u0 + threadIdx.x / LPH;
    float s = 0.f;
    long long tok = 0;
    int h = 0;
    if (u < units) {
      if (units <= 0xffffffffll) {   // (a 64-bit division is a third of the loop's instructions)
        tok = unsigned(u) / unsigned(Hq);
      } else {
        tok = u / Hq;
      }
      h = int(u - tok * Hq);
      float x[8], y[8];
      unpack8(ld16(dO + tok * lddo + h * HD + l * 8), x);
      unpack8(ld16(O + tok * ldo + h * HD + l * 8), y);
#pragma unroll
      for (int i = 0; i < 8; ++i) s += x[i] * y[i];
    }
#pragma unroll
    for (int o = LPH / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (u < units && l == 0) delta[1LL * h * T + tok] = s;
  }
}

__device__ __forceinline__ void ld_row32(uint32_t taddr, float (&s)[32]) {
  uint32_t t0[32];
  tmem_ld_32x32b_x32(taddr, t0);
  tmem_ld_wait();
#pragma unroll
  for (int c = 0; c < 32; ++c) s[c] = __uint_as_float(t0[c]);
}

// Write 32 values of one row into columns [32*half, 32*half+32) of a 128-row x 64-column bf16 tile
// stored K-major with the 128-byte swizzle.
__device__ __forceinline__ void st_half_row_bf16_swz(uint8_t* tile, int row, int half,
                                                     const float (&v)[32]) {
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint4 q;
    q.x = pack_bf16x2(v[c * 8 + 0], v[c * 8 + 1]);
    q.y = pack_bf16x2(v[c * 8 + 2], v[c * 8 + 3]);
    q.z = pack_bf16x2(v[c * 8 + 4], v[c * 8 + 5]);
    q.w = pack_bf16x2(v[c * 8 + 6], v[c * 8 + 7]);
    *reinterpret_cast<uint4*>(tile + swz128_offset(row, half * 4 + c)) = q;
  }
}

// 16-column variants for kernels whose threads own a quarter of a 64-column block.
__device__ __forceinline__ void ld_row16(uint32_t taddr, float (&s)[16]) {
  uint32_t t0[16];
  tmem_ld_32x32b_x16(taddr, t0);
  tmem_ld_wait();
#pragma unroll
  for (int c = 0; c < 16; ++c) s[c] = __uint_as_float(t0[c]);
}

// Write 16 values of one row into columns [16*quarter, 16*quarter+16) of a 128-row x 64-column
// bf16 tile stored K-major with the 128-byte swizzle.
__device__ __forceinline__ void st_quarter_row_bf16_swz(uint8_t* tile, int row, int quarter,
                                                        const float (&v)[16]) {
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    uint4 q;
    q.x = pack_bf16x2(v[c * 8 + 0], v[c * 8 + 1]);
    q.y = pack_bf16x2(v[c * 8 + 2], v[c * 8 + 3]);
    q.z = pack_bf16x2(v[c * 8 + 4], v[c * 8 + 5]);
    q.w = pack_bf16x2(v[c * 8 + 6], v[c * 8 + 7]);
    *reinterpret_cast<uint4*>(tile + swz128_offset(row, quarter * 2 + c)) = q;
  }
}

// Store NCOLS (a multiple of 16) accumulator columns of one row as bf16 to dst when `pred`.
template <int NCOLS>
__device__ __forceinline__ void store_acc_cols16(uint32_t taddr, bf16* dst, bool pred) {
#pragma unroll 1
  for (int c = 0; c < NCOLS / 16; ++c) {
    uint32_t o[16];
    tmem_ld_32x32b_x16(taddr + c * 16, o);
    tmem_ld_wait();
    if (pred) {
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        uint4 q;
        q.x = pack_bf16x2(__uint_as_float(o[8 * v + 0]), __uint_as_float(o[8 * v + 1]));
        q.y = pack_bf16x2(__uint_as_float(o[8 * v + 2]), __uint_as_float(o[8 * v + 3]));
        q.z = pack_bf16x2(__uint_as_float(o[8 * v + 4]), __uint_as_float(o[8 * v + 5]));
        q.w = pack_bf16x2(__uint_as_float(o[8 * v + 6]), __uint_as_float(o[8 * v + 7]));
        *reinterpret_cast<uint4*>(dst + c * 16 + v * 8) = q;
      }
    }
  }
}

// Store NCOLS accumulator columns (fp32, starting at taddr) of one row as bf16 to dst when `pred`.
template <int NCOLS>
__device__ __forceinline__ void store_acc_cols(uint32_t taddr, bf16* dst, bool pred) {
#pragma unroll 1
  for (int c = 0; c < NCOLS / 32; ++c) {
    uint32_t o[32];
    tmem_ld_32x32b_x32(taddr + c * 32, o);
    tmem_ld_wait();
    if (pred) {
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        uint4 q;
        q.x = pack_bf16x2(__uint_as_float(o[8 * v + 0]), __uint_as_float(o[8 * v + 1]));
        q.y = pack_bf16x2(__uint_as_float(o[8 * v + 2]), __uint_as_float(o[8 * v + 3]));
        q.z = pack_bf16x2(__uint_as_float(o[8 * v + 4]), __uint_as_float(o[8 * v + 5]));
        q.w = pack_bf16x2(__uint_as_float(o[8 * v + 6]), __uint_as_float(o[8 * v + 7]));
        *reinterpret_cast<uint4*>(dst + c * 32 + v * 8) = q;
      }
    }
  }
}

// Store one accumulator row (HD fp32 columns starting at taddr) as bf16 to dst when `pred`.
template <int HD>
__device__ __forceinline__ void store_acc_row(uint32_t taddr, bf16* dst, bool pred) {
#pragma unroll 1
  for (int c = 0; c < HD / 32; ++c) {
    uint32_t o[32];
    tmem_ld_32x32b_x32(taddr + c * 32, o);
    tmem_ld_wait();
    if (pred) {
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        uint4 q;
        q.x = pack_bf16x2(__uint_as_float(o[8 * v + 0]), __uint_as_float(o[8 * v + 1]));
        q.y = pack_bf16x2(__uint_as_float(o[8 * v + 2]), __uint_as_float(o[8 * v + 3]));
        q.z = pack_bf16x2(__uint_as_float(o[8 * v + 4]), __uint_as_float(o[8 * v + 5]));
        q.w = pack_bf16x2(__uint_as_float(o[8 * v + 6]), __uint_as_float(o[8 * v + 7]));
        *reinterpret_cast<uint4*>(dst + c * 32 + v * 8) = q;
      }
    }
  }
}

// ------------------------------------------------------------------------------------ dQ
constexpr int kBwdThreads = 256;

template <int HD>
struct DqCfg {
  static constexpr int PANELS = HD / 64;
  static constexpr int Q_BYTES = 128 * HD * 2;
  static constexpr int KV_BYTES = kAttnKvBlock * HD * 2;
  static constexpr int DS_BYTES = 128 * kAttnKvBlock * 2;
  // dS is written over the V block (V is dead once dP = dO·Vᵀ has completed) when it fits.
  static constexpr bool DS_IN_V = KV_BYTES >= DS_BYTES;
  static constexpr int SMEM_BYTES = 2 * Q_BYTES + 2 * KV_BYTES + (DS_IN_V ? 0 : DS_BYTES) + 1024 + 128;
  static constexpr int DQ_COL = 128;
  static constexpr int TMEM_COLS = (128 + HD) <= 256 ? 256 : 512;
};

template <int HD>
__global__ void __launch_bounds__(kBwdThreads)
    attn_dq_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmdO,
                   const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                   AttnBwdArgs a) {
  using C = DqCfg<HD>;
  pdl_wait();
  pdl_trigger();
  AttnPlanView plan{a.plan};
  if (int(blockIdx.x) >= plan.count()) return;
  const int b = plan.seq(blockIdx.x);
  const int qt = plan.tile(blockIdx.x);
  const int hk = blockIdx.y;
  const int G = a.Hq / a.Hk;
  const int QT = 128 / G;
  const int seq0 = a.seq_start[b];
  const int len = a.seq_end[b] - seq0;
  const int q0 = qt * QT;
  const int kv_end = a.causal ? min(len, q0 + QT) : len;
  const int nblk = (kv_end + kAttnKvBlock - 1) / kAttnKvBlock;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sQ = smem;
  uint8_t* sdO = sQ + C::Q_BYTES;
  uint8_t* sK = sdO + C::Q_BYTES;
  uint8_t* sV = sK + C::KV_BYTES;
  uint8_t* sdS = C::DS_IN_V ? sV : (sV + C::KV_BYTES);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + C::KV_BYTES + (C::DS_IN_V ? 0 : C::DS_BYTES));
  uint64_t* bar_q = bars;
  uint64_t* bar_kv = bars + 1;
  uint64_t* bar_s = bars + 2;
  uint64_t* bar_dq = bars + 3;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 4);

  const int tid = threadIdx.x;
  const int warp = warp_index();
  const int half = warp >> 2;  // which 32 of the 64 KV columns this thread handles
  auto load_kv = [&](int j) {
    mbar_expect_tx(bar_kv, 2 * C::KV_BYTES);
#pragma unroll
    for (int p = 0; p < C::PANELS; ++p) {
      tma_load_2d(sK + p * (kAttnKvBlock * 128), &tmK, bar_kv, hk * HD + p * 64,
                  seq0 + j * kAttnKvBlock);
      tma_load_2d(sV + p * (kAttnKvBlock * 128), &tmV, bar_kv, hk * HD + p * 64,
                  seq0 + j * kAttnKvBlock);
    }
  };
  // first loads before the TMEM allocation and the CTA barrier: their latency runs under the set-up
  if (tid == 0) {
    mbar_init(bar_q, 1);
    mbar_init(bar_kv, 1);
    mbar_init(bar_s, 1);
    mbar_init(bar_dq, 1);
    mbar_fence_init();
    mbar_expect_tx(bar_q, 2 * C::Q_BYTES);
    for (int g = 0; g < G; ++g)
#pragma unroll
      for (int p = 0; p < C::PANELS; ++p) {
        tma_load_2d(sQ + p * (128 * 128) + g * QT * 128, &tmQ, bar_q, (hk * G + g) * HD + p * 64,
                    seq0 + q0);
        tma_load_2d(sdO + p * (128 * 128) + g * QT * 128, &tmdO, bar_q, (hk * G + g) * HD + p * 64,
                    seq0 + q0);
      }
    load_kv(0);
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_row = tmem_base + (uint32_t((warp & 3) * 32) << 16);

  const int r = tid & 127;
  const int g = r / QT;
  const int qpos = q0 + r % QT;
  const bool row_valid = qpos < len;
  const long long tok = 1LL * seq0 + qpos;
  const int head = hk * G + g;
  const float lse2 = row_valid ? a.lse[1LL * head * a.T + tok] * kLog2eF : 0.f;
  const float dlt = row_valid ? a.delta[1LL * head * a.T + tok] : 0.f;
  constexpr uint32_t idesc_s = umma_idesc_bf16(128, kAttnKvBlock, 0, 0);
  constexpr uint32_t idesc_dq = umma_idesc_bf16(128, HD, 0, 1);
  bool failed = false;
  {
    const bool ok = mbar_wait(bar_q, 0);
    if (__syncthreads_or(!ok)) {
      report_status(a.status, kStatusTimeoutProducer);
      failed = true;
    }
  }
  // One CTA-wide barrier per KV block (before the dQ product is issued). Thread 0 alone waits for
  // the loads and for the dQ product that frees the K / V slot; every thread waits for the score
  // products itself; whether a wait ran out anywhere is agreed on at the barrier.
  for (int j = 0; j < nblk && !failed; ++j) {
    bool ok = true;
    if (warp == 0 && elect_one()) {
      ok = mbar_wait(bar_kv, j & 1);
      if (ok) {
        tc_fence_after();
        const uint32_t qa = smem_u32(sQ), da = smem_u32(sdO);
        const uint32_t ka = smem_u32(sK), va = smem_u32(sV);
#pragma unroll
        for (int ks = 0; ks < HD / 16; ++ks) {
          const uint32_t aoff = (ks / 4) * (128 * 128) + (ks % 4) * 32;
          const uint32_t boff = (ks / 4) * (kAttnKvBlock * 128) + (ks % 4) * 32;
          umma_bf16(tmem_base, umma_smem_desc(qa + aoff, 16, 1024),
                    umma_smem_desc(ka + boff, 16, 1024), idesc_s, ks > 0 ? 1u : 0u);
        }
#pragma unroll
        for (int ks = 0; ks < HD / 16; ++ks) {
          const uint32_t aoff = (ks / 4) * (128 * 128) + (ks % 4) * 32;
          const uint32_t boff = (ks / 4) * (kAttnKvBlock * 128) + (ks % 4) * 32;
          umma_bf16(tmem_base + 64, umma_smem_desc(da + aoff, 16, 1024),
                    umma_smem_desc(va + boff, 16, 1024), idesc_s, ks > 0 ? 1u : 0u);
        }
        umma_commit(bar_s);
      }
    }
    ok = ok && mbar_wait(bar_s, j & 1);
    tc_fence_after();
    float ds[32];
    {
      float s[32];
      ld_row32(tmem_row + half * 32, s);
      ld_row32(tmem_row + 64 + half * 32, ds);
      const int kv0 = j * kAttnKvBlock + half * 32;
#pragma unroll
      for (int c = 0; c < 32; ++c) {
        const int kvpos = kv0 + c;
        const bool valid = row_valid && kvpos < len && (!a.causal || kvpos <= qpos);
        const float p = valid ? exp2f(s[c] * a.scale_log2 - lse2) : 0.f;
        ds[c] = p * (ds[c] - dlt) * a.scale;
      }
    }
    // S and dP are complete (bar_s), so the V block may be overwritten by dS
    st_half_row_bf16_swz(sdS, r, half, ds);
    fence_proxy_async_smem();
    tc_fence_before();
    if (__syncthreads_or(!ok)) {
      report_status(a.status, kStatusTimeoutMma);
      failed = true;
      break;
    }
    if (warp == 0 && elect_one()) {
      tc_fence_after();
      const uint32_t sa = smem_u32(sdS);
      const uint32_t ka = smem_u32(sK);
#pragma unroll
      for (int ks = 0; ks < kAttnKvBlock / 16; ++ks)
        umma_bf16(tmem_base + C::DQ_COL, umma_smem_desc(sa + ks * 32, 16, 1024),
                  umma_smem_desc(ka + ks * 2048, kAttnKvBlock * 128, 1024), idesc_dq,
                  (j > 0 || ks > 0) ? 1u : 0u);
      umma_commit(bar_dq);
      // the K block and the dS / V slot are in use until this block's dQ product is done; a wait
      // that runs out here leaves the next block unloaded, and its wait then fails for everybody
      if (j + 1 < nblk) {
        if (mbar_wait(bar_dq, j & 1))
          load_kv(j + 1);
        else
          report_status(a.status, kStatusTimeoutMma);
      }
    }
  }
  if (!failed) {
    const bool ok = mbar_wait(bar_dq, (nblk - 1) & 1);
    if (__syncthreads_or(!ok)) {
      report_status(a.status, kStatusTimeoutMma);
      failed = true;
    }
  }
  if (!failed) {
    tc_fence_after();
    store_acc_cols<HD / 2>(tmem_row + C::DQ_COL + half * (HD / 2),
                           a.dQ + tok * a.lddq + head * HD + half * (HD / 2), row_valid);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem_base, C::TMEM_COLS);
}

// ------------------------------------------------------------------------------------ dK / dV
template <int HD>
struct DkvCfg {
  static constexpr int PANELS = HD / 64;
  static constexpr int KV_BYTES = 128 * HD * 2;  // resident K tile and V tile
  static constexpr int QB_BYTES = 64 * HD * 2;   // one query block of Q or dO
  static constexpr int QBUFS = 3;                // TMA ring depth for (Q, dO) blocks
  static constexpr int PT_BYTES = 128 * 64 * 2;
  static constexpr int STAT_BYTES = QBUFS * 128 * 4;   // lse and delta of a block's 64 queries
  static constexpr int SMEM_BYTES = 2 * KV_BYTES + 2 * QBUFS * QB_BYTES + 2 * PT_BYTES + STAT_BYTES +
                                    1024 /*align*/ + 256;
  // TMEM: two (Sᵀ, dPᵀ) buffers of 64 + 64 columns, then the dV and dK accumulators.
  static constexpr int DV_COL = 256;
  static constexpr int DK_COL = 256 + HD;
  static constexpr int TMEM_COLS = 512;
  static_assert(256 + 2 * HD <= 512, "head_dim too large for the dK/dV accumulators");
};

// Math thread t (of 512) owns accumulator row t % 128 and a quarter (t / 128) of the 64 columns of a
// score block. With 256 (two warps per scheduler) the softmax-gradient math of a step was bound by
// instruction latency, not by the tensor pipe. Loads and products have warps of their own: when
// thread 0 issued them between its own loads and stores, all others waited 3800 of the 5600 clocks
// of a step for its warp. What is left per step is the tensor work (four products of 128 x 64 x HD) and
// the chain scores -> math -> shared memory -> accumulation, overlapped over two steps.
// Measured (whole backward, us; products issued by thread 0 -> warps of their own -> persistent grid):
//   64 sequences of 16..64 and 64 of 128..512 tokens, 16/8 heads of 128   588 -> 484 -> 458
//   8 x 2048 tokens, 16/8 heads                                          1341 -> 972 -> 936
//   32 of 256..1024 tokens, 32/8 heads                                   1438 -> 1062 -> 1049
constexpr int kDkvMath = 512;
constexpr int kDkvThreads = kDkvMath + 64;

// A work item of the persistent grid: one 128-row KV tile (hk < 0: no more items), its first query
// block and its steps (query blocks x heads of the group).
struct DkvItem {
  int hk, seq0, len, kv0;
};
__device__ __forceinline__ int dkv_first(const DkvItem& t, int causal) {
  return causal ? t.kv0 / 64 : 0;
}
__device__ __forceinline__ int dkv_steps(const DkvItem& t, int causal, int G) {
  return ((t.len + 63) / 64 - dkv_first(t, causal)) * G;   // >= 1: the tile's rows are queries too
}

template <int HD>
__global__ void __launch_bounds__(kDkvThreads, 1)
    attn_dkv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmdO,
                    const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                    AttnBwdArgs a) {
  using C = DkvCfg<HD>;
  const int G = a.Hq / a.Hk;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sK = smem;
  uint8_t* sV = sK + C::KV_BYTES;
  uint8_t* sQ = sV + C::KV_BYTES;               // [QBUFS]
  uint8_t* sdO = sQ + C::QBUFS * C::QB_BYTES;   // [QBUFS]
  uint8_t* sPT = sdO + C::QBUFS * C::QB_BYTES;
  uint8_t* sdST = sPT + C::PT_BYTES;
  float* sStat = reinterpret_cast<float*>(sdST + C::PT_BYTES);  // [QBUFS][2][64]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sStat + C::STAT_BYTES / 4);
  uint64_t* bar_kv = bars;
  uint64_t* bar_q = bars + 1;     // [QBUFS] Q and dO of a step have landed
  uint64_t* bar_st = bars + 4;    // [QBUFS] its lse and delta are in place
  uint64_t* bar_e = bars + 7;     // [QBUFS] its accumulation products are complete: slot free
  uint64_t* bar_s = bars + 10;    // [2] scores of a step are in tensor memory
  uint64_t* bar_p = bars + 12;    // Pᵀ and dSᵀ of a step are in shared memory
  uint64_t* bar_acc = bars + 13;  // ... and have been read by its accumulation products
  uint64_t* bar_kve = bars + 14;  // the item's last scores are complete: K and V may be replaced
  uint64_t* work_full = bars + 15;   // [2]
  uint64_t* work_empty = bars + 17;  // [2]
  DkvItem* s_work = reinterpret_cast<DkvItem*>(bars + 20);  // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(s_work + 2);

  const int tid = threadIdx.x;
  const int warp = warp_index();
  const int lane = tid & 31;

  if (tid == kDkvMath) {
    mbar_init(bar_kv, 1);
    for (int i = 0; i < C::QBUFS; ++i) {
      mbar_init(&bar_q[i], 1);
      mbar_init(&bar_st[i], 32);
      mbar_init(&bar_e[i], 1);
    }
    mbar_init(&bar_s[0], 1);
    mbar_init(&bar_s[1], 1);
    mbar_init(bar_p, kDkvMath / 32);
    mbar_init(bar_acc, 1);
    mbar_init(bar_kve, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&work_full[i], 1);
      mbar_init(&work_empty[i], kDkvMath / 32 + 1);   // the math warps and the products' issuer
    }
    mbar_fence_init();
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();
  pdl_trigger();

  if (warp == kDkvMath / 32) {
    // -------------------------------------------------------------------- work items, loads
    // (the lanes agree on the waits before they go on to the next item: where one ran out in some
    // of them only, those would leave the loop whose shuffles the others take part in. A vote per
    // step took 0.5-1.5 % of the backward; within an item they meet behind the loop.)
    AttnPlanView plan{a.plan};
    const int total = plan.count() * a.Hk;
    int w = int(blockIdx.x), n = 0;   // n: steps so far, over all items
    bool ok = true;
    for (int it = 0; ok; ++it) {
      DkvItem t{-1, 0, 0, 0};
      if (w < total) {                // heads vary fastest; the first KV tiles have the most queries
        const int i = w / a.Hk;
        const int b = plan.seq(i);
        t.hk = w - i * a.Hk;
        t.seq0 = a.seq_start[b];
        t.len = a.seq_end[b] - t.seq0;
        t.kv0 = plan.tile(i) * 128;
      }
      const int slot = it & 1;
      ok = __all_sync(0xffffffffu, mbar_wait(&work_empty[slot], ((it >> 1) & 1) ^ 1u));
      if (ok && lane == 0) {
        s_work[slot] = t;
        mbar_arrive(&work_full[slot]);
      }
      if (!ok || t.hk < 0) break;
      // K and V of the item as soon as the last one's scores are complete: under its last math,
      // its accumulation products and its store
      ok = __all_sync(0xffffffffu, mbar_wait(bar_kve, (it & 1) ^ 1u));
      if (ok && elect_one()) {
        mbar_expect_tx(bar_kv, 2 * C::KV_BYTES);
#pragma unroll
        for (int p = 0; p < C::PANELS; ++p) {
          tma_load_2d(sK + p * (128 * 128), &tmK, bar_kv, t.hk * HD + p * 64, t.seq0 + t.kv0);
          tma_load_2d(sV + p * (128 * 128), &tmV, bar_kv, t.hk * HD + p * 64, t.seq0 + t.kv0);
        }
      }
      const int qb_start = dkv_first(t, a.causal), steps = dkv_steps(t, a.causal, G);
      for (int i = 0; i < steps && ok; ++i, ++n) {
        const int buf = n % C::QBUFS;
        ok = mbar_wait(&bar_e[buf], ((n / C::QBUFS) & 1) ^ 1u);
        if (!ok) break;
        const int qb = qb_start + i / G;
        const int head = t.hk * G + i % G;
        if (lane == 0) {
          mbar_expect_tx(&bar_q[buf], 2 * C::QB_BYTES);
#pragma unroll
          for (int p = 0; p < C::PANELS; ++p) {
            tma_load_2d(sQ + buf * C::QB_BYTES + p * (64 * 128), &tmQ, &bar_q[buf],
                        head * HD + p * 64, t.seq0 + qb * 64);
            tma_load_2d(sdO + buf * C::QB_BYTES + p * (64 * 128), &tmdO, &bar_q[buf],
                        head * HD + p * 64, t.seq0 + qb * 64);
          }
        }
        float* st = sStat + buf * 128;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int c = lane + 32 * h;
          const int qp = qb * 64 + c;
          const long long at = 1LL * head * a.T + t.seq0 + qp;
          st[c] = qp < t.len ? a.lse[at] * kLog2eF : 0.f;
          st[64 + c] = qp < t.len ? a.delta[at] : 0.f;
        }
        mbar_arrive(&bar_st[buf]);
      }
      // the next item is drawn when this one's last loads are out, three steps before its end: drawn
      // earlier it would wait here while other SMs run out of work
      unsigned drawn = 0;
      if (lane == 0) drawn = atomicAdd(a.counter, 1u);
      ok = __all_sync(0xffffffffu, ok);
      w = int(__shfl_sync(0xffffffffu, drawn, 0)) + int(gridDim.x);
    }
    if (!ok) {
      if (lane == 0) report_status(a.status, kStatusTimeoutProducer);
      const unsigned long long t0 = globaltimer_ns();   // copies in flight land meanwhile
      while (globaltimer_ns() - t0 < 200000ull) {
      }
    }
    __syncwarp();
  } else if (warp == kDkvMath / 32 + 1) {
    // -------------------------------------------------------------------- products
    if (elect_one()) {
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, 64, 0, 0);
      constexpr uint32_t idesc_acc = umma_idesc_bf16(128, HD, 0, 1);
      const uint64_t kd = umma_smem_desc(smem_u32(sK), 16, 1024);
      const uint64_t vd = umma_smem_desc(smem_u32(sV), 16, 1024);
      const uint64_t pd = umma_smem_desc(smem_u32(sPT), 16, 1024);
      const uint64_t sd = umma_smem_desc(smem_u32(sdST), 16, 1024);
      // Step i issues the scores of block i (Sᵀ = K·Qᵀ, dPᵀ = V·dOᵀ, into TMEM buffer i & 1, which
      // step i - 2's math has read) and the accumulation products of block i - 1.
      int n = 0;   // steps so far, over all items
      bool ok = true;
      for (int it = 0; ok; ++it) {
        const int slot = it & 1;
        ok = mbar_wait(&work_full[slot], (it >> 1) & 1);
        if (!ok) break;
        const DkvItem t = s_work[slot];
        mbar_arrive(&work_empty[slot]);
        if (t.hk < 0) break;
        const int steps = dkv_steps(t, a.causal, G);
        ok = mbar_wait(bar_kv, it & 1);
#pragma unroll 1
        for (int i = 0; i <= steps && ok; ++i) {
          if (i < steps) {
            const int buf = (n + i) % C::QBUFS;
            ok = mbar_wait(&bar_q[buf], ((n + i) / C::QBUFS) & 1);
            if (!ok) break;
            tc_fence_after();
            const uint64_t qd = umma_smem_desc(smem_u32(sQ + buf * C::QB_BYTES), 16, 1024);
            const uint64_t dd = umma_smem_desc(smem_u32(sdO + buf * C::QB_BYTES), 16, 1024);
            const uint32_t dcol = tmem_base + ((n + i) & 1) * 128;
#pragma unroll
            for (int ks = 0; ks < HD / 16; ++ks) {
              const int aoff = ((ks / 4) * (128 * 128) + (ks % 4) * 32) >> 4;
              const int boff = ((ks / 4) * (64 * 128) + (ks % 4) * 32) >> 4;
              umma_bf16(dcol, kd + aoff, qd + boff, idesc_s, ks > 0 ? 1u : 0u);
            }
#pragma unroll
            for (int ks = 0; ks < HD / 16; ++ks) {
              const int aoff = ((ks / 4) * (128 * 128) + (ks % 4) * 32) >> 4;
              const int boff = ((ks / 4) * (64 * 128) + (ks % 4) * 32) >> 4;
              umma_bf16(dcol + 64, vd + aoff, dd + boff, idesc_s, ks > 0 ? 1u : 0u);
            }
            umma_commit(&bar_s[(n + i) & 1]);
            if (i + 1 == steps) umma_commit(bar_kve);
          }
          if (i > 0) {
            const int j = i - 1, buf = (n + j) % C::QBUFS;
            ok = mbar_wait(bar_p, (n + j) & 1);
            if (!ok) break;
            tc_fence_after();
            const uint64_t qd = umma_smem_desc(smem_u32(sQ + buf * C::QB_BYTES), 64 * 128, 1024);
            const uint64_t dd = umma_smem_desc(smem_u32(sdO + buf * C::QB_BYTES), 64 * 128, 1024);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              umma_bf16(tmem_base + C::DV_COL, pd + ks * 2, dd + ks * (2048 >> 4), idesc_acc,
                        (j > 0 || ks > 0) ? 1u : 0u);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              umma_bf16(tmem_base + C::DK_COL, sd + ks * 2, qd + ks * (2048 >> 4), idesc_acc,
                        (j > 0 || ks > 0) ? 1u : 0u);
            umma_commit(bar_acc);
            umma_commit(&bar_e[buf]);
          }
        }
        n += steps;
      }
      if (!ok) report_status(a.status, kStatusTimeoutMma);
    }
    __syncwarp();
  } else {
    // -------------------------------------------------------------------- softmax gradient
    const int quarter = warp >> 2;  // which 16 of the 64 score columns this thread handles
    const uint32_t tmem_row = tmem_base + (uint32_t((warp & 3) * 32) << 16);
    const int r = tid & 127;
    int n = 0;   // steps so far, over all items
    for (int it = 0;; ++it) {
      const int slot = it & 1;
      bool ok = __all_sync(0xffffffffu, mbar_wait(&work_full[slot], (it >> 1) & 1));
      if (!ok) {
        if (lane == 0) report_status(a.status, kStatusTimeoutEpilogue);
        break;
      }
      const DkvItem t = s_work[slot];
      __syncwarp();
      if (lane == 0) mbar_arrive(&work_empty[slot]);
      if (t.hk < 0) break;
      const int qb_start = dkv_first(t, a.causal), steps = dkv_steps(t, a.causal, G);
      const int kvpos = t.kv0 + r, len = t.len;
      const bool row_valid = kvpos < len;
      for (int i = 0; i < steps; ++i, ++n) {
        const int sb = n & 1, buf = n % C::QBUFS;
        ok = mbar_wait(&bar_st[buf], (n / C::QBUFS) & 1) && mbar_wait(&bar_s[sb], (n >> 1) & 1);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        uint32_t t0[16], t1[16];
        tmem_ld_32x32b_x16(tmem_row + sb * 128 + quarter * 16, t0);
        tmem_ld_32x32b_x16(tmem_row + sb * 128 + 64 + quarter * 16, t1);
        tmem_ld_wait();
        float pt[16], dst[16];
        {
          const float* lse2 = sStat + buf * 128 + quarter * 16;
          const float* dl = lse2 + 64;
          const int qbase = (qb_start + i / G) * 64 + quarter * 16;
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            const int qp = qbase + c;
            const bool valid = row_valid && qp < len && (!a.causal || kvpos <= qp);
            const float p = valid ? exp2f(__uint_as_float(t0[c]) * a.scale_log2 - lse2[c]) : 0.f;
            pt[c] = p;
            dst[c] = p * (__uint_as_float(t1[c]) - dl[c]) * a.scale;
          }
        }
        if (n > 0) {
          // the previous step's products have read the Pᵀ / dSᵀ tiles
          ok = __all_sync(0xffffffffu, mbar_wait(bar_acc, (n - 1) & 1));
          if (!ok) break;
        }
        st_quarter_row_bf16_swz(sPT, r, quarter, pt);
        st_quarter_row_bf16_swz(sdST, r, quarter, dst);
        fence_proxy_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_p);
      }
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(bar_acc, (n - 1) & 1));
      if (ok) {
        tc_fence_after();
        const long long tok = 1LL * t.seq0 + kvpos;
        store_acc_cols16<HD / 4>(tmem_row + C::DV_COL + quarter * (HD / 4),
                                 a.dV + tok * a.lddv + t.hk * HD + quarter * (HD / 4), row_valid);
        store_acc_cols16<HD / 4>(tmem_row + C::DK_COL + quarter * (HD / 4),
                                 a.dK + tok * a.lddk + t.hk * HD + quarter * (HD / 4), row_valid);
        // (the next item's first products into these accumulators wait for bar_p, behind the reads)
        tc_fence_before();
      } else {
        if (lane == 0) report_status(a.status, kStatusTimeoutEpilogue);
        break;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem_base, C::TMEM_COLS);
  finish_grid(a.plan, a.capacity);
}

template <int HD>
int launch_bwd(const void* dO, long long lddo, const void* q, long long ldq, const void* k,
               long long ldk, const void* v, long long ldv, const void* o, long long ldo,
               float* delta, const int* plan_q, int cap_q, const int* plan_kv, int cap_kv,
               AttnBwdArgs a, cudaStream_t st) {
  const int G = a.Hq / a.Hk;
  const int QT = 128 / G;
  {
    constexpr int UPB = 256 / (HD / 8);
    long long grid = (1LL * a.T * a.Hq + UPB - 1) / UPB;
    const long long cap = 1LL * row_num_sms() * 16;
    if (grid > cap) grid = cap;
    a.plan = plan_q;
    a.capacity = cap_q;
    const int rc = launch_pdl(attn_delta_kernel<HD>, dim3(int(grid)), dim3(256), 0, st,
                              pdl_enabled(4LL * a.T * a.Hq * HD), 1, (const bf16*)dO, lddo, (const bf16*)o,
                              ldo, delta, a);
    if (rc) return rc;
  }
  CUtensorMap tmQ, tmdO, tmK, tmV;
  int rc;
  // dQ kernel: Q / dO tiles of QT tokens per head, K / V blocks of 64.
  if ((rc = make_tmap_2d(&tmQ, q, 2, (uint64_t)a.Hq * HD, a.T, (uint64_t)ldq * 2, 64, QT, true))) return rc;
  if ((rc = make_tmap_2d(&tmdO, dO, 2, (uint64_t)a.Hq * HD, a.T, (uint64_t)lddo * 2, 64, QT, true))) return rc;
  if ((rc = make_tmap_2d(&tmK, k, 2, (uint64_t)a.Hk * HD, a.T, (uint64_t)ldk * 2, 64, 64, true))) return rc;
  if ((rc = make_tmap_2d(&tmV, v, 2, (uint64_t)a.Hk * HD, a.T, (uint64_t)ldv * 2, 64, 64, true))) return rc;
  {
    using C = DqCfg<HD>;
    auto kern = attn_dq_kernel<HD>;
    static bool configured = false;
    if (!configured) {
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES) !=
          cudaSuccess)
        return -10;
      configured = true;
    }
    a.plan = plan_q;
    rc = launch_pdl(kern, dim3(cap_q, a.Hk), dim3(kBwdThreads), C::SMEM_BYTES, st, pdl_enabled(), 1,
                    tmQ, tmdO, tmK, tmV, a);
    if (rc) return rc;
  }
  // dK/dV kernel: resident K / V tiles of 128 rows, Q / dO blocks of 64 tokens.
  if ((rc = make_tmap_2d(&tmQ, q, 2, (uint64_t)a.Hq * HD, a.T, (uint64_t)ldq * 2, 64, 64, true))) return rc;
  if ((rc = make_tmap_2d(&tmdO, dO, 2, (uint64_t)a.Hq * HD, a.T, (uint64_t)lddo * 2, 64, 64, true))) return rc;
  if ((rc = make_tmap_2d(&tmK, k, 2, (uint64_t)a.Hk * HD, a.T, (uint64_t)ldk * 2, 64, 128, true))) return rc;
  if ((rc = make_tmap_2d(&tmV, v, 2, (uint64_t)a.Hk * HD, a.T, (uint64_t)ldv * 2, 64, 128, true))) return rc;
  {
    using C = DkvCfg<HD>;
    auto kern = attn_dkv_kernel<HD>;
    static bool configured = false;
    if (!configured) {
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES) !=
          cudaSuccess)
        return -10;
      configured = true;
    }
    a.plan = plan_kv;
    a.capacity = cap_kv;
    a.counter = reinterpret_cast<unsigned*>(const_cast<int*>(plan_kv)) + 1 + 2 * cap_kv;
    const long long upper = 1LL * cap_kv * a.Hk;
    const int grid = int(upper < row_num_sms() ? upper : row_num_sms());
    return launch_pdl(kern, dim3(grid), dim3(kDkvThreads), C::SMEM_BYTES, st, pdl_enabled(), 1, tmQ,
                      tmdO, tmK, tmV, a);
  }
}

}  // namespace
}  // namespace lb

using namespace lb;

// plan_q: tiles of 128 / (Hq/Hk) tokens; plan_kv: tiles of 128 tokens. delta: [Hq, T] scratch.
extern "C" int lb_attn_bwd(const void* dO, long long lddo, const void* q, long long ldq,
                           const void* k, long long ldk, const void* v, long long ldv,
                           const void* o, long long ldo, const float* lse, float* delta,
                           const int* seq_start, const int* seq_end, const int* plan_q, int cap_q,
                           const int* plan_kv,
                           int cap_kv, void* dq, long long lddq, void* dk, long long lddk, void* dv,
                           long long lddv, int T, int Hq, int Hk, int hd, float softmax_scale,
                           int causal, int* status, void* stream) {
  if (T <= 0) return 0;
  if (Hk <= 0 || Hq % Hk != 0) return -3;
  const int G = Hq / Hk;
  if (G != 1 && G != 2 && G != 4 && G != 8) return -3;
  if ((lddo | ldq | ldk | ldv | ldo | lddq | lddk | lddv) & 7) return -3;
  AttnBwdArgs a{seq_start, seq_end, nullptr, lse, delta, (bf16*)dq, lddq, (bf16*)dk, lddk, (bf16*)dv, lddv,
                T, Hq, Hk, softmax_scale, softmax_scale * kLog2eF, causal, status, 0, nullptr};
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (hd != 128 && hd != 64) return -3;
  if (hd == 128)
    return launch_bwd<128>(dO, lddo, q, ldq, k, ldk, v, ldv, o, ldo, delta, plan_q, cap_q, plan_kv,
                           cap_kv, a, st);
  if (hd == 64)
    return launch_bwd<64>(dO, lddo, q, ldq, k, ldk, v, ldv, o, ldo, delta, plan_q, cap_q, plan_kv,
                          cap_kv, a, st);
  return -3;
}
