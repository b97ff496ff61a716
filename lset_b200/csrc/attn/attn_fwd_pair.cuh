// Varlen flash attention forward for head dims 64 and 128: two query tiles per CTA.
//
// What bounds it: per 128 x 128 block of scores the two products take 1024 tensor clocks at
// head dim 128 and the 16384 exponentials 1024 clocks of the SM's 16-a-clock unit, so neither may
// wait for the other. A kernel in which the same 128 threads wait for the score product, do the
// softmax and then wait for P·V (attn_fwd_kernel in attn_fwd.cu, two CTAs per SM) spends most of its
// time in those waits. Here the roles are separate warps and one CTA (one per SM) works on two query
// tiles of one sequence and KV head, which share every K and V tile (the arrangement published for
// FlashAttention-4, with its rescale only where the maximum rose by more than 2^8):
//
//   warps 0-3   softmax of tile 0 (thread = row)      warps 4-7   softmax of tile 1
//   warp 8      work items, TMA loads                 warp 9      tcgen05.mma issuer
//
// While one tile's softmax runs, the tensor core works on the other tile's products. K and V come
// in blocks of 128 tokens through a ring of four slots (K, V, K, V). Scores stay in tensor memory;
// P (bf16) replaces the first half of its scores there and is read by the second product from
// tensor memory, so shared memory only feeds K and V. Scores are masked only in blocks that the
// sequence end or the diagonal crosses, and of a tile's last block only the 32-column chunks it
// needs are computed. Warp 8 draws the next work item and looks it up while the current one is
// being worked on; the others find it in shared memory.
//
// Measured on a B200 (us; one-tile kernel with two CTAs per SM before -> this kernel):
//   10 x 4096 tokens, 16/8 heads of 128, causal     1584 -> 741 (930 TFLOP/s), bidirectional 1355
//   128 sequences of 128..512, same heads           266  -> 207
//   64 of 16..64 and 64 of 128..512, same heads     151  -> 127
// The short ones pay per work item: its first products and its store overlap with nothing. Where most
// sequences fit in one tile the one-tile kernel is faster (AttnPlan._one_tile).
//
// Tensor memory: S0 | S1 | O0 | O1, 128 columns each.
#pragma once

#include "../common/pdl.h"
#include "../common/ptx.cuh"
#include "attn_common.cuh"

namespace lb {
namespace {

constexpr int kPairBlock = 128;     // KV tokens per block
constexpr int kPairThreads = 320;
constexpr int kPairSlots = 4;       // K / V slots

struct AttnPairArgs {
  const int* seq_start;
  const int* seq_end;
  const int* plan;        // tiles of 2 * (128 / G) tokens
  int capacity;
  unsigned* counter;      // work items past the first wave; finish_grid puts it back to zero
  __nv_bfloat16* O;
  long long ldo;
  float* lse;             // [Hq, T]
  int T, Hq, Hk;
  float scale_log2;       // > 0: the maximum is taken before the scaling
  int negate_q;           // the softmax scale is negative: scores of -Q
  int causal;
  int* status;
};

template <int HD>
struct PairCfg {
  static constexpr int PANELS = HD / 64;
  static constexpr int PANEL_BYTES = 128 * 128;
  static constexpr int Q_BYTES = 128 * HD * 2;         // one tile
  static constexpr int SLOT_BYTES = kPairBlock * HD * 2;
  // per softmax warp: 32 rows x 32 bf16 columns of O on their way to global memory (rows 80 bytes
  // apart: no bank conflicts for one row per lane nor for four lanes per row)
  static constexpr int OUT_BYTES = 32 * 80;
  static constexpr int SMEM_BYTES =
      2 * Q_BYTES + kPairSlots * SLOT_BYTES + 8 * OUT_BYTES + 1024 + 256;
  static constexpr int TMEM_COLS = 512;
  static constexpr int S_COL = 0, O_COL = 256;
};

__device__ __forceinline__ float ex2_(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float max3_(float a, float b, float c) {
  float y;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
  return y;
}
// Two fp32 values in one 64-bit register pair.
__device__ __forceinline__ unsigned long long pair_(float lo, float hi) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ float2 unpair_(unsigned long long v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
__device__ __forceinline__ unsigned long long add2_(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long mul2_(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// Waits for the tensor-memory loads of this thread; the registers pass through it, so that nothing
// that uses them is moved in front of it while a load issued earlier is still in flight.
__device__ __forceinline__ void tmem_ld_wait_for(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]),
                 "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
                 "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]),
                 "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
                 "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]),
                 "+r"(r[30]), "+r"(r[31])
               :
               : "memory");
}

// Bounded wait (kWaitLimitNs) in few instructions: there are a dozen of them in the kernel, and its
// code is fetched through an instruction cache that the softmax alone nearly fills.
__device__ __forceinline__ bool pair_wait(uint64_t* bar, uint32_t parity) {
  if (mbar_try_wait(bar, parity)) return true;
  auto now = [] {
    uint32_t t;
    asm volatile("mov.u32 %0, %globaltimer_lo;" : "=r"(t));
    return t;
  };
  const uint32_t t0 = now();
  do {
    if (mbar_try_wait(bar, parity)) return true;
  } while (now() - t0 < uint32_t(kWaitLimitNs));
  return false;
}

// A work item: two adjacent query tiles of one sequence and KV head (hk < 0: no more items).
struct PairItem {
  int hk, seq0, len, q0;
};
// KV tokens that tile k of the item sees (0: the tile lies behind the sequence).
__device__ __forceinline__ int pair_kv_end(const PairItem& t, int k, int QT, int causal) {
  const int q0 = t.q0 + k * QT;
  return q0 < t.len ? (causal ? min(t.len, q0 + QT) : t.len) : 0;
}
__device__ __forceinline__ int pair_blocks(int kv_end) {
  return (kv_end + kPairBlock - 1) / kPairBlock;
}
// 32-column chunks of block j that a tile ending at kv_end needs.
__device__ __forceinline__ int pair_chunks(int kv_end, int j) {
  return min(4, (kv_end - j * kPairBlock + 31) / 32);
}

template <int HD>
__global__ void __launch_bounds__(kPairThreads, 1)
    attn_fwd_pair_kernel(const __grid_constant__ CUtensorMap tmQ,
                         const __grid_constant__ CUtensorMap tmK,
                         const __grid_constant__ CUtensorMap tmV, AttnPairArgs a) {
  using C = PairCfg<HD>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sQ = smem;
  uint8_t* sKV = smem + 2 * C::Q_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sKV + kPairSlots * C::SLOT_BYTES);
  uint64_t* q_full = bars;
  uint64_t* q_empty = bars + 1;
  uint64_t* kv_full = bars + 2;                 // [4]
  uint64_t* kv_empty = bars + 6;                // [4]
  uint64_t* s_full = bars + 10;                 // [2]
  uint64_t* p_full = bars + 12;                 // [2]
  uint64_t* o_full = bars + 14;                 // [2]
  uint64_t* work_full = bars + 16;              // [2]
  uint64_t* work_empty = bars + 18;             // [2]
  PairItem* s_work = reinterpret_cast<PairItem*>(bars + 20);  // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(s_work + 2);
  uint8_t* sOut = reinterpret_cast<uint8_t*>(bars) + 256;

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  const int G = a.Hq / a.Hk;
  const int QT = 128 / G;               // a power of two, as G
  const int qt_shift = 31 - __clz(QT);

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    mbar_init(q_empty, 1);
    for (int i = 0; i < kPairSlots; ++i) {
      mbar_init(&kv_full[i], 1);
      mbar_init(&kv_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 4);       // one arrival per softmax warp of the tile
      mbar_init(&o_full[i], 1);
      mbar_init(&work_full[i], 1);
      mbar_init(&work_empty[i], 9);   // eight softmax warps and the MMA issuer
    }
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (warp == 9) {
    tmem_alloc(tmem_slot, C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();
  pdl_trigger();

  if (warp == 8) {
    // -------------------------------------------------------------------- work items, loads
    if (elect_one()) {
      // Heads vary fastest, tiles run from the last to the first: under a causal mask the longest
      // items of a sequence come first.
      AttnPlanView plan{a.plan};
      const int tiles = plan.count();
      const int total = tiles * a.Hk;
      auto decode = [&](int w) {
        PairItem t{-1, 0, 0, 0};
        if (w < total) {
          const int row = w / a.Hk, i = tiles - 1 - row;
          const int b = plan.seq(i);
          t.hk = w - row * a.Hk;
          t.seq0 = a.seq_start[b];
          t.len = a.seq_end[b] - t.seq0;
          t.q0 = plan.tile(i) * (2 * QT);
        }
        return t;
      };
      int n = 0;          // K and V tiles loaded so far
      bool ok = true;
      int w = int(blockIdx.x);
#pragma unroll 1
      for (int it = 0; ok; ++it) {
        const PairItem t = decode(w);
        const int slot = it & 1;
        if (!pair_wait(&work_empty[slot], ((it >> 1) & 1) ^ 1u)) {
          report_status(a.status, kStatusTimeoutProducer);
          break;
        }
        s_work[slot] = t;
        mbar_arrive(&work_full[slot]);
        if (t.hk < 0) break;
        if (!pair_wait(q_empty, (it & 1) ^ 1u)) {
          report_status(a.status, kStatusTimeoutProducer);
          break;
        }
        const int kv1 = pair_kv_end(t, 1, QT, a.causal);
        const int nmax = max(pair_blocks(pair_kv_end(t, 0, QT, a.causal)), pair_blocks(kv1));
        const int ntile = kv1 > 0 ? 2 : 1;
        mbar_expect_tx(q_full, ntile * C::Q_BYTES);
        // Q of tile 0, K, Q of tile 1, V; then K, V of every further block
#pragma unroll 1
        for (int c = 0; c < 2 * nmax; ++c) {
          if (c < ntile) {
#pragma unroll 1
            for (int g = 0; g < G; ++g)
#pragma unroll
              for (int p = 0; p < C::PANELS; ++p)
                tma_load_2d(sQ + c * C::Q_BYTES + p * C::PANEL_BYTES + g * QT * 128, &tmQ, q_full,
                            (t.hk * G + g) * HD + p * 64, t.seq0 + t.q0 + c * QT);
          }
          const int s = n & (kPairSlots - 1);
          ok = pair_wait(&kv_empty[s], ((n / kPairSlots) & 1) ^ 1u);
          if (!ok) break;
          mbar_expect_tx(&kv_full[s], C::SLOT_BYTES);
#pragma unroll
          for (int p = 0; p < C::PANELS; ++p)
            tma_load_2d(sKV + s * C::SLOT_BYTES + p * C::PANEL_BYTES, (c & 1) ? &tmV : &tmK,
                        &kv_full[s], t.hk * HD + p * 64, t.seq0 + (c >> 1) * kPairBlock);
          ++n;
        }
        if (!ok) report_status(a.status, kStatusTimeoutProducer);
        // the next item is drawn when this one's last loads are out: drawn earlier it would wait
        // here while other SMs run out of work
        w = int(atomicAdd(a.counter, 1u)) + int(gridDim.x);
      }
      if (!ok) {
        const unsigned long long t0 = globaltimer_ns();   // copies in flight land meanwhile
        while (globaltimer_ns() - t0 < 200000ull) {
        }
      }
    }
    __syncwarp();
  } else if (warp == 9) {
    // -------------------------------------------------------------------- MMA issuer
    if (elect_one()) {
      constexpr uint32_t idesc_o = umma_idesc_bf16(128, HD, 0, 1);
      // One copy of each product's instructions for both tiles: the kernel's code is fetched through
      // an instruction cache (see pair_wait).
      int n = 0;                  // KV blocks consumed so far
      int pv0 = 0, pv1 = 0;       // P·V products issued so far, per tile
      bool ok = true;
      for (int it = 0; ok; ++it) {
        const int slot = it & 1;
        ok = pair_wait(&work_full[slot], (it >> 1) & 1);
        if (!ok) break;
        const PairItem t = s_work[slot];
        mbar_arrive(&work_empty[slot]);
        if (t.hk < 0) break;
        const int kv_end0 = pair_kv_end(t, 0, QT, a.causal);
        const int kv_end1 = pair_kv_end(t, 1, QT, a.causal);
        const int nblk0 = pair_blocks(kv_end0), nblk1 = pair_blocks(kv_end1);
        const int nmax = max(nblk0, nblk1);
        ok = pair_wait(q_full, it & 1);
        // Step j issues P·V of block j - 1 and the scores of block j, tile by tile.
#pragma unroll 1
        for (int j = 0; j <= nmax && ok; ++j) {
          const int ck = 2 * (n + j), cv = ck - 1;   // ring positions of K_j and V_{j-1}
          if (j > 0) ok = pair_wait(&kv_full[cv & 3], (cv >> 2) & 1);
          if (ok && j < nmax) ok = pair_wait(&kv_full[ck & 3], (ck >> 2) & 1);
          if (!ok) break;
#pragma unroll 1
          for (int k = 0; k < 2; ++k) {
            const int nblk = k ? nblk1 : nblk0, kv_end = k ? kv_end1 : kv_end0;
            int pv = k ? pv1 : pv0;
            const uint32_t tS = tmem_base + C::S_COL + k * 128;
            if (j > 0 && j <= nblk) {
              ok = pair_wait(&p_full[k], pv & 1);
              if (!ok) break;
              tc_fence_after();
              const uint32_t va = smem_u32(sKV + (cv & 3) * C::SLOT_BYTES);
              const int steps = 2 * pair_chunks(kv_end, j - 1);
              const uint64_t vd = umma_smem_desc(va, C::PANEL_BYTES, 1024);
              const uint32_t tO = tmem_base + C::O_COL + k * 128;
              umma_bf16_ts(tO, tS, vd, idesc_o, j > 1 ? 1u : 0u);
#pragma unroll
              for (int ks = 1; ks < kPairBlock / 16; ++ks)
                if (ks < steps) umma_bf16_ts(tO, tS + ks * 8, vd + ks * (2048 >> 4), idesc_o, 1u);
              umma_commit(&o_full[k]);
              ++pv;
              if (k) pv1 = pv; else pv0 = pv;
            }
            if (j < nblk) {
              // the scores replace P of this tile's last product, which has to be complete
              if (pv > 0) ok = pair_wait(&o_full[k], (pv - 1) & 1);
              if (!ok) break;
              tc_fence_after();
              const uint32_t qa = smem_u32(sQ + k * C::Q_BYTES);
              const uint32_t ka = smem_u32(sKV + (ck & 3) * C::SLOT_BYTES);
              const uint32_t idesc_s = umma_idesc_bf16(128, 32 * pair_chunks(kv_end, j), 0, 0) |
                                       (uint32_t(a.negate_q) << 13);
              const uint64_t qd = umma_smem_desc(qa, 16, 1024), kd = umma_smem_desc(ka, 16, 1024);
#pragma unroll
              for (int ks = 0; ks < HD / 16; ++ks) {
                const int off = ((ks >> 2) * C::PANEL_BYTES + (ks & 3) * 32) >> 4;
                umma_bf16(tS, qd + off, kd + off, idesc_s, ks > 0 ? 1u : 0u);
              }
              umma_commit(&s_full[k]);
            }
          }
          if (!ok) break;
          if (j > 0) umma_commit(&kv_empty[cv & 3]);
          if (j < nmax) umma_commit(&kv_empty[ck & 3]);
          if (j + 1 == nmax) umma_commit(q_empty);
        }
        n += nmax;
      }
      if (!ok) report_status(a.status, kStatusTimeoutMma);
    }
    __syncwarp();
  } else {
    // -------------------------------------------------------------------- softmax
    const int k = warp >> 2;                 // tile of the pair
    const int r = threadIdx.x & 127;         // row
    const uint32_t lane_base = tmem_base + (uint32_t((warp & 3) * 32) << 16);
    const uint32_t tS = lane_base + C::S_COL + k * 128, tO = lane_base + C::O_COL + k * 128;
    int cnt = 0;                             // blocks of this tile so far
    const float scale = a.scale_log2;
    for (int it = 0;; ++it) {
      const int slot = it & 1;
      if (!__all_sync(0xffffffffu, pair_wait(&work_full[slot], (it >> 1) & 1))) {
        report_status(a.status, kStatusTimeoutEpilogue);
        break;
      }
      const PairItem t = s_work[slot];
      __syncwarp();
      if (lane == 0) mbar_arrive(&work_empty[slot]);
      if (t.hk < 0) break;
      const int kv_end = pair_kv_end(t, k, QT, a.causal);
      const int nblk = pair_blocks(kv_end);
      if (nblk == 0) continue;
      const int q0 = t.q0 + k * QT;
      const int qpos = q0 + (r & (QT - 1));
      const bool valid = qpos < t.len;
      const int limit = a.causal ? min(t.len, qpos + 1) : t.len;   // columns this row may see
      const int full_cols = a.causal ? min(t.len, q0 + 1) : t.len; // columns every row may see
      float m_ref = -INFINITY, l_sum = 0.f;
      bool ok = true;
      for (int j = 0; j < nblk; ++j, ++cnt) {
        ok = __all_sync(0xffffffffu, pair_wait(&s_full[k], cnt & 1));
        if (!ok) break;
        tc_fence_after();
        // the whole row at once: a load of 32 columns has a latency of some 300 clocks
        uint32_t s[4][32];
#pragma unroll
        for (int h = 0; h < 4; ++h) tmem_ld_32x32b_x32(tS + h * 32, s[h]);
#pragma unroll
        for (int h = 0; h < 4; ++h) tmem_ld_wait_for(s[h]);
        const int kv0 = j * kPairBlock;
        const int nc = pair_chunks(kv_end, j);     // the chunks behind are stale: masked, no P
        if (kv0 + kPairBlock > full_cols) {
          const int lim = limit - kv0;
#pragma unroll
          for (int c = 0; c < 128; ++c)
            if (c >= lim) s[c >> 5][c & 31] = __float_as_uint(-INFINITY);
        }
        // The reference of the exponentials moves by whole halves of 64 columns, and only when the
        // maximum rose by more than 2^8 somewhere in the warp (lazy rescale); products, differences
        // and the row sum are rounded one by one, columns in order. These are the roundings of the
        // one-tile kernel: the two give the same bits unless a second half moves the reference.
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int c = 0; c < 128; c += 2) {
          float& m = mx[(c >> 6) * 2 + ((c >> 1) & 1)];
          m = max3_(m, __uint_as_float(s[c >> 5][c & 31]), __uint_as_float(s[c >> 5][(c & 31) + 1]));
        }
        float m_new = fmaxf(m_ref, fmaxf(mx[0], mx[1]) * scale), m_to = m_ref;
        if (__any_sync(0xffffffffu, valid && m_new > m_to + 8.f)) m_to = m_new;
        m_new = fmaxf(m_to, fmaxf(mx[2], mx[3]) * scale);
        if (__any_sync(0xffffffffu, valid && m_new > m_to + 8.f)) m_to = m_new;
        // (the scores of this block were issued after the previous P·V was complete: O may be touched)
        if (__any_sync(0xffffffffu, m_to != m_ref)) {
          const float alpha = m_to == -INFINITY ? 1.f : ex2_(m_ref - m_to);
          l_sum *= alpha;
          m_ref = m_to;
          if (j > 0) {
#pragma unroll 1
            for (int c = 0; c < HD / 32; ++c) {
              uint32_t o[32];
              tmem_ld_32x32b_x32(tO + c * 32, o);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
              tmem_st_32x32b_x32(tO + c * 32, o);
            }
          }
        }
        const float m_use = m_ref == -INFINITY ? 0.f : m_ref;
        const unsigned long long m2 = pair_(-m_use, -m_use);
#pragma unroll
        for (int h = 0; h < 4; ++h)
          if (h < nc) {
            uint32_t p[16];
#pragma unroll
            for (int c = 0; c < 16; ++c) {
              // (the packed product would be contracted with the packed sum)
              const float2 x = unpair_(add2_(pair_(__fmul_rn(__uint_as_float(s[h][2 * c]), scale),
                                                   __fmul_rn(__uint_as_float(s[h][2 * c + 1]),
                                                             scale)), m2));
              const float p0 = ex2_(x.x), p1 = ex2_(x.y);
              l_sum += p0;
              l_sum += p1;
              p[c] = pack_bf16x2(p0, p1);
            }
            tmem_st_32x32b_x16(tS + h * 16, p);
          }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[k]);
      }
      if (ok) ok = __all_sync(0xffffffffu, pair_wait(&o_full[k], (cnt - 1) & 1));
      if (!ok) {
        report_status(a.status, kStatusTimeoutMma);
        break;
      }
      tc_fence_after();
      const float inv = l_sum > 0.f ? 1.f / l_sum : 0.f;
      const long long tok = 1LL * t.seq0 + qpos;
      const int head = t.hk * G + (r >> qt_shift);
      // 32 columns at a time through shared memory, so that four lanes store 64 contiguous bytes
      // of a row (one row per lane would touch 32 rows with every store)
      uint8_t* stage = sOut + warp * C::OUT_BYTES;
      __nv_bfloat16* out_row[4];
      bool out_ok[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int rr = (warp & 3) * 32 + (lane >> 2) + 8 * i;
        const int qp = q0 + (rr & (QT - 1));
        out_ok[i] = qp < t.len;
        out_row[i] = a.O + (1LL * t.seq0 + qp) * a.ldo + (t.hk * G + (rr >> qt_shift)) * HD +
                     (lane & 3) * 8;
      }
      const unsigned long long inv2 = pair_(inv, inv);
#pragma unroll 1
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t o[32];
        tmem_ld_32x32b_x32(tO + c * 32, o);
        tmem_ld_wait_for(o);
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          uint32_t w[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 f = unpair_(mul2_(pair_(__uint_as_float(o[8 * v + 2 * i]),
                                                 __uint_as_float(o[8 * v + 2 * i + 1])), inv2));
            w[i] = pack_bf16x2(f.x, f.y);
          }
          *reinterpret_cast<uint4*>(stage + lane * 80 + v * 16) = make_uint4(w[0], w[1], w[2], w[3]);
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (out_ok[i])
            *reinterpret_cast<uint4*>(out_row[i] + c * 32) = *reinterpret_cast<const uint4*>(
                stage + ((lane >> 2) + 8 * i) * 80 + (lane & 3) * 16);
        __syncwarp();
      }
      if (valid && a.lse != nullptr)
        a.lse[1LL * head * a.T + tok] =
            l_sum > 0.f ? (m_ref * kLn2F + logf(l_sum)) : -INFINITY;
      // the reads of O above come before the next item's first P·V: that product waits for p_full,
      // which this warp signals behind them
      tc_fence_before();
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 9) tmem_dealloc(tmem_base, C::TMEM_COLS);
  clear_outside(a.plan, a.capacity, a.seq_start, a.seq_end, a.O, a.ldo, a.T, a.Hq * HD / 8);
  finish_grid(a.plan, a.capacity);   // thread 0 belongs to warp 0; the item counter is final: the
                                     // barrier above came after the last item was drawn
}

}  // namespace
}  // namespace lb
