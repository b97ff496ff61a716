// bf16 GEMM for products that a 256 x 256 tile per CTA pair leaves most of the chip idle on: few
// tokens (a query, a small training batch) against weights of any size.
//
// Such a product is bound by how fast the weights reach the tensor cores, and one SM takes in
// about 100 bytes a clock however few rows there are. So the work is cut until every SM has some:
// 128 x 128 down to 64 x 32 tiles, and the contraction of a tile split over a cluster of up to eight
// CTAs. Each CTA of the cluster leaves its fp32 partial tile in its own shared memory; after a
// cluster barrier every CTA sums a share of the tile over the cluster through distributed shared
// memory, in rank order (no atomics: the result does not depend on timing), and stores it. One
// tile per CTA; up to four CTAs share an SM, and one's set-up and epilogue run under the others' main
// loops; a CTA with an SM of its own takes all of the shared memory for its operand ring.
//
//   warp 0      TMA producer          warp 1   tcgen05.mma issuer
//   warps 2-5   accumulator -> shared memory -> (cluster sum) -> global memory
//
// Projections that share an input, an output or a token contraction (q, k, v; gate, up) are one
// launch: see LbSmallGemm. The gated pair takes gate and up rows of the same features into one
// tile and writes act(gate) * up from the epilogue; the GELU of a single product (BERT's) is written there too
// (650 x 3072 x 768: 8 us, with a launch of its own 12).
//
// Measurements: see lb_gemm_small_plan.
#include "gemm_small.h"

#include <cuda_bf16.h>

#include "../common/pdl.h"
#include "../common/ptx.cuh"
#include "../common/tma_desc.h"

namespace lb {

namespace {

constexpr int BK = 64;
constexpr int kThreads = 192;
constexpr int kMaxSplits = 8;
constexpr int kMaxStages = 16;          // of the operand ring
constexpr int kRingExtra = 1024 + 512;  // alignment, barriers

struct SmallArgs {
  int M, N;
  int kb_total, splits;
  int nparts, mode;
  int ext[3];       // extent of each part
  int first[3];     // first tile (kParallelN / M) or first k-block (kParallelK) of each part
  int tiles_n;
  void* C[3];
  long long ldc[3];
  const __nv_bfloat16* bias[3];
  void* glu_h;
  long long ld_h;
  float scale;      // of the rounded product (0: none)
  int b_ready;
  int by_part;      // kParallelK of several parts: CTA r of a cluster contracts part r
  int block_bytes;  // what the loads of one k-block bring
  int stages, kps;  // of the operand ring: stages of kps k-blocks
  int* status;
};

template <int BM, int BN>
struct SCfg {
  static constexpr int A_BYTES = BM * BK * 2;
  static constexpr int B_BYTES = BN * BK * 2;
  static constexpr int BLOCK_BYTES = A_BYTES + B_BYTES;
  static constexpr int PITCH = BN + 4;  // floats per row of the partial tile: 16-byte row accesses
                                        // of eight lanes then fall into different banks
  // the partial tile reuses the operand ring
  static constexpr int MIN_BLOCKS = (BM * PITCH * 4 + BLOCK_BYTES - 1) / BLOCK_BYTES;
  static constexpr int smem_bytes(int blocks) { return blocks * BLOCK_BYTES + kRingExtra; }
};

__device__ __forceinline__ uint32_t cta_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// (the aligned forms want the whole warp: threads that left a loop early meet the others first)
__device__ __forceinline__ void cluster_sync_() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
  uint32_t out;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(addr), "r"(rank));
  return out;
}
__device__ __forceinline__ float4 ld_cluster4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}

// The values of the stand-alone activation kernels (row/act.cu): the same bits. GLU: 3 = GELU (erf), of the
// product itself; of the gate of a pair 1 = SiLU, 2 =
// tanh-GELU.
template <int GLU>
__device__ __forceinline__ float act_of(float x) {
  if constexpr (GLU == 1) {
    return x * __frcp_rn(1.f + __expf(-x));
  } else if constexpr (GLU == 3) {
    return 0.5f * x * (1.f + erff(x * 0.7071067811865476f));
  } else {
    const float k0 = 0.7978845608028654f, k1 = 0.044715f;
    return 0.5f * x * (1.f + tanhf(k0 * (x + k1 * x * x * x)));
  }
}

__device__ __forceinline__ float bf16_rn(float x) {
  return __bfloat162float(__float2bfloat16_rn(x));
}

// Sum over the cluster of four consecutive floats at byte offset `off` of every partial tile. Products
// of several parts (by_part) are added up in bf16, one after the other: the roundings of launches
// that each add to the result in memory.
__device__ __forceinline__ float4 cluster_sum4(uint32_t base, uint32_t off, int splits,
                                               int by_part = 0) {
  if (splits == 1) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(base + off)
                 : "memory");
    return v;
  }
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int s0 = 0; s0 < splits; s0 += 4) {  // all of a group's loads before its additions
    float4 t[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      t[j] = s0 + j < splits ? ld_cluster4(map_rank(base, s0 + j) + off)
                             : make_float4(0.f, 0.f, 0.f, 0.f);
    if (by_part) {  // (at most three parts: one group)
      acc = t[0];
#pragma unroll
      for (int j = 1; j < 3; ++j)
        if (j < splits) {
          acc.x = bf16_rn(bf16_rn(acc.x) + bf16_rn(t[j].x));
          acc.y = bf16_rn(bf16_rn(acc.y) + bf16_rn(t[j].y));
          acc.z = bf16_rn(bf16_rn(acc.z) + bf16_rn(t[j].z));
          acc.w = bf16_rn(bf16_rn(acc.w) + bf16_rn(t[j].w));
        }
      return acc;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      acc.x += t[j].x;
      acc.y += t[j].y;
      acc.z += t[j].z;
      acc.w += t[j].w;
    }
  }
  return acc;
}

template <int A_MN, int B_MN, int BM, int BN, typename OutT, int GLU>
__global__ void __launch_bounds__(kThreads)
    gemm_small_kernel(const __grid_constant__ CUtensorMap tmA,
                      const __grid_constant__ CUtensorMap tmB0,
                      const __grid_constant__ CUtensorMap tmB1,
                      const __grid_constant__ CUtensorMap tmB2, SmallArgs g) {
  using C = SCfg<BM, BN>;
  const int stages = g.stages, kps = g.kps;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + stages * kps * C::BLOCK_BYTES);
  uint64_t* empty = full + kMaxStages;
  uint64_t* tfull = empty + kMaxStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfull + 1);

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  const int S = g.splits;
  const int rank = S > 1 ? int(cta_rank()) : 0;
  const int tile = int(blockIdx.x) / S;
  // contraction of this CTA: a share of the whole (>= 1 block: S <= kb_total), or one part
  const int kb0 = g.by_part ? g.first[rank] : rank * g.kb_total / S;
  const int kb1 = g.by_part ? (rank + 1 < S ? g.first[rank + 1] : g.kb_total)
                            : (rank + 1) * g.kb_total / S;
  const int nkb = kb1 - kb0;

  // tile -> part, origin in C, origin of the rows / columns read from A and B
  const int tm = tile / g.tiles_n, tn = tile - tm * g.tiles_n;
  int part = 0;
  if (g.mode != kParallelK) {
    const int t = g.mode == kParallelN ? tn : tm;
    while (part + 1 < g.nparts && t >= g.first[part + 1]) ++part;
  }
  constexpr bool PAIR = GLU == 1 || GLU == 2;
  constexpr int kCols = PAIR ? BN / 2 : BN;            // output columns of a tile
  int m0 = tm * BM, n0 = tn * kCols, am0 = m0, m_ext = g.M, n_ext = g.N;
  if (g.mode == kParallelN && !PAIR) {
    n0 = (tn - g.first[part]) * BN;
    n_ext = g.ext[part];
  } else if (g.mode == kParallelM) {
    m0 = (tm - g.first[part]) * BM;
    m_ext = g.ext[part];
    am0 = m0;
    for (int p = 0; p < part; ++p) am0 += g.ext[p];
  }
  if (PAIR) n_ext = g.ext[0];

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tfull, 1);
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB0);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      const int bp = g.mode == kParallelN ? part : (g.by_part ? rank : 0);
      const CUtensorMap* tb = bp == 0 ? &tmB0 : (bp == 1 ? &tmB1 : &tmB2);
      const int kb_b = kb0 - (g.by_part ? g.first[rank] : 0);
      auto load_a = [&](int i, int s) {   // i: k-block, s: ring position in blocks
        uint8_t* sa = smem + s * C::BLOCK_BYTES;
        uint64_t* bar = &full[kps == 1 ? s : s >> 1];
        const int kc = (kb0 + i) * BK;
        if (A_MN) {
#pragma unroll
          for (int c = 0; c < BM / 64; ++c)
            tma_load_2d(sa + c * (BK * 128), &tmA, bar, am0 + 64 * c, kc);
        } else {
          tma_load_2d(sa, &tmA, bar, kc, am0);
        }
      };
      auto load_b = [&](int i, int s) {
        uint8_t* sb = smem + s * C::BLOCK_BYTES + C::A_BYTES;
        uint64_t* bar = &full[kps == 1 ? s : s >> 1];
        const int kc = (kb_b + i) * BK;
        if (PAIR) {  // gate rows, then up rows of the same features
          tma_load_2d(sb, &tmB0, bar, kc, n0);
          tma_load_2d(sb + (BN / 2) * 128, &tmB1, bar, kc, n0);
        } else if (B_MN) {
#pragma unroll
          for (int c = 0; c < BN / 64; ++c)
            tma_load_2d(sb + c * (BK * 128), tb, bar, n0 + 64 * c, kc);
        } else {
          tma_load_2d(sb, tb, bar, kc, n0);
        }
      };
      const int pre = min(nkb, stages * kps);
      for (int i = 0, s = 0; i < pre; i += kps, ++s)
        mbar_expect_tx(&full[s], g.block_bytes * min(kps, nkb - i));
      if (g.b_ready) {
        for (int i = 0; i < pre; ++i) load_b(i, i);
        pdl_wait();
        for (int i = 0; i < pre; ++i) load_a(i, i);
      } else {
        pdl_wait();
        for (int i = 0; i < pre; ++i) {
          load_a(i, i);
          load_b(i, i);
        }
      }
      bool ok = true;
      int s = 0;
      uint32_t phase = 0;
      for (int i = pre; i < nkb; i += kps) {
        if (!mbar_wait(&empty[s], phase)) {
          report_status(g.status, kStatusTimeoutProducer);
          ok = false;
          break;
        }
        const int here = min(kps, nkb - i);
        mbar_expect_tx(&full[s], g.block_bytes * here);
#pragma unroll 1
        for (int j = 0; j < here; ++j) {
          load_a(i + j, s * kps + j);
          load_b(i + j, s * kps + j);
        }
        if (++s == stages) {
          s = 0;
          phase ^= 1u;
        }
      }
      if (!ok) {
        // copies already requested land within microseconds: a bounded grace period before exit
        const unsigned long long t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 200000ull) {
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      constexpr uint32_t idesc = umma_idesc_bf16(BM, BN, A_MN, B_MN);
      bool ok = true;
      int s = 0;
      uint32_t phase = 0;
      for (int i = 0; i < nkb; i += kps) {
        if (!mbar_wait(&full[s], phase)) {
          report_status(g.status, kStatusTimeoutMma);
          ok = false;
          break;
        }
        tc_fence_after();
        const int here = min(kps, nkb - i);
#pragma unroll 1
        for (int j = 0; j < here; ++j) {
          const uint32_t sa = smem_u32(smem + (s * kps + j) * C::BLOCK_BYTES);
          const uint32_t sb = sa + C::A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            const uint64_t adesc = A_MN ? umma_smem_desc(sa + k * 2048, BK * 128, 1024)
                                        : umma_smem_desc(sa + k * 32, 16, 1024);
            const uint64_t bdesc = B_MN ? umma_smem_desc(sb + k * 2048, BK * 128, 1024)
                                        : umma_smem_desc(sb + k * 32, 16, 1024);
            umma_bf16(tmem_base, adesc, bdesc, idesc, (i + j > 0 || k > 0) ? 1u : 0u);
          }
        }
        umma_commit(&empty[s]);
        if (++s == stages) {
          s = 0;
          phase ^= 1u;
        }
      }
      if (ok) umma_commit(tfull);
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ accumulator -> shared memory
    pdl_wait();
    pdl_trigger();
    const int q = warp & 3;
    const bool ok = mbar_wait(tfull, 0);
    if (!ok && lane == 0) report_status(g.status, kStatusTimeoutEpilogue);
    tc_fence_after();
    // 64-row tiles: 16 rows in the lower half of each warp's lanes
    constexpr int kRows = BM / 4;
    if (__all_sync(0xffffffffu, ok) && m0 + q * kRows < m_ext) {
      float* prow = reinterpret_cast<float*>(smem) + (q * kRows + lane) * C::PITCH;
#pragma unroll
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t r[32];
        tmem_ld_32x32b_x32(tmem_base + (uint32_t(q * 32) << 16) + c * 32, r);
        tmem_ld_wait();
        if (lane < kRows)
#pragma unroll
        for (int j = 0; j < 8; ++j)
          *reinterpret_cast<float4*>(prow + c * 32 + 4 * j) =
              make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]),
                          __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
      }
    }
    tc_fence_before();
  }
  pdl_wait();   // for itself in every thread: all of them store below
  if (S > 1)
    cluster_sync_();
  else
    __syncthreads();

  // ---------------------------------------------------------------------- sum and store
  // (all 192 threads; after a failed wait the values are meaningless and the status word says so)
  const int rows = min(BM, m_ext - m0);
  const uint32_t base = smem_u32(smem);
  if (sizeof(OutT) == 2) {
    constexpr int VPR = kCols / 8;
    const int total = rows * VPR;
    const int per = (total + S - 1) / S;
    const int hi = min(total, (rank + 1) * per);
    for (int v = rank * per + int(threadIdx.x); v < hi; v += kThreads) {
      const int row = v / VPR, c = (v % VPR) * 8;
      if (n0 + c >= n_ext) continue;
      const uint32_t off = uint32_t(row * C::PITCH + c) * 4u;
      float4 a0 = cluster_sum4(base, off, S, g.by_part);
      float4 a1 = cluster_sum4(base, off + 16u, S, g.by_part);
      if (!PAIR && g.bias[part] != nullptr) {
        const uint4 bq = *reinterpret_cast<const uint4*>(g.bias[part] + n0 + c);
        const float2 b0 = unpack_bf16x2(bq.x), b1 = unpack_bf16x2(bq.y);
        const float2 b2 = unpack_bf16x2(bq.z), b3 = unpack_bf16x2(bq.w);
        a0 = make_float4(a0.x + b0.x, a0.y + b0.y, a0.z + b1.x, a0.w + b1.y);
        a1 = make_float4(a1.x + b2.x, a1.y + b2.y, a1.z + b3.x, a1.w + b3.y);
      }
      uint4 pk;
      pk.x = pack_bf16x2(a0.x, a0.y);
      pk.y = pack_bf16x2(a0.z, a0.w);
      pk.z = pack_bf16x2(a1.x, a1.y);
      pk.w = pack_bf16x2(a1.z, a1.w);
      if (!GLU && g.scale != 0.f) {
        uint32_t w[4] = {pk.x, pk.y, pk.z, pk.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 v = unpack_bf16x2(w[j]);
          w[j] = pack_bf16x2(v.x * g.scale, v.y * g.scale);
        }
        pk = make_uint4(w[0], w[1], w[2], w[3]);
      }
      const long long grow = m0 + row;
      if constexpr (PAIR) {
        const float4 u0 = cluster_sum4(base, off + BN / 2 * 4u, S);
        const float4 u1 = cluster_sum4(base, off + BN / 2 * 4u + 16u, S);
        uint4 pu;
        pu.x = pack_bf16x2(u0.x, u0.y);
        pu.y = pack_bf16x2(u0.z, u0.w);
        pu.z = pack_bf16x2(u1.x, u1.y);
        pu.w = pack_bf16x2(u1.z, u1.w);
        if (g.C[0] != nullptr) {
          *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(g.C[0]) + grow * g.ldc[0] +
                                    n0 + c) = pk;
          *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(g.C[1]) + grow * g.ldc[1] +
                                    n0 + c) = pu;
        }
        const uint32_t gw[4] = {pk.x, pk.y, pk.z, pk.w}, uw[4] = {pu.x, pu.y, pu.z, pu.w};
        uint32_t hw[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 gv = unpack_bf16x2(gw[j]), uv = unpack_bf16x2(uw[j]);
          hw[j] = pack_bf16x2(act_of<GLU>(gv.x) * uv.x, act_of<GLU>(gv.y) * uv.y);
        }
        *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(g.glu_h) + grow * g.ld_h + n0 +
                                  c) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
      } else {
        if (GLU != 3 || g.C[0] != nullptr)
          *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(g.C[part]) +
                                    grow * g.ldc[part] + n0 + c) = pk;
        if constexpr (GLU == 3) {
          const uint32_t w[4] = {pk.x, pk.y, pk.z, pk.w};
          uint32_t hw[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 v = unpack_bf16x2(w[j]);
            hw[j] = pack_bf16x2(act_of<3>(v.x), act_of<3>(v.y));
          }
          *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(g.glu_h) + grow * g.ld_h + n0 + c) =
              make_uint4(hw[0], hw[1], hw[2], hw[3]);
        }
      }
    }
  } else {
    constexpr int VPR = kCols / 4;
    const int total = rows * VPR;
    const int per = (total + S - 1) / S;
    const int hi = min(total, (rank + 1) * per);
    for (int v = rank * per + int(threadIdx.x); v < hi; v += kThreads) {
      const int row = v / VPR, c = (v % VPR) * 4;
      if (n0 + c >= n_ext) continue;
      const float4 a = cluster_sum4(base, uint32_t(row * C::PITCH + c) * 4u, S);
      asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(
                       reinterpret_cast<float*>(g.C[part]) + (m0 + row) * g.ldc[part] + n0 + c),
                   "f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w)
                   : "memory");
    }
  }
  // nobody gives its shared memory back while a peer may still read it
  if (S > 1)
    cluster_sync_();
  else
    __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, BN);
}

int small_sms() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
      n = 148;
  }
  return n;
}

inline int ceil_div(int a, int b) { return (a + b - 1) / b; }

int kblocks(const LbSmallGemm* p) {
  if (p->mode != kParallelK) return ceil_div(p->K, BK);
  int n = 0;
  for (int i = 0; i < p->nparts; ++i) n += ceil_div(p->ext[i], BK);
  return n;
}

int tiles_along(const LbSmallGemm* p, int mode, int whole, int tile) {
  if (p->mode != mode) return ceil_div(whole, tile);
  int n = 0;
  for (int i = 0; i < p->nparts; ++i) n += ceil_div(p->ext[i], tile);
  return n;
}

constexpr int kSmemLimit = 227 * 1024;
struct SmallTile {
  int bm, bn, min_blocks;
};
// 64-row tiles cut a long contraction of few tokens finer (what a CTA takes in bounds it), 32 columns
// more so; 128 x 128 has the least traffic per product, for many tiles.
constexpr SmallTile kSmallTiles[] = {{128, 128, SCfg<128, 128>::MIN_BLOCKS},
                                     {128, 64, SCfg<128, 64>::MIN_BLOCKS},
                                     {64, 64, SCfg<64, 64>::MIN_BLOCKS},
                                     {64, 32, SCfg<64, 32>::MIN_BLOCKS}};

// The operand ring of each of `grid` CTAs: the k-blocks in it and per stage. The CTAs that find place
// on an SM side by side share its memory: with few CTAs one has all of it, and its loads cover the
// latency of the weights (4 blocks of 24 KB in flight: 17.3 us for 160 x 1024 x 3072, 8: 12.9).
// Returns how many CTAs an SM holds.
int ring_of(int bm, int bn, int grid, int cluster, int* blocks_out, int* kps_out) {
  const int block_bytes = (bm + bn) * BK * 2;
  int min_blocks = 0;
  for (const SmallTile& t : kSmallTiles)
    if (t.bm == bm && t.bn == bn) min_blocks = t.min_blocks;
  // (clusters do not fill every SM: one CTA per SM each, 144 CTAs in clusters of three or four took two waves)
  int per_sm = ceil_div(grid, cluster > 1 ? small_sms() * 3 / 4 : small_sms());
  if (per_sm > 4) per_sm = 4;
  int blocks = (224 * 1024 / per_sm - 1024 - kRingExtra) / block_bytes;
  if (blocks > kMaxStages) blocks = kMaxStages;
  if (blocks < min_blocks) blocks = min_blocks;
  // two blocks a stage halve the hand-overs between the threads that load and issue; a short ring is
  // handed over in single blocks
  *kps_out = blocks >= 6 ? 2 : 1;
  *blocks_out = blocks = blocks / *kps_out * *kps_out;
  const int fit = kSmemLimit / (blocks * block_bytes + kRingExtra + 1024);
  return fit < per_sm ? fit : per_sm;
}

bool gated(const LbSmallGemm* p) { return p->glu_h != nullptr && p->glu_kind != 2; }
bool by_part(const LbSmallGemm* p) { return p->mode == kParallelK && p->nparts > 1; }

int count_tiles(const LbSmallGemm* p, int bm, int bn, int* tiles_n) {
  const int tm = tiles_along(p, kParallelM, p->M, bm);
  const int tn = gated(p) ? ceil_div(p->ext[0], bn / 2)
                                     : tiles_along(p, kParallelN, p->N, bn);
  *tiles_n = tn;
  return tm * tn;
}

bool shape_ok(const LbSmallGemm* p) {
  if (p->M <= 0 || p->N <= 0 || p->K <= 0 || p->nparts < 1 || p->nparts > 3) return false;
  if (p->lda & 7) return false;
  for (int i = 0; i < p->nparts; ++i) {
    if (p->ext[i] <= 0 || (p->ext[i] & 7)) return false;
    if (p->mode != kParallelM && (p->ldb[i] & 7)) return false;
    if (p->mode == kParallelK && (p->ext[i] % BK) != 0) return false;  // a k-block has one weight
  }
  if (p->mode == kParallelM && (p->ldb[0] & 7)) return false;
  if (p->mode != kParallelN && (p->N & 7)) return false;
  for (int i = 0; i < (p->mode == kParallelK ? 1 : p->nparts); ++i)
    if (p->C[i] != nullptr && (p->ldc[i] & (p->out_fp32 ? 3 : 7))) return false;
  if (p->glu_h != nullptr &&
      (p->mode != kParallelN || p->a_mn || p->b_mn || p->out_fp32 || (p->ld_h & 7) ||
       (gated(p) ? p->nparts != 2 || p->ext[0] != p->ext[1] : p->nparts != 1)))
    return false;
  if (p->a_mn && !p->b_mn) return false;        // not a product of a linear layer
  if (p->out_fp32 != (p->a_mn ? 1 : 0)) return false;
  for (int i = 0; i < p->nparts; ++i)
    if (p->bias[i] != nullptr &&
        (p->mode != kParallelN || gated(p) || p->out_fp32 ||
         (reinterpret_cast<uintptr_t>(p->bias[i]) & 15u) != 0))
      return false;
  return true;
}

// Modelled time of a weight gradient over kLongSum k-blocks or more, for the comparison with the tile kernels
// alone: which of them takes it decides whether it is summed whole or in pieces, hence its bits and, through the
// clip coefficient, those of every weight of the step. So this and its counterpart in lb_gemm_tile_cost stay
// as they were fitted first (128-row tiles in rings of four and three stages), whatever the kernel has become
// since.
double long_sum_cost(const LbSmallGemm* p, int kb) {
  double best = 1e30;
  for (int bn = 64; bn <= 128; bn += 64) {
    int tn;
    const int tiles = count_tiles(p, 128, bn, &tn);
    const double waves = ceil_div(tiles, 2 * small_sms()), per_sm = ceil_div(tiles, small_sms());
    const double block = per_sm * (128 + bn) * 2.0, latency = waves * 2600.0 / (bn == 64 ? 4.0 : 3.0);
    const double cost =
        2.0 + waves * (1.1 + 1.8 * 128 * bn / 8192.0) + kb * (block > latency ? block : latency) / 1900.0;
    if (cost < best) best = cost;
  }
  return best;
}

template <int A_MN, int B_MN, int BM, int BN, typename OutT, int GLU>
int launch_small(const CUtensorMap& tA, const CUtensorMap* tB, const SmallArgs& g, int grid,
                 cudaStream_t st) {
  using C = SCfg<BM, BN>;
  auto kern = gemm_small_kernel<A_MN, B_MN, BM, BN, OutT, GLU>;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit) !=
        cudaSuccess)
      return -10;
    configured = true;
  }
  SmallArgs a = g;
  int blocks;
  ring_of(BM, BN, grid, g.splits, &blocks, &a.kps);
  a.stages = blocks / a.kps;
  return launch_pdl(kern, dim3(grid), dim3(kThreads), C::smem_bytes(blocks), st, pdl_enabled(),
                    g.splits, tA, tB[0], tB[1], tB[2], a);
}

template <int BM, int BN>
int dispatch(const LbSmallGemm* p, const CUtensorMap& tA, const CUtensorMap* tB, const SmallArgs& g,
             int grid, cudaStream_t st) {
  if (p->glu_h != nullptr && !gated(p))
    return launch_small<0, 0, BM, BN, __nv_bfloat16, 3>(tA, tB, g, grid, st);
  if (p->glu_h != nullptr)
    return p->glu_kind == 0 ? launch_small<0, 0, BM, BN, __nv_bfloat16, 1>(tA, tB, g, grid, st)
                            : launch_small<0, 0, BM, BN, __nv_bfloat16, 2>(tA, tB, g, grid, st);
  if constexpr (BN >= 64) {
    if (p->a_mn) return launch_small<1, 1, BM, BN, float, 0>(tA, tB, g, grid, st);
    if (p->b_mn) return launch_small<0, 1, BM, BN, __nv_bfloat16, 0>(tA, tB, g, grid, st);
  }
  return launch_small<0, 0, BM, BN, __nv_bfloat16, 0>(tA, tB, g, grid, st);
}

}  // namespace
}  // namespace lb

using namespace lb;

// Microseconds, fitted (10 % rms) to 2300 measurements of products of transformer blocks (widths 768 to
// 2560, FFNs up to 9728) at 1 to 1400 tokens with every tile and split, weights cold; what it chooses is
// 1.7 % slower than the best of them in the geometric mean. A launch, and per wave of resident CTAs its
// set-up, a split's cluster barriers, and for each k-block the largest of what the SM takes in (103
// bytes a clock), the issue of its products and the latency of the loads in flight; the store of the
// tiles; and no less than the bytes take from memory.
//   tokens x N x K                     before    now (us per launch of a graph, weights cold)
//   32 x 1024 x 3072                   19.3      10.1   64 x 32 tiles, sixteen k-blocks in flight
//   160 x 1024 x 3072                  20.0      10.4
//   660 x 1024 x 2048                  15.2      10.5
//   160 x (2048, 1024, 1024) x 1024    10.6       8.2
//   160 x 1024 x (3072, 3072) (dgrad)  22.5      16.2
//   32 x 1024 x 3072, split            9.0        7.2
extern "C" double lb_gemm_small_plan(const LbSmallGemm* p, int* bn_out, int* splits_out) {
  if (!shape_ok(p)) return -1.0;
  const int sms = small_sms();
  const int kb = kblocks(p);
  // Split only where the caller takes sums in another order (in a training step a different
  // rounding of one layer shows in the loss after the next update): an unsplit product has the bits
  // that the tile kernels give. Nothing is lost for the weight gradients, which are never faster
  // split. A product of several parts always has a CTA per part.
  const bool parts = by_part(p);
  const int max_splits = p->a_mn || !p->may_split || parts ? 1 : kMaxSplits;
  int kb_part = 0;
  for (int i = 0; parts && i < p->nparts; ++i)
    kb_part = ceil_div(p->ext[i], BK) > kb_part ? ceil_div(p->ext[i], BK) : kb_part;
  const double out_cols = gated(p) ? p->ext[0] : p->N;
  const double bytes = 2.0 * p->K * (double(p->M) + p->N) + (p->out_fp32 ? 8.0 : 2.0) * p->M * out_cols;
  double best = 1e30;
  for (const SmallTile& t : kSmallTiles) {
    if (t.bn < 64 && p->b_mn) continue;   // (rows of 64 columns are the unit of those loads)
    const int a_rows = p->M < t.bm && !p->a_mn ? p->M : t.bm;
    int tn;
    const int tiles = count_tiles(p, t.bm, t.bn, &tn);
    for (int s1 = 1; s1 <= max_splits && s1 <= kb; s1 *= 2) {
      const int s = parts ? p->nparts : s1;
      const int ctas = tiles * s;
      int blocks, kps;
      const int res = ring_of(t.bm, t.bn, ctas, s, &blocks, &kps);
      const int capacity = res * (sms - (s == 8 ? 20 : (s == 4 ? 8 : (s == 3 ? 7 : 0))));
      const int waves = ceil_div(ctas, capacity);
      int rest = ceil_div(ctas - (waves - 1) * capacity, sms);
      if (rest > res) rest = res;
      const double in = (a_rows + t.bn) * 128.0 / 103.0;
      const double least = kps == 2 ? 290.0 : 600.0, flight = 2500.0 / blocks;
      const double floor_clk = least > flight ? least : flight;
      const double full = in * res > floor_clk ? in * res : floor_clk;
      const double last = in * rest > floor_clk ? in * rest : floor_clk;
      const double split = s == 1 ? 0.0 : (s <= 3 ? 1.3 : (s == 4 ? 1.7 : 2.8));
      double cost = 3.4 + waves * (0.8 + split) +
                    (p->out_fp32 ? 1.28 : 1.43) * a_rows * t.bn / 8192.0 * ceil_div(ctas, sms) +
                    (parts ? kb_part : ceil_div(kb, s)) * ((waves - 1) * full + last) / 1900.0;
      const double memory = 3.0 + bytes / 3.96e6;
      if (cost < memory) cost = memory + 1e-3 * cost;   // (of several at that bound the least busy)
      if (cost < best) {
        best = cost;
        *bn_out = t.bn | t.bm << 16;
        *splits_out = s;
      }
    }
  }
  return p->out_fp32 && kb >= kLongSum ? long_sum_cost(p, kb) : best;
}

extern "C" int lb_gemm_small(const LbSmallGemm* p) { return lb_gemm_small_scaled(p, 0.f); }

extern "C" int lb_gemm_small_scaled(const LbSmallGemm* p, float scale) {
  if (p->M <= 0 || p->N <= 0) return 0;
  if (!shape_ok(p) || (scale != 0.f && (p->out_fp32 || p->glu_h != nullptr))) return -3;
  // tile: columns, and rows in the upper half (0: 128)
  int tile = p->bn, splits = p->splits;
  if (tile == 64 || tile == 128) tile |= 128 << 16;
  bool known = false;
  for (const SmallTile& t : kSmallTiles)
    known = known || (tile == (t.bn | t.bm << 16) && !(t.bn < 64 && p->b_mn));
  if (!known || splits <= 0) {
    int t2 = 64, s2 = 1;
    lb_gemm_small_plan(p, &t2, &s2);
    if (!known) tile = t2;
    if (splits <= 0) splits = s2;
  }
  const int bn = tile & 0xffff, BM = tile >> 16;
  const int kb = kblocks(p);
  if (by_part(p)) {
    splits = p->nparts;
  } else {
    if (splits != 1 && splits != 2 && splits != 4 && splits != 8) return -3;
    while (splits > kb) splits /= 2;
  }

  CUtensorMap tA, tB[3];
  int rc;
  // An operand with fewer rows than a tile is loaded as that: rows that a copy fills in behind its end
  // cost more than rows that it fetches (input gradient 16 x 2560 x 9728 with 112 of 128 rows filled in
  // 37.2 us, 25.7 without; 1 x 6144 x 4096 61.5, 40.8). What is left in shared memory below them goes
  // to accumulator rows and columns that nobody reads.
  const int a_box = !p->a_mn && p->M < BM ? p->M : BM;
  const int b_box = !p->b_mn && !gated(p) && p->nparts == 1 && p->N < bn ? p->N : bn;
  int a_inner = p->a_mn ? p->M : p->K;
  rc = p->a_mn ? make_tmap_2d(&tA, p->A, 2, (uint64_t)a_inner, (uint64_t)p->K,
                              (uint64_t)p->lda * 2, 64, BK, true)
               : make_tmap_2d(&tA, p->A, 2, (uint64_t)a_inner, (uint64_t)p->M,
                              (uint64_t)p->lda * 2, BK, a_box, true);
  if (rc) return rc;
  const int nb = p->mode == kParallelM ? 1 : p->nparts;
  for (int i = 0; i < nb; ++i) {
    const int n = p->mode == kParallelN ? p->ext[i] : p->N;
    const int k = p->mode == kParallelK ? p->ext[i] : p->K;
    rc = p->b_mn ? make_tmap_2d(&tB[i], p->B[i], 2, (uint64_t)n, (uint64_t)k,
                                (uint64_t)p->ldb[i] * 2, 64, BK, true)
                 : make_tmap_2d(&tB[i], p->B[i], 2, (uint64_t)k, (uint64_t)n,
                                (uint64_t)p->ldb[i] * 2, BK, gated(p) ? bn / 2 : b_box,
                                true);
    if (rc) return rc;
  }
  for (int i = nb; i < 3; ++i) tB[i] = tB[0];

  SmallArgs g{};
  g.M = p->M;
  g.N = p->N;
  g.kb_total = kb;
  g.splits = splits;
  g.nparts = p->nparts;
  g.mode = p->mode;
  const int unit = p->mode == kParallelN ? bn : (p->mode == kParallelK ? BK : BM);
  int at = 0;
  for (int i = 0; i < 3; ++i) {
    g.first[i] = at;
    if (i < p->nparts) {
      g.ext[i] = p->ext[i];
      g.C[i] = p->C[i];
      g.bias[i] = static_cast<const __nv_bfloat16*>(p->bias[i]);
      g.ldc[i] = p->ldc[i];
      at += ceil_div(p->ext[i], unit);
    }
  }
  const int tiles = count_tiles(p, BM, bn, &g.tiles_n);
  g.glu_h = p->glu_h;
  g.ld_h = p->ld_h;
  g.scale = scale;
  g.b_ready = p->b_ready && pdl_enabled();
  g.by_part = by_part(p);
  g.block_bytes = (a_box + b_box) * BK * 2;
  g.status = p->status;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(p->stream);
  const int grid = tiles * splits;
  if (BM == 64)
    return bn == 32 ? dispatch<64, 32>(p, tA, tB, g, grid, st)
                    : dispatch<64, 64>(p, tA, tB, g, grid, st);
  return bn == 64 ? dispatch<128, 64>(p, tA, tB, g, grid, st)
                  : dispatch<128, 128>(p, tA, tB, g, grid, st);
}
