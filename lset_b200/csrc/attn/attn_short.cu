// Attention of a pass without gradients over few short sequences, with the per-head norms and the
// rotation of q and k in front of it: q, k and v as the projection leaves them to the attention's output in one
// launch.
//
// Such a call is a chain of latencies, not of work: the rotation's launch, and in the tile kernels barriers,
// tensor memory, descriptors and a 128-row tile for the 24 tokens of a search query. Here a CTA of four warps
// or eight takes one head of one sequence, 64 of its tokens; rows go from global to shared memory through the
// registers that norm and rotate them, and 16 x 8 x 16 tensor instructions (mma.sync), a warp's own 16 query rows,
// need nothing to be set up. Keys are walked 64 at a time with a running maximum, so any length is computed
// rightly; lb_attn_short_ok says where this is the faster way.
//
// Bound by the chain of its loads: bounds, positions and angles (fetched under the launch in front), rows, then
// the products. One search query on 28 layers of 16 + 8 heads of 128: 1.44 -> 1.30 ms; 24 short texts on
// 12 layers of 12 heads of 64: 1.17 -> 1.12 ms.
#include "../common/api.h"
#include "../common/pdl.h"
#include "../common/row.cuh"
#include "../row/rope.cuh"
#include "attn_common.cuh"

namespace lb {
namespace {

using bf16 = __nv_bfloat16;

constexpr int kShortRows = 64;

struct ShortArgs {
  const bf16 *q, *k, *v;   // [T, heads, HD], rows ld apart
  long long ld;
  const bf16 *qw, *kw;     // norm weights (do_norm)
  const float *cos, *sin;  // null: no rotation
  const void* pos;
  int pos_i64;
  const int *seq_start, *seq_end;
  const int* plan;         // for the rows outside every sequence
  int capacity;
  bf16* O;
  long long ldo;
  int T, Hq, Hk;
  int blocks;              // of 64 query rows a sequence, each a CTA's
  float eps, w_off, scale_log2;
  int do_norm, causal;
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <int HD>
struct ShortCfg {
  static constexpr int PITCH = HD + 8;   // elements: the rows of an ldmatrix fall into different banks
  static constexpr int TILE = kShortRows * PITCH;
  static constexpr int SMEM_BYTES = 3 * TILE * 2;
};

template <int HD, bool ROPE, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, WARPS == 8 ? 2 : 3) attn_short_kernel(ShortArgs a) {
  using C = ShortCfg<HD>;
  constexpr int kThreads = WARPS * 32;
  constexpr int COLS = HD * 4 / WARPS;   // output columns of a warp: two warps share 16 query rows' scores, or none
  constexpr int LPH = HD / 16, GROUPS = kThreads / LPH;
  constexpr int VECS = HD / 8;
  extern __shared__ __align__(16) bf16 smem_short[];
  __shared__ __align__(16) float swt[2 * HD];
  bf16* sQ = smem_short;
  bf16* sK = sQ + C::TILE;
  bf16* sV = sK + C::TILE;
  const uint32_t uQ = uint32_t(__cvta_generic_to_shared(sQ)), uK = uint32_t(__cvta_generic_to_shared(sK)),
                 uV = uint32_t(__cvta_generic_to_shared(sV));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int qb = blockIdx.x % a.blocks, bh = blockIdx.x / a.blocks;
  const int h = bh % a.Hq, b = bh / a.Hq;
  const int hk = h / (a.Hq / a.Hk);
  // (bounds, positions, angles and weights are older than the launch in front)
  const int seq0 = a.seq_start[b], len = a.seq_end[b] - seq0;
  if (ROPE && a.do_norm)
    for (int i = tid; i < 2 * HD; i += kThreads)
      swt[weight_at<HD>(i)] = __bfloat162float(i < HD ? a.qw[i] : a.kw[i - HD]) + a.w_off;
  // A group of LPH lanes norms and rotates a row (u < new_q: of q, then of k), UB of them at a time; the angles
  // of the first ones are fetched under the launch in front.
  constexpr int UB = 2;
  [[maybe_unused]] const int g = tid / LPH, lg = tid % LPH;
  [[maybe_unused]] f2 cs[UB][4], sn[UB][4];
  auto row_of = [&](int u, int new_q, int q0, int kv0) { return u < new_q ? q0 + u : kv0 + u - new_q; };
  auto angles = [&](int u0, int new_q, int units, int q0, int kv0) {
#pragma unroll
    for (int j = 0; j < UB; ++j) {
      const int u = u0 + j * GROUPS + g;
      load_angles<HD / 2>(a.cos, a.sin,
                          u < units ? rope_pos(a.pos, a.pos_i64, seq0 + row_of(u, new_q, q0, kv0)) : -1,
                          lg * 8, cs[j], sn[j]);
    }
  };
  bool ahead = ROPE;
  if (ROPE && qb * kShortRows < len) {
    const int q0 = qb * kShortRows, nq = min(kShortRows, len - q0);
    angles(0, nq, nq + min(kShortRows, a.causal ? min(len, q0 + kShortRows) : len), q0, 0);
  }
  __syncthreads();
  pdl_wait();
  pdl_trigger();
  clear_outside(a.plan, a.capacity, a.seq_start, a.seq_end, a.O, a.ldo, a.T, a.Hq * HD / 8);

  const bf16* qp = a.q + 1LL * seq0 * a.ld + h * HD;
  const bf16* kp = a.k + 1LL * seq0 * a.ld + hk * HD;
  const bf16* vp = a.v + 1LL * seq0 * a.ld + hk * HD;
  for (int q0 = qb * kShortRows; q0 < len; q0 += a.blocks * kShortRows) {
    const int nq = min(kShortRows, len - q0);
    const int kv_end = a.causal ? min(len, q0 + kShortRows) : len;
    const int row0 = (warp & 3) * 16;         // of this warp's query rows
    const int col0 = (warp >> 2) * COLS;      // and output columns
    float o[COLS / 8][4];
#pragma unroll
    for (int i = 0; i < COLS / 8; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[i][e] = 0.f;
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};

    for (int kv0 = 0; kv0 < kv_end; kv0 += kShortRows) {
      const int nk = min(kShortRows, kv_end - kv0);
      __syncthreads();   // nobody reads the tiles of before any more
      // values; rows up to the next multiple of 16 are zeros, which their zero probabilities multiply
      for (int i = tid; i < ((nk + 15) & ~15) * VECS; i += kThreads) {
        const int r = i / VECS, c = i % VECS;
        cp_async16(uV + (r * C::PITCH + c * 8) * 2, vp + 1LL * (kv0 + min(r, nk - 1)) * a.ld + c * 8, r < nk);
      }
      const int new_q = kv0 == 0 ? nq : 0;   // rows of q, then rows of k
      if constexpr (ROPE) {
        for (int u0 = 0; u0 < new_q + nk; u0 += GROUPS * UB) {
          uint4 raw[UB][2];
#pragma unroll
          for (int j = 0; j < UB; ++j) {
            const int u = u0 + j * GROUPS + g;
            const int row = u < new_q + nk ? row_of(u, new_q, q0, kv0) : kv0;
            const bf16* src = (u < new_q ? qp : kp) + 1LL * row * a.ld + lg * 8;
            raw[j][0] = ld16(src);
            raw[j][1] = ld16(src + HD / 2);
          }
          if (!ahead) angles(u0, new_q, new_q + nk, q0, kv0);
          ahead = false;
#pragma unroll
          for (int j = 0; j < UB; ++j) {
            const int u = u0 + j * GROUPS + g;
            f2 y[2][4];
            rope_head<HD>(raw[j], a.do_norm, swt + (u < new_q ? 0 : HD) + lg * 4, a.eps, cs[j], sn[j], y,
                          [](float) {});
            if (u < new_q + nk) {
              bf16* dst = u < new_q ? sQ + u * C::PITCH : sK + (u - new_q) * C::PITCH;
              st16(dst + lg * 8, pack8(y[0]));
              st16(dst + HD / 2 + lg * 8, pack8(y[1]));
            }
          }
        }
      } else {
        for (int i = tid; i < (new_q + nk) * VECS; i += kThreads) {
          const int u = i / VECS, c = i % VECS;
          const bool is_q = u < new_q;
          const int r = is_q ? u : u - new_q;
          cp_async16((is_q ? uQ : uK) + (r * C::PITCH + c * 8) * 2,
                     (is_q ? qp + 1LL * (q0 + r) * a.ld : kp + 1LL * (kv0 + r) * a.ld) + c * 8, true);
        }
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();
      if (row0 >= nq) continue;

      // scores of 16 rows x 16 columns at a time; columns that no row of the warp sees are left out
      const int cols = a.causal ? min(nk, q0 + row0 + 16 - kv0) : nk;
      float s[4][2][4];
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
          for (int e = 0; e < 4; ++e) s[p][t][e] = 0.f;
#pragma unroll
      for (int ks = 0; ks < HD / 16; ++ks) {
        uint32_t qa[4];
        ldsm4(uQ + ((row0 + (lane & 15)) * C::PITCH + ks * 16 + (lane >> 4) * 8) * 2, qa);
#pragma unroll
        for (int p = 0; p < 4; ++p)
          if (p * 16 < cols) {
            uint32_t kb[4];
            ldsm4(uK + ((p * 16 + (lane & 7) + (lane >> 4) * 8) * C::PITCH + ks * 16 +
                        ((lane >> 3) & 1) * 8) * 2, kb);
            mma16816(s[p][0], qa, kb[0], kb[1]);
            mma16816(s[p][1], qa, kb[2], kb[3]);
          }
      }
      float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int col = kv0 + p * 16 + t * 8 + (lane & 3) * 2 + (e & 1);
            const int row = q0 + row0 + (lane >> 2) + (e >> 1) * 8;
            const bool valid = col < len && (!a.causal || col <= row);
            s[p][t][e] = valid ? s[p][t][e] * a.scale_log2 : -INFINITY;
            mx[e >> 1] = fmaxf(mx[e >> 1], s[p][t][e]);
          }
      float alpha[2], use[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 1));
        mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 2));
        const float now = fmaxf(m[i], mx[i]);
        use[i] = now == -INFINITY ? 0.f : now;
        alpha[i] = exp2f(m[i] - use[i]);
        m[i] = now;
        l[i] *= alpha[i];
      }
      uint32_t pa[4][4];
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int t = 0; t < 2; ++t) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            s[p][t][e] = exp2f(s[p][t][e] - use[e >> 1]);
            l[e >> 1] += s[p][t][e];
          }
          pa[p][2 * t] = bf16_of_f2(f2_of(s[p][t][0], s[p][t][1]));
          pa[p][2 * t + 1] = bf16_of_f2(f2_of(s[p][t][2], s[p][t][3]));
        }
      if (kv0 > 0) {
#pragma unroll
        for (int i = 0; i < COLS / 8; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) o[i][e] *= alpha[e >> 1];
      }
#pragma unroll
      for (int p = 0; p < 4; ++p)
        if (p * 16 < cols) {
#pragma unroll
          for (int d = 0; d < COLS / 16; ++d) {
            uint32_t vb[4];
            ldsm4_t(uV + ((p * 16 + (lane & 15)) * C::PITCH + col0 + d * 16 + (lane >> 4) * 8) * 2, vb);
            mma16816(o[2 * d], pa[p], vb[0], vb[1]);
            mma16816(o[2 * d + 1], pa[p], vb[2], vb[3]);
          }
        }
    }

    if (row0 < nq) {
      float inv[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1);
        l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
        inv[i] = l[i] > 0.f ? 1.f / l[i] : 0.f;
      }
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int r = row0 + (lane >> 2) + k * 8;
        if (r < nq) {
          bf16* dst = a.O + (1LL * seq0 + q0 + r) * a.ldo + h * HD + col0 + (lane & 3) * 2;
#pragma unroll
          for (int i = 0; i < COLS / 8; ++i)
            *reinterpret_cast<uint32_t*>(dst + i * 8) =
                bf16_of_f2(f2_of(o[i][2 * k] * inv[k], o[i][2 * k + 1] * inv[k]));
        }
      }
    }
  }
}

template <int HD, bool ROPE, int WARPS>
int run_short(const ShortArgs& a, unsigned ctas, cudaStream_t st) {
  auto kern = attn_short_kernel<HD, ROPE, WARPS>;
  static const bool ready = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 ShortCfg<HD>::SMEM_BYTES) == cudaSuccess;
  if (!ready) return -10;
  return launch_pdl(kern, dim3(ctas), dim3(WARPS * 32), ShortCfg<HD>::SMEM_BYTES, st, pdl_enabled(), 1, a);
}

// Eight warps share a CTA's rotations and outputs, where those are what takes the time or SMs are idle anyway;
// else four, of which more CTAs fit (3072 CTAs of 24 tokens without rotation: 38 us with eight, 22 with
// four; 96 CTAs: 4.0 and 4.7).
template <int HD>
int run_short_hd(const ShortArgs& a, unsigned ctas, cudaStream_t st) {
  if (a.cos != nullptr) return run_short<HD, true, 8>(a, ctas, st);
  return int(ctas) <= row_num_sms() ? run_short<HD, false, 8>(a, ctas, st) : run_short<HD, false, 4>(a, ctas, st);
}

}  // namespace
}  // namespace lb

using namespace lb;

// Whether B sequences of at most max_len tokens are faster this way than through the rotation's launch
// and the tile kernels. With rotation the CTA of each query head rotates the keys of its group again, so only
// while the CTAs fill one wave. Of longer sequences several CTAs rotate, or read, the same keys.
// Measured (us a call, rotation and tile kernels / here):
//   16 + 8 heads of 128:  1 x 24 tokens 10.1 / 6.3, 1 x 64 11.9 / 8.3, 16 x 24 11.5 / 8.0, 16 x 64 13.8 / 11.0,
//                         64 x 24 20.0 / 24.2; 4 x 128 14.5 / 12.7, 16 x 128 18.2 / 27.3, 1 x 256 16.2 / 20.7
//   32 + 8 heads of 64:   4 x 64 11.3 / 6.0, 16 x 64 (512 CTAs) 12.9 / 13.2
//   32 + 8 heads of 128:  4 x 64 13.9 / 8.6, 16 x 24 12.5 / 14.2; 4 x 128 15.4 / 17.1
//   12 heads of 64, none: 1 x 24 6.5 / 3.9, 16 x 24 8.4 / 4.3, 256 x 24 43 / 20, 256 x 64 45 / 34;
//                         16 x 128 9.9 / 8.9, 64 x 128 20 / 25
// (In a model 65 to 128 tokens gain nothing either way: 3 of up to 120 on 28 layers 1974 / 1967 - 2023.)
extern "C" int lb_attn_short_ok(int B, int max_len, int Hq, int Hk, int hd, int rotation) {
  if (B <= 0 || max_len <= 0 || Hk <= 0 || Hq % Hk != 0 || (hd != 64 && hd != 128)) return 0;
  const int G = Hq / Hk;   // (as of lb_attn_fwd)
  if (G != 1 && G != 2 && G != 4 && G != 8) return 0;
  const long long ctas = 1LL * B * Hq;
  return max_len <= kShortRows && (rotation ? ctas <= 2 * row_num_sms() : ctas < (1LL << 31));
}

// q, k, v: [T, heads, hd], rows ld elements apart, as a projection leaves them; cos, sin (null: no rotation)
// and qw, kw (null: no norm) as of lb_qk_norm_rope_fwd. Sequences as of lb_attn_fwd; plan: any of theirs, for the
// rows that belong to none. max_len: of the sequences; longer ones cost time, not results.
extern "C" int lb_attn_short(const void* q, const void* k, const void* v, long long ld, const void* qw,
                             const void* kw, const float* cos, const float* sin, const void* pos, int pos_i64,
                             const int* seq_start, const int* seq_end, const int* plan, int capacity, void* o,
                             long long ldo, int T, int B, int max_len, int Hq, int Hk, int hd, float eps,
                             float w_off, float softmax_scale, int causal, void* stream) {
  if (T <= 0 || B <= 0) return 0;
  if (Hk <= 0 || Hq % Hk != 0 || ((ld | ldo) & 7) || (hd != 64 && hd != 128) || max_len <= 0) return -3;
  if ((cos == nullptr) != (sin == nullptr) || (cos != nullptr && pos == nullptr)) return -3;
  if ((qw == nullptr) != (kw == nullptr) || (qw != nullptr && cos == nullptr)) return -3;
  const int blocks = (max_len + kShortRows - 1) / kShortRows;
  if (1LL * B * Hq * blocks >= (1LL << 31)) return -3;
  ShortArgs a{(const bf16*)q, (const bf16*)k, (const bf16*)v, ld, (const bf16*)qw, (const bf16*)kw, cos, sin,
              pos, pos_i64, seq_start, seq_end, plan, capacity, (bf16*)o, ldo, T, Hq, Hk, blocks, eps, w_off,
              softmax_scale * kLog2eF, qw != nullptr, causal};
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const unsigned ctas = unsigned(B) * Hq * blocks;
  return hd == 128 ? run_short_hd<128>(a, ctas, st) : run_short_hd<64>(a, ctas, st);
}
