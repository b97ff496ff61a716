// Per-head RMSNorm and rotary embedding of one head by HD / 16 lanes: the arithmetic that the rotation's
// kernels and the attention of short sequences share.
#pragma once

#include "../common/row.cuh"

namespace lb {

__device__ __forceinline__ int rope_pos(const void* pos, int pos_i64, long long tok) {
  return pos_i64 ? int(reinterpret_cast<const long long*>(pos)[tok])
                 : reinterpret_cast<const int*>(pos)[tok];
}

// Where weight i of q's and k's 2 * HD is in shared memory: [q or k][half][4 of 8][lane][4], so that the
// lanes of a head read neighbouring 16 bytes (eight floats in a row a lane cost twice the banks).
template <int HD>
__device__ __forceinline__ int weight_at(int i) {
  constexpr int HALF = HD / 2, LPH = HD / 16;
  const int e = i % HD, c = e % HALF;
  return i - e + ((e / HALF * 2 + c % 8 / 4) * LPH + c / 8) * 4 + c % 4;
}

// The angles of a position (or zeros) for the eight elements from e0.
template <int HALF>
__device__ __forceinline__ void load_angles(const float* cos, const float* sin, int pos, int e0, f2 (&c)[4],
                                            f2 (&s)[4]) {
  float4 v[4] = {};
  if (pos >= 0) {
    const float4* cp = reinterpret_cast<const float4*>(cos + 1LL * pos * HALF + e0);
    const float4* sp = reinterpret_cast<const float4*>(sin + 1LL * pos * HALF + e0);
    v[0] = cp[0];
    v[1] = cp[1];
    v[2] = sp[0];
    v[3] = sp[1];
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    c[2 * i] = f2_of(v[i].x, v[i].y);
    c[2 * i + 1] = f2_of(v[i].z, v[i].w);
    s[2 * i] = f2_of(v[2 + i].x, v[2 + i].y);
    s[2 * i + 1] = f2_of(v[2 + i].z, v[2 + i].w);
  }
}
__device__ __forceinline__ f2 f2_neg(f2 v) { return v ^ 0x8000000080000000ull; }

// A lane's eight elements of either half of a head (`raw`) to their rotated values; `wt`: its first weight
// (see weight_at; only read with do_norm). All lanes of the warp call it. The head's rstd goes to `rstd_is`.
template <int HD, typename Rstd>
__device__ __forceinline__ void rope_head(const uint4 (&raw)[2], bool do_norm, const float* wt, float eps,
                                           const f2 (&c)[4], const f2 (&s)[4], f2 (&y)[2][4],
                                          Rstd rstd_is) {
  constexpr int LPH = HD / 16;
  f2 x[2][4];
  if (do_norm) {
    // element i of either half in one pair: two sums of squares, each in the order of its half
    const uint32_t lo[4] = {raw[0].x, raw[0].y, raw[0].z, raw[0].w};
    const uint32_t hi[4] = {raw[1].x, raw[1].y, raw[1].z, raw[1].w};
    f2 p[8], ss = 0ull;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      p[2 * i] = f2_of(__uint_as_float(lo[i] << 16), __uint_as_float(hi[i] << 16));
      p[2 * i + 1] = f2_of(__uint_as_float(lo[i] & 0xffff0000u), __uint_as_float(hi[i] & 0xffff0000u));
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) ss = f2_fma(p[i], p[i], ss);
    const float2 halves = f2_get(ss);
    float sum = halves.x + halves.y;
#pragma unroll
    for (int o = LPH / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float rstd = rsqrtf(sum / float(HD) + eps);
    rstd_is(rstd);
    const f2 r2 = f2_of(rstd, rstd);
#pragma unroll
    for (int q = 0; q < 2; ++q) {   // columns 4q .. 4q + 3 of either half
      float2 n[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) n[i] = f2_get(f2_mul(p[4 * q + i], r2));
      const float4 w0 = *reinterpret_cast<const float4*>(wt + q * LPH * 4);
      const float4 w1 = *reinterpret_cast<const float4*>(wt + (2 + q) * LPH * 4);
      x[0][2 * q] = f2_mul(f2_bf16_round(f2_of(n[0].x, n[1].x)), f2_of(w0.x, w0.y));
      x[0][2 * q + 1] = f2_mul(f2_bf16_round(f2_of(n[2].x, n[3].x)), f2_of(w0.z, w0.w));
      x[1][2 * q] = f2_mul(f2_bf16_round(f2_of(n[0].y, n[1].y)), f2_of(w1.x, w1.y));
      x[1][2 * q + 1] = f2_mul(f2_bf16_round(f2_of(n[2].y, n[3].y)), f2_of(w1.z, w1.w));
    }
  } else {
    unpack8(raw[0], x[0]);
    unpack8(raw[1], x[1]);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    y[0][i] = f2_fma(x[0][i], c[i], f2_neg(f2_mul(x[1][i], s[i])));
    y[1][i] = f2_fma(x[1][i], c[i], f2_mul(x[0][i], s[i]));
  }
}

}  // namespace lb
