// Dynamic-scaling casts from bf16 to 8-bit floats (e4m3 / e5m2) for the kind::f8f6f4 GEMM.
//
// Two kernels:
//   fp8_amax_kernel  max |x| per tensor, per row or per column (bit pattern of a non-negative
//                    float, reduced with integer atomicMax)
//   fp8_cast_kernel  q = sat(x * fmax / amax) as 8-bit floats, written row-major and / or transposed
//                    (the GEMM wants both operands K-major, so the products of the backward pass read
//                    transposed copies), plus the dequantisation factors amax / fmax.
//
// Takes the place of torchao's float8 cast kernels behind the reference's FP8 training switch
// (lset/train/quantization/fp8.py:11-45).
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace lb {
namespace {

constexpr float kAmaxFloor = 1e-12f;

__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// MODE 0: one value for the tensor; 1: one per row; 2: one per column.
// Block: 256 threads over a 64-row x 256-column tile; lane = 8 consecutive columns. Bound by memory: the
// loads of a thread's eight rows are requested together.
// Measured with four rows a thread / eight (us, L2 flushed): 21760 x 19456 160 / 137 (94 % of copy
// bandwidth), 21760 x 2560 36 / 29, 2560 x 2560 12 / 11.
constexpr int kAmaxRows = 8;  // a warp
template <int MODE>
__global__ void __launch_bounds__(256) fp8_amax_kernel(const __nv_bfloat16* __restrict__ x, int R,
                                                       int C, long long ldx,
                                                       unsigned* __restrict__ out) {
  __shared__ unsigned s_col[256];
  __shared__ unsigned s_warp[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c0 = blockIdx.x * 256 + lane * 8;
  const int r0 = (blockIdx.y * 8 + warp) * kAmaxRows;
  if (MODE == 2) s_col[threadIdx.x] = 0u;
  if (MODE == 2) __syncthreads();
  float cm[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  float tmax = 0.f;
  uint4 q[kAmaxRows];
#pragma unroll
  for (int i = 0; i < kAmaxRows; ++i)
    q[i] = r0 + i < R && c0 < C ? *reinterpret_cast<const uint4*>(x + (long long)(r0 + i) * ldx + c0)
                                : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
  for (int i = 0; i < kAmaxRows; ++i) {
    const int r = r0 + i;
    float rm = 0.f;
    {
      const uint32_t w[4] = {q[i].x, q[i].y, q[i].z, q[i].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float a = fabsf(bf16_lo(w[j])), b = fabsf(bf16_hi(w[j]));
        cm[2 * j] = fmaxf(cm[2 * j], a);
        cm[2 * j + 1] = fmaxf(cm[2 * j + 1], b);
        rm = fmaxf(rm, fmaxf(a, b));
      }
    }
    if (MODE == 1) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) rm = fmaxf(rm, __shfl_xor_sync(0xffffffffu, rm, o));
      if (lane == 0 && r < R && rm > 0.f) atomicMax(out + r, __float_as_uint(rm));
    }
    tmax = fmaxf(tmax, rm);
  }
  if (MODE == 0) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, o));
    if (lane == 0) s_warp[warp] = __float_as_uint(tmax);
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned m = 0u;
      for (int i = 0; i < 8; ++i) m = max(m, s_warp[i]);
      if (m > 0u) atomicMax(out, m);
    }
  }
  if (MODE == 2) {
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (cm[j] > 0.f) atomicMax(&s_col[lane * 8 + j], __float_as_uint(cm[j]));
    __syncthreads();
    const int c = blockIdx.x * 256 + threadIdx.x;
    if (c < C && s_col[threadIdx.x] > 0u) atomicMax(out + c, s_col[threadIdx.x]);
  }
}

template <int E5M2>
__device__ __forceinline__ uint32_t cvt4(float a, float b, float c, float d) {
  constexpr __nv_fp8_interpretation_t kind = E5M2 ? __NV_E5M2 : __NV_E4M3;
  const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, kind);
  const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(c, d), __NV_SATFINITE, kind);
  return lo | (hi << 16);
}

// The bytes of four words of a 4 x 4 block, transposed.
__device__ __forceinline__ void transpose4(uint32_t (&w)[4]) {
  const uint32_t ab0 = __byte_perm(w[0], w[1], 0x5140), ab1 = __byte_perm(w[0], w[1], 0x7362);
  const uint32_t cd0 = __byte_perm(w[2], w[3], 0x5140), cd1 = __byte_perm(w[2], w[3], 0x7362);
  w[0] = __byte_perm(ab0, cd0, 0x5410);
  w[1] = __byte_perm(ab0, cd0, 0x7632);
  w[2] = __byte_perm(ab1, cd1, 0x5410);
  w[3] = __byte_perm(ab1, cd1, 0x7632);
}

// Block: 256 threads over a 128 x 128 tile. Scale of element (r, c): fmax / max(amax, floor) with
// amax per tensor (MODE 0), per row (1) or per column (2).
//
// Bound by memory. A thread casts two blocks of four rows and eight columns and transposes each in registers;
// the words, four rows of a column, go through shared memory, so that either output is written in
// pieces of 128 bytes. Word `rg` of a column of group cg lies at rg ^ 2 cg: the words that a warp writes at a time are
// in different banks, and four of a column stay together for the 16-byte reads.
// Measured with 64 x 64 tiles, transposed byte by byte / here (us, both outputs, L2 flushed): 21760 x 19456
// 348 / 271 (95 % of copy bandwidth), 21760 x 6144 117 / 90, 19456 x 2560 49 / 39, 2560 x 2560 14 / 12.
constexpr int kCastTile = 128;
template <int MODE, int E5M2>
__global__ void __launch_bounds__(256)
    fp8_cast_kernel(const __nv_bfloat16* __restrict__ x, int R, int C, long long ldx,
                    const unsigned* __restrict__ amax, uint8_t* __restrict__ out, long long ldo,
                    uint8_t* __restrict__ out_t, long long ldt, float* __restrict__ inv_scale) {
  constexpr float kFmax = E5M2 ? 57344.f : 448.f;
  __shared__ __align__(16) uint32_t tile[kCastTile * kCastTile / 4];  // [column][four rows]
  __shared__ float s_scale[kCastTile];
  const int r0 = blockIdx.y * kCastTile, c0 = blockIdx.x * kCastTile;
  const int cg = threadIdx.x & 15, c = c0 + cg * 8;
  uint4 v[2][4];
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = r0 + (threadIdx.x >> 4) * 4 + u * 64 + i;
      v[u][i] = r < R && c < C ? *reinterpret_cast<const uint4*>(x + (long long)r * ldx + c)
                               : make_uint4(0u, 0u, 0u, 0u);
    }
  if (threadIdx.x < kCastTile) {
    float am;
    if (MODE == 0) {
      am = __uint_as_float(amax[0]);
    } else if (MODE == 1) {
      am = (r0 + threadIdx.x < R) ? __uint_as_float(amax[r0 + threadIdx.x]) : 1.f;
    } else {
      am = (c0 + threadIdx.x < C) ? __uint_as_float(amax[c0 + threadIdx.x]) : 1.f;
    }
    am = fmaxf(am, kAmaxFloor);
    s_scale[threadIdx.x] = kFmax / am;
    if (inv_scale != nullptr) {
      if (MODE == 0) {
        if (threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0) inv_scale[0] = am / kFmax;
      } else if (MODE == 1) {
        if (blockIdx.x == 0 && r0 + threadIdx.x < R) inv_scale[r0 + threadIdx.x] = am / kFmax;
      } else {
        if (blockIdx.y == 0 && c0 + threadIdx.x < C) inv_scale[c0 + threadIdx.x] = am / kFmax;
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int rg = (threadIdx.x >> 4) + u * 16;
    uint32_t q[2][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int lr = rg * 4 + i;
      const uint32_t w[4] = {v[u][i].x, v[u][i].y, v[u][i].z, v[u][i].w};
      float f[8];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        f[j] = (j & 1 ? bf16_hi(w[j / 2]) : bf16_lo(w[j / 2])) *
               s_scale[MODE == 2 ? cg * 8 + j : (MODE == 1 ? lr : 0)];
      const bool inside = r0 + lr < R && c < C;
      q[0][i] = inside ? cvt4<E5M2>(f[0], f[1], f[2], f[3]) : 0u;
      q[1][i] = inside ? cvt4<E5M2>(f[4], f[5], f[6], f[7]) : 0u;
      if (out != nullptr && inside)
        *reinterpret_cast<uint2*>(out + (long long)(r0 + lr) * ldo + c) = make_uint2(q[0][i], q[1][i]);
    }
    if (out_t != nullptr) {
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        transpose4(q[k]);
#pragma unroll
        for (int j = 0; j < 4; ++j) tile[(cg * 8 + k * 4 + j) * 32 + (rg ^ (2 * cg))] = q[k][j];
      }
    }
  }
  if (out_t == nullptr) return;
  __syncthreads();
  // row c of out_t holds column c of x: 16 rows of x a piece
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int tc = (threadIdx.x >> 3) + k * 32, m = threadIdx.x & 7, g = tc >> 3;
    uint4 w = *reinterpret_cast<const uint4*>(tile + tc * 32 + 4 * (m ^ (g >> 1)));
    if (g & 1) w = make_uint4(w.z, w.w, w.x, w.y);
    if (c0 + tc < C && r0 + m * 16 < ldt)
      *reinterpret_cast<uint4*>(out_t + (long long)(c0 + tc) * ldt + r0 + m * 16) = w;
  }
}

}  // namespace
}  // namespace lb

// max |x| of a bf16 matrix [R, C] (row stride ldx elements; C and ldx multiples of 8).
// mode 0: out[0]; 1: out[R]; 2: out[C]. `out` receives the bit patterns (zero where all zero).
extern "C" int lb_fp8_amax(const void* x, int R, int C, long long ldx, int mode, unsigned* out,
                           void* stream_) {
  using namespace lb;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (R <= 0 || C <= 0) return 0;
  if ((C & 7) || (ldx & 7) || mode < 0 || mode > 2) return -3;
  const size_t n = mode == 0 ? 1 : (mode == 1 ? size_t(R) : size_t(C));
  if (cudaMemsetAsync(out, 0, n * sizeof(unsigned), stream) != cudaSuccess) return -11;
  dim3 grid((C + 255) / 256, (R + 8 * kAmaxRows - 1) / (8 * kAmaxRows));
  const __nv_bfloat16* xp = reinterpret_cast<const __nv_bfloat16*>(x);
  if (mode == 0)
    fp8_amax_kernel<0><<<grid, 256, 0, stream>>>(xp, R, C, ldx, out);
  else if (mode == 1)
    fp8_amax_kernel<1><<<grid, 256, 0, stream>>>(xp, R, C, ldx, out);
  else
    fp8_amax_kernel<2><<<grid, 256, 0, stream>>>(xp, R, C, ldx, out);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

// Quantise x [R, C] with the maxima from lb_fp8_amax (same mode). out: [R, ldo] bytes (nullable),
// out_t: [C, ldt] bytes (nullable; ldt >= R and a multiple of 16, bytes past R are written as
// zero up to ldt), inv_scale: dequantisation factors (1, R or C floats; nullable).
extern "C" int lb_fp8_cast(const void* x, int R, int C, long long ldx, int mode,
                           const unsigned* amax, int e5m2, void* out, long long ldo, void* out_t,
                           long long ldt, float* inv_scale, void* stream_) {
  using namespace lb;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (R <= 0 || C <= 0) return 0;
  if ((C & 7) || (ldx & 7) || mode < 0 || mode > 2) return -3;
  if (out != nullptr && ((ldo & 7) || ldo < C)) return -3;
  if (out_t != nullptr && ((ldt & 15) || ldt < R)) return -3;
  dim3 grid((C + kCastTile - 1) / kCastTile, (R + kCastTile - 1) / kCastTile);
  const __nv_bfloat16* xp = reinterpret_cast<const __nv_bfloat16*>(x);
  uint8_t* o = reinterpret_cast<uint8_t*>(out);
  uint8_t* ot = reinterpret_cast<uint8_t*>(out_t);
#define LB_CAST(MODE, E)                                                                    \
  fp8_cast_kernel<MODE, E><<<grid, 256, 0, stream>>>(xp, R, C, ldx, amax, o, ldo, ot, ldt, \
                                                     inv_scale)
  if (e5m2) {
    if (mode == 0) LB_CAST(0, 1);
    else if (mode == 1) LB_CAST(1, 1);
    else LB_CAST(2, 1);
  } else {
    if (mode == 0) LB_CAST(0, 0);
    else if (mode == 1) LB_CAST(1, 0);
    else LB_CAST(2, 0);
  }
#undef LB_CAST
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}
