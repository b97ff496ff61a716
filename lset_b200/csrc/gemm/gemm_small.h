// Products whose 256 x 256 tiles leave most of the chip idle; see gemm_small.cu.
#pragma once

extern "C" {

// C = A · op(B) in bf16 x bf16 -> fp32 accumulation, for one to three weights side by side.
//   kParallelN  C[:, part p] = A · B_pᵀ          (projections of one input; part p has ext[p] columns)
//   kParallelK  C = sum_p A[:, part p] · B_p     (their input gradients; ext[p] columns of A; the
//               products are rounded to bf16 and added up in bf16, as launches of their own would)
//   kParallelM  C_p (+)= A[:, part p]ᵀ · B       (their weight gradients; ext[p] columns of A)
// a_mn / b_mn, leading dimensions and alignment as in lb_gemm_bf16.
struct LbSmallGemm {
  const void* A;
  const void* B[3];
  void* C[3];          // kParallelK: C[0] only
  long long lda, ldb[3], ldc[3];
  int M, N, K;         // extents of the whole product; the partitioned one is the sum of ext[]
  int ext[3];
  int nparts, mode;
  int a_mn, b_mn;
  int out_fp32;        // C is fp32, and the product is added to it (red.global.add)
  const void* bias[3]; // bf16, added to the columns of a part (kParallelN without glu_h); null: none
  // Gated pair (kParallelN, two parts of the same ext): also h = act(C_0) * C_1 [M, ext[0]], with both
  // factors rounded to bf16 first; C[0] == null leaves the products themselves unwritten.
  // glu_kind 2 (kParallelN, one part): h = GELU(C_0) [M, N], of the rounded product with its bias; C[0] == null
  // leaves that unwritten.
  void* glu_h;
  long long ld_h;
  int glu_kind;        // 0 = SiLU, 1 = tanh-GELU, 2 = GELU (erf) of one product
  // The B operands were complete before the kernel in front of this one on the stream began, so
  // their tiles may be requested while that kernel is still running.
  int b_ready;
  int may_split;       // the contraction may be summed in pieces (another order, another rounding)
  int bn, splits;      // 0 = chosen by lb_gemm_small_plan
  int* status;
  void* stream;
};

// From this many k-blocks of 64 on the tile kernels may add up a weight gradient in pieces.
enum { kLongSum = 64 };

// Modelled time of the product on this kernel and the tile width and split it would take (a negative
// value: not taken), and of one product on the CTA-pair kernel (fp32: a weight gradient, whose
// contraction that kernel splits; bias: the one-CTA kernel's, which adds it).
double lb_gemm_small_plan(const LbSmallGemm* p, int* bn, int* splits);
double lb_gemm_tile_cost(int M, int N, int K, int fp32, int bias);
int lb_gemm_small(const LbSmallGemm* p);
// The same, a bf16 result (not an activation's) rounded, multiplied by `scale` and rounded again; 0: not.
int lb_gemm_small_scaled(const LbSmallGemm* p, float scale);

}  // extern "C"

enum { kParallelN = 0, kParallelK = 1, kParallelM = 2 };
