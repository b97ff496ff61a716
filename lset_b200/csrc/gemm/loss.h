// Contrastive losses on the score product, forward and backward in one call each; see gemm_bf16.cu.
#pragma once

extern "C" {

// s = (q · kᵀ) * inv_temperature. Mirrored field by field in lset_b200/ops/loss.py.
//   InfoNCE (labels null): the positive of query r is passage r + target_offset; N a multiple of 8 in the
//     backward.
//     loss = loss_scale * sum_r (LSE_c s_rc − s_r,positive)
//     W[r, c] = (exp(s_rc − lse[r]) − [c is the positive]) * coef
//   label matrix: int8 labels [M, ld_labels] (ld_labels a multiple of 32, >= N, padded with a negative
//     value; < 0 ignored), t = tw (fp32 [M, ld_tw], same padding rule, zeros) or max(label, 0):
//     loss = loss_scale * sum_r row_w[r] · (LSE_{valid c} s_rc − row_scale[r] · sum_c t_rc s_rc)
//     W[r, c] = ([label_rc >= 0] · exp(s_rc − lse[r]) − row_scale[r] · t_rc) · row_w[r] · coef
//   loss_mode 1 (multi-positive NCE): lse[r] is the LSE over the negatives (label == 0) only and loss is
//     not meaningful, the caller forms it from lse and the positives' scores;
//     W: positives (sigmoid(s − lse) − 1) · row_w · coef, negatives exp(s − lse) · row_scale · row_w · coef
//   coef = grad[0] * grad_scale; dq = W · k, dk = Wᵀ · q.
struct LbLoss {
  const void* q;         // [M, D] bf16, rows ldq apart
  const void* k;         // [N, D] bf16, rows ldk apart
  long long ldq, ldk;
  int M, N, D;
  float inv_temperature;
  long long target_offset;
  const void* labels;
  long long ld_labels;
  const float* tw;
  long long ld_tw;
  const float* row_scale;
  const float* row_w;
  int loss_mode;
  float loss_scale;
  float* scratch;        // forward
  float* lse;            // [M], written by the forward and read by the backward
  float* loss;           // forward: device scalar, written
  const float* grad;     // backward: device scalar
  float grad_scale;
  int panel;             // columns of W
  void* W;               // [M, panel] bf16, rows ldw apart (a multiple of 8)
  long long ldw;
  void* dq;              // [M, D] bf16 (null: not wanted); with several panels the result is in dq32
  float* dq32;           // [M, D]
  void* dk;              // [N, D] bf16 or null
  int* status;
  void* stream;
};
int lb_loss_fwd(const LbLoss* p);
int lb_loss_bwd(const LbLoss* p);

}  // extern "C"
