// Lists of flat buffers for the optimiser kernels; see optim.cu.
#pragma once

extern "C" {

// Mirrored field by field in lset_b200/dist/sharded.py.
struct LbOptGroup {
  float* p;          // fp32 master weights
  float* g;          // fp32 gradients
  float* m;
  float* v;
  void* p_bf16;      // nullable: bf16 compute copy written after the update
  long long n;
  int slot;          // which of the two sums of squares the gradient belongs to
};
int lb_sumsq_scratch_floats(int count);
int lb_sumsq_groups(const LbOptGroup* groups, int count, float* scratch, float* out, void* stream);
int lb_adamw_groups(const LbOptGroup* groups, int count, float lr, float beta1, float beta2, float eps,
                    float wd, float bc1, float bc2_sqrt, float grad_scale, const float* coef,
                    int zero_grad, void* stream);

}  // extern "C"
