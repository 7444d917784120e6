// The Adam update of one parameter, shared by the kernels that apply it: the pass over flat buffers and
// the epilogue of the weight-gradient products.  Written out in fused multiply-adds, so that a
// parameter's new value does not depend on which of them made it.
#pragma once
#include <cuda_runtime.h>

namespace tp {

// p, m, v, model: fp32 master weights, moments and the 16-bit copy of one matrix or flat range.
struct AdamBuffers {
  float *p, *m, *v;
  void* model;
  const float* state;   // step count, 1 - beta1^t, 1 - beta2^t (adam_tick_kernel)
  float lr, beta1, beta2, eps, weight_decay, grad_scale;
};

struct AdamCoef {
  float step, inv_bc2_sqrt, decay, beta1, one_beta1, beta2, one_beta2, eps, grad_scale;
};

// (reads `state`: after the kernel has waited for its predecessor)
__device__ __forceinline__ AdamCoef adam_coef(const AdamBuffers& a) {
  AdamCoef c;
  c.step = a.lr / a.state[1];
  c.inv_bc2_sqrt = rsqrtf(a.state[2]);
  c.decay = a.lr * a.weight_decay;
  c.beta1 = a.beta1;
  c.one_beta1 = 1.0f - a.beta1;
  c.beta2 = a.beta2;
  c.one_beta2 = 1.0f - a.beta2;
  c.eps = a.eps;
  c.grad_scale = a.grad_scale;
  return c;
}

__device__ __forceinline__ void adam_update(float g, float& p, float& m, float& v, const AdamCoef& c) {
  const float gs = __fmul_rn(g, c.grad_scale);
  m = __fmaf_rn(c.beta1, m, __fmul_rn(c.one_beta1, gs));
  v = __fmaf_rn(c.beta2, v, __fmul_rn(__fmul_rn(c.one_beta2, gs), gs));
  const float denom = __fmaf_rn(sqrtf(v), c.inv_bc2_sqrt, c.eps);
  p = __fmaf_rn(-c.decay, p, __fmaf_rn(-c.step, m / denom, p));
}
__device__ __forceinline__ void adam_update(const float4& g, float4& p, float4& m, float4& v, const AdamCoef& c) {
  adam_update(g.x, p.x, m.x, v.x, c);
  adam_update(g.y, p.y, m.y, v.y, c);
  adam_update(g.z, p.z, m.z, v.z, c);
  adam_update(g.w, p.w, m.w, v.w, c);
}

}  // namespace tp
