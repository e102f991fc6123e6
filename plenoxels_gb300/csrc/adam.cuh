// One Adam update of a grid cell (torch.optim.Adam, no weight decay, no amsgrad), shared by the
// optimiser passes (optim.cu) and the pooled gradient's update (pool.cu).
#pragma once

#include <cmath>

#include "pgb_device.cuh"

namespace pgb {

struct AdamConst {
  float one_minus_b1, b2, one_minus_b2, step_size, inv_bc2_sqrt, eps;
  int rest_stays;  // a cell with gradient and moments 0 keeps its value (adam_const)
};

__device__ __forceinline__ float adam_one(float& p, float g, float& m, float& s, const AdamConst& k) {
  m = m + k.one_minus_b1 * (g - m);        // exp_avg.lerp_(grad, 1 - beta1)
  s = s * k.b2 + k.one_minus_b2 * g * g;   // exp_avg_sq.mul_(beta2).addcmul_(grad, grad, 1 - beta2)
  const float denom = sqrtf(s) * k.inv_bc2_sqrt + k.eps;
  p = p - k.step_size * (m / denom);
  return fabsf(g);
}

// Updates the four channels of a cell; returns |g|.
__device__ __forceinline__ float4 adam_cell(float4& p, const float4& g, float4& m, float4& s,
                                            const AdamConst& k) {
  float4 a;
  a.x = adam_one(p.x, g.x, m.x, s.x, k);
  a.y = adam_one(p.y, g.y, m.y, s.y, k);
  a.z = adam_one(p.z, g.z, m.z, s.z, k);
  a.w = adam_one(p.w, g.w, m.w, s.w, k);
  return a;
}

__device__ __forceinline__ bool any_nonzero(const float4& v) {
  return v.x != 0.f || v.y != 0.f || v.z != 0.f || v.w != 0.f;  // true for NaN
}

__device__ __forceinline__ float4 add4(const float4& a, const float4& b) {
  return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}

inline AdamConst adam_const(double lr, double beta1, double beta2, double eps, int64_t step) {
  // torch.optim.Adam (non-capturable path): bias corrections in double on the host
  const double bc1 = 1.0 - std::pow(beta1, (double)step);
  const double bc2 = 1.0 - std::pow(beta2, (double)step);
  AdamConst k;
  k.one_minus_b1 = (float)(1.0 - beta1);
  k.b2 = (float)beta2;
  k.one_minus_b2 = (float)(1.0 - beta2);
  k.step_size = (float)(lr / bc1);
  k.inv_bc2_sqrt = (float)(1.0 / std::sqrt(bc2));
  k.eps = (float)eps;
  // 0 * x and 0 / eps are 0 unless a constant is infinite, NaN or eps is 0
  k.rest_stays = std::isfinite(k.one_minus_b1) && std::isfinite(k.b2) && std::isfinite(k.one_minus_b2) &&
                 std::isfinite(k.step_size) && std::isfinite(k.inv_bc2_sqrt) && std::isfinite(k.eps) &&
                 k.eps > 0.f;
  return k;
}

}  // namespace pgb
