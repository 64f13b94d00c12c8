// The AdamW step of one element, and of four neighbours, shared by the kernels that apply it.
#pragma once
#include "kernels.h"

namespace hipress {
namespace cuda {

__device__ __forceinline__ void adamw_one(const AdamWApply& a, float bc1, float rsqrt_bc2, float g,
                                          float& p, float& m, float& v) {
  p -= a.lr * a.weight_decay * p;  // decoupled weight decay
  m = a.beta1 * m + (1.0f - a.beta1) * g;
  v = a.beta2 * v + (1.0f - a.beta2) * g * g;
  const float denom = sqrtf(v) * rsqrt_bc2 + a.eps;
  p -= (a.lr / bc1) * (m / denom);
}

// Bias corrections of the step (read from the device when the step is replayed from a graph).
__device__ __forceinline__ void adamw_bias(const AdamWApply& a, float& bc1, float& rsqrt_bc2) {
  const float step = float(a.step_dev != nullptr ? int(*a.step_dev) : a.step);
  bc1 = 1.0f - powf(a.beta1, step);
  rsqrt_bc2 = 1.0f / sqrtf(1.0f - powf(a.beta2, step));
}

// Elements 4i .. 4i+3 of 16-byte aligned arrays.
__device__ __forceinline__ void adamw_four(const AdamWApply& a, float bc1, float rsqrt_bc2, int64_t i, float4 g4) {
  const float4 p4 = reinterpret_cast<const float4*>(a.param)[i];
  const float4 m4 = reinterpret_cast<const float4*>(a.exp_avg)[i];
  const float4 v4 = reinterpret_cast<const float4*>(a.exp_avg_sq)[i];
  const float g[4] = {g4.x, g4.y, g4.z, g4.w};
  float p[4] = {p4.x, p4.y, p4.z, p4.w};
  float m[4] = {m4.x, m4.y, m4.z, m4.w}, v[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) adamw_one(a, bc1, rsqrt_bc2, g[k], p[k], m[k], v[k]);
  reinterpret_cast<float4*>(a.exp_avg)[i] = make_float4(m[0], m[1], m[2], m[3]);
  reinterpret_cast<float4*>(a.exp_avg_sq)[i] = make_float4(v[0], v[1], v[2], v[3]);
  reinterpret_cast<float4*>(a.param)[i] = make_float4(p[0], p[1], p[2], p[3]);
}
__device__ __forceinline__ void adamw_at(const AdamWApply& a, float bc1, float rsqrt_bc2, int64_t i, float g) {
  float p = a.param[i], m = a.exp_avg[i], v = a.exp_avg_sq[i];
  adamw_one(a, bc1, rsqrt_bc2, g, p, m, v);
  a.exp_avg[i] = m;
  a.exp_avg_sq[i] = v;
  a.param[i] = p;
}

}  // namespace cuda
}  // namespace hipress
