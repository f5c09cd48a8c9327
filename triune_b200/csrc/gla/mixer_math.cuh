// Arithmetic of one token of a recurrent mixer, shared by the kernels that decode (mixer_step.cu and the one-launch step): each operation
// rounds in one way, whatever a compiler would contract around it, so that all of them give the same numbers.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>

#include "gla.cuh"

namespace tb {

__device__ __forceinline__ float mix_feature(float raw) { return raw > 0.f ? raw + 1.f : __expf(raw); }  // elu + 1
__device__ __forceinline__ float mix_decay(float logit) {
  return __expf(fmaxf(__fsub_rn(fminf(logit, 0.f), log1pf(__expf(-fabsf(logit)))), GLA_MIN_LOG_DECAY));
}
__device__ __forceinline__ float mix_inverse_norm(float squares) { return 1.f / fmaxf(sqrtf(squares), 1e-6f); }
// Half-split rotation of the first (or second) half's element f with its partner in the other half.
__device__ __forceinline__ float mix_rotate(float f, float partner, float cs, float sn, bool first) {
  const float other = __fmul_rn(partner, sn);
  return __fmaf_rn(f, cs, first ? -other : other);
}
__device__ __forceinline__ float mix_state(float s, float decay, float k, float u) { return __fmaf_rn(k, u, __fmul_rn(decay, s)); }
__device__ __forceinline__ float mix_strength(float logit) { return 1.f / (1.f + __expf(-logit)); }
// Eight terms of the write strength's product.
__device__ __forceinline__ float mix_dot8(const uint4& x, const uint4& w, float sum) {
  const uint32_t a[4] = {x.x, x.y, x.z, x.w}, b[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    sum = __fmaf_rn(__uint_as_float(a[j] << 16), __uint_as_float(b[j] << 16), sum);
    sum = __fmaf_rn(__uint_as_float(a[j] & 0xffff0000u), __uint_as_float(b[j] & 0xffff0000u), sum);
  }
  return sum;
}

}  // namespace tb
