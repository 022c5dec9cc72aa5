// One row of LayerNorm / RMSNorm from 16-byte vectors in registers (norm.cu; decode.cu normalises the few rows of a decoding step as it reads them).
#pragma once
#include "common.cuh"

namespace elfa {

__device__ __forceinline__ uint4 norm_add(const uint4& x, const uint4& r) {
  uint4 o;
  const uint32_t *px = reinterpret_cast<const uint32_t*>(&x), *pr = reinterpret_cast<const uint32_t*>(&r);
  uint32_t* po = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
  for (int j = 0; j < 4; ++j) po[j] = pack_bf16(bf16_lo(px[j]) + bf16_lo(pr[j]), bf16_hi(px[j]) + bf16_hi(pr[j]));
  return o;
}
// adds a vector's values and their squares
__device__ __forceinline__ void norm_sums(const uint4& x, float& s1, float& s2) {
  const uint32_t* pv = reinterpret_cast<const uint32_t*>(&x);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float a = bf16_lo(pv[j]), c = bf16_hi(pv[j]);
    s1 += a + c;
    s2 += a * a + c * c;
  }
}
template <bool RMS>
__device__ __forceinline__ void norm_moments(float s1, float s2, int D, float eps, float& mean, float& rstd) {
  const float inv_d = 1.0f / (float)D;
  mean = RMS ? 0.f : s1 * inv_d;
  float var = s2 * inv_d - mean * mean;
  var = fmaxf(var, 0.f);
  rstd = rsqrtf(var + eps);
}
__device__ __forceinline__ uint4 norm_scale(const uint4& x, float mean, float rstd, const uint4& w, const uint4& b) {
  uint4 o;
  const uint32_t *pv = reinterpret_cast<const uint32_t*>(&x), *pw = reinterpret_cast<const uint32_t*>(&w), *pb = reinterpret_cast<const uint32_t*>(&b);
  uint32_t* po = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float lo = (bf16_lo(pv[j]) - mean) * rstd * bf16_lo(pw[j]) + bf16_lo(pb[j]);
    const float hi = (bf16_hi(pv[j]) - mean) * rstd * bf16_hi(pw[j]) + bf16_hi(pb[j]);
    po[j] = pack_bf16(lo, hi);
  }
  return o;
}

}  // namespace elfa
