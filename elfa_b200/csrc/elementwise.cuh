// The elementwise operations by number (elementwise.cu; decode.cu applies the activations while it reads).
#pragma once
#include "common.cuh"

namespace elfa {

enum { OP_GELU = 0, OP_GELU_BWD = 1, OP_ADD = 2, OP_MUL = 3, OP_SILU = 4, OP_SILU_BWD = 5, OP_RELU = 6, OP_RELU_BWD = 7,
       OP_GELU_ERF = 8, OP_GELU_ERF_BWD = 9, OP_SCALE = 10 };

template <int OP>
__device__ __forceinline__ float apply(float a, float b, float alpha) {
  if (OP == OP_GELU) return gelu_tanh(a);
  if (OP == OP_GELU_BWD) return b * dgelu_tanh(a);  // a = pre-activation, b = upstream gradient
  if (OP == OP_ADD) return a + alpha * b;
  if (OP == OP_MUL) return a * b;
  if (OP == OP_SILU) return a / (1.f + __expf(-a));
  if (OP == OP_SILU_BWD) {
    const float s = 1.f / (1.f + __expf(-a));
    return b * s * (1.f + a * (1.f - s));
  }
  if (OP == OP_RELU) return fmaxf(a, 0.f);
  if (OP == OP_RELU_BWD) return a > 0.f ? b : 0.f;
  if (OP == OP_GELU_ERF) return 0.5f * a * (1.f + erff(a * 0.7071067811865476f));
  if (OP == OP_GELU_ERF_BWD) {
    const float cdf = 0.5f * (1.f + erff(a * 0.7071067811865476f));
    const float pdf = 0.3989422804014327f * __expf(-0.5f * a * a);
    return b * (cdf + a * pdf);
  }
  if (OP == OP_SCALE) return a * alpha;
  return a;
}

}  // namespace elfa
