// Activations of the elementwise kernels and of epilogues, in fp32.
#pragma once
#include "common.cuh"

CB_DEVICE float silu_f(float x) { return x / (1.f + __expf(-x)); }
CB_DEVICE float sigmoid_f(float x) { return 1.f / (1.f + __expf(-x)); }
CB_DEVICE float gelu_tanh_f(float x) {
  const float k = 0.7978845608028654f;
  return 0.5f * x * (1.f + tanhf(k * (x + 0.044715f * x * x * x)));
}
CB_DEVICE float gelu_tanh_grad_f(float x) {
  const float k = 0.7978845608028654f;
  const float t = tanhf(k * (x + 0.044715f * x * x * x));
  return 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * k * (1.f + 3.f * 0.044715f * x * x);
}
CB_DEVICE float gelu_erf_f(float x) { return 0.5f * x * (1.f + erff(x * 0.7071067811865476f)); }
CB_DEVICE float gelu_erf_grad_f(float x) {
  return 0.5f * (1.f + erff(x * 0.7071067811865476f)) + x * 0.3989422804014327f * __expf(-0.5f * x * x);
}

// ACT: 0 silu, 1 gelu (tanh), 2 gelu (erf), 3 squared relu
template <int ACT> CB_DEVICE float act_f(float x) {
  if (ACT == 3) { const float r = fmaxf(x, 0.f); return r * r; }
  return ACT == 0 ? silu_f(x) : (ACT == 1 ? gelu_tanh_f(x) : gelu_erf_f(x));
}
template <int ACT> CB_DEVICE float act_grad_f(float x) {
  if (ACT == 3) return 2.f * fmaxf(x, 0.f);
  if (ACT == 0) { const float s = sigmoid_f(x); return s * (1.f + x * (1.f - s)); }
  return ACT == 1 ? gelu_tanh_grad_f(x) : gelu_erf_grad_f(x);
}
