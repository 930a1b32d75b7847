// Code of one element (reference: src/sq_quantization.cu:24-61), shared by sq_compress and by the compressor's fused
// encoder: the expression is the reference's, term by term, so codes carry the reference kernel's bits.
#pragma once
#include "common.cuh"

namespace f2c {

template <int BITS>
__device__ __forceinline__ float sq_encode(float x, const float* __restrict__ cb) {
  if (BITS == 1) return x <= 0.0f ? 0.0f : 1.0f;
  constexpr float drange = (float)(1 << (BITS - 1));
  float fmin = __ldg(cb + 0), fmax = __ldg(cb + 1), emin = __ldg(cb + 2), emax = __ldg(cb + 3);
  bool neg = x <= 0.0f;
  float v = fabsf(x);
  v = fminf(fmaxf(v, fmin), fmax);
  v = log2f(v);
  v = (v - emin) / (emax - emin) * drange;
  v = floorf(v);
  v = neg ? -1.0f - v : v;
  if (BITS < 8) v += drange;
  return v;
}

}  // namespace f2c
