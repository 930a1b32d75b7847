// What the k-means kernels share: the cosine distance (kmeans.cu, kmeans_tc.cuh), and a fit's state and fixed-point sums (kmeans_fit.cu,
// kmeans_tc.cuh).
#pragma once
#include "common.cuh"

namespace f2c {

// one expression for all exact scorers: labels must not depend on which of them assigned a point
__device__ __forceinline__ float finish_cosine(float dot, float xx, float cc) {
  float den = sqrtf(xx) * sqrtf(cc);
  return den > 0.0f ? 1.0f - dot / den : 1.0f;
}

struct FitState {       // first 256 bytes of the workspace; the host reads the first four words
  int32_t done;
  int32_t iterations;
  int32_t not_finite;   // the data hold inf or NaN: nothing is iterated, the caller says so
  int32_t assign_error; // code of the last bounded wait of the tensor-core kernel that ran out (the exact scorer then assigned every point)
  uint32_t pad;
  uint32_t arrived;
  double shift;
};

constexpr int kFitMaxCtas = 256;  // of the cooperative kernel: what a workspace has room for, whatever device was current when its size was asked for

// Sums are exact and independent of the order of the additions: a value becomes a fixed-point integer, this many bits below the largest
// magnitude of its column, and integers commute.
__device__ __forceinline__ int fraction_bits(int64_t n) {
  const int lg = 64 - __clzll((unsigned long long)n);  // 2^lg > n
  return min(43, 61 - lg);
}

// |x| <= 2^e for the float with these bits; a value of the column becomes an integer multiple of 2^(e - bits)
__device__ __forceinline__ int exponent(uint32_t max_bits) { return max_bits == 0u ? 0 : (int)(max_bits >> 23) - 126; }
__device__ __forceinline__ double power2(int e) { return __hiloint2double((1023 + e) << 20, 0); }  // |e| < 1023

}  // namespace f2c
