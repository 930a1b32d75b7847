// Gradient through dropout and ReLU, and the bias gradient behind them, in one pass: dy = h > 0 ? scale * g : 0 where h is the
// layer's output after both (zero exactly where the ReLU or the dropout made it so), db += column sums of dy.  As torch
// operators this is a mask product, a ReLU backward and a vector-matrix product: 36 us for 59,000 x 128 on a B200.
// HBM bound: two matrices in, one out.  A thread keeps four columns for life, so its column sums stay in registers; a CTA adds
// them up in shared memory and to db once.  Measured: 16 us (5.7 TB/s).
#include "common.cuh"

namespace f2c {
namespace {

constexpr int kThreads = 256;

template <bool VEC>
__global__ void __launch_bounds__(kThreads) sage_mask_kernel(const float* __restrict__ g, const float* __restrict__ h, float scale,
                                                             float* __restrict__ dy, float* __restrict__ db, int64_t rows, int n, int units) {
  constexpr int E = VEC ? 4 : 1;
  extern __shared__ float sums[];
  for (int i = threadIdx.x; i < n; i += kThreads) sums[i] = 0.0f;
  __syncthreads();
  const int lanes = units < kThreads ? kThreads / units : 1;  // rows a CTA works on at a time
  const int local = units < kThreads ? (int)threadIdx.x / units : 0;
  const int64_t step = (int64_t)gridDim.x * lanes;
  for (int u = units < kThreads ? (int)threadIdx.x - local * units : (int)threadIdx.x; u < units && local < lanes; u += kThreads) {
    float s[E] = {};
    const int c = u * E;
#pragma unroll 4
    for (int64_t r = (int64_t)blockIdx.x * lanes + local; r < rows; r += step) {
      const int64_t at = r * n + c;
      if (VEC) {
        const float4 a = __ldcs(reinterpret_cast<const float4*>(g + at)), b = __ldcs(reinterpret_cast<const float4*>(h + at));
        const float4 v = make_float4(b.x > 0.f ? a.x * scale : 0.f, b.y > 0.f ? a.y * scale : 0.f, b.z > 0.f ? a.z * scale : 0.f,
                                     b.w > 0.f ? a.w * scale : 0.f);
        *reinterpret_cast<float4*>(dy + at) = v;
        s[0] += v.x; s[E > 1 ? 1 : 0] += v.y; s[E > 2 ? 2 : 0] += v.z; s[E > 3 ? 3 : 0] += v.w;
      } else {
        const float v = h[at] > 0.f ? g[at] * scale : 0.f;
        dy[at] = v;
        s[0] += v;
      }
    }
    if (db != nullptr) {
#pragma unroll
      for (int e = 0; e < E; ++e) atomicAdd(sums + c + e, s[e]);
    }
    if (units < kThreads) break;
  }
  if (db == nullptr) return;
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += kThreads) atomicAdd(db + i, sums[i]);
}

}  // namespace
}  // namespace f2c

using namespace f2c;

extern "C" int f2c_sage_mask(const float* g, const float* h, float scale, float* dy, float* db, int64_t rows, int64_t n, void* stream) {
  const char* op = "sage_mask";
  F2C_REQUIRE(rows >= 0 && n >= 0 && n <= 8192, F2C_ERR_LIMIT, "%s: bad shape", op);
  if (rows * n == 0) return F2C_OK;
  F2C_REQUIRE(g && h && dy, F2C_ERR_INVALID, "%s: null pointer", op);
  const bool vec = n % 4 == 0 && aligned(g, 16) && aligned(h, 16) && aligned(dy, 16);
  const int units = (int)(vec ? n / 4 : n);
  const int lanes = units < kThreads ? kThreads / units : 1;
  int64_t grid = ceil_div(rows, (int64_t)lanes * 4);
  if (grid > 8 * current_sm_count()) grid = 8 * current_sm_count();
  auto kern = vec ? sage_mask_kernel<true> : sage_mask_kernel<false>;
  kern<<<(unsigned)grid, kThreads, (size_t)n * 4, (cudaStream_t)stream>>>(g, h, scale, dy, db, rows, (int)n, units);
  return check_launch(op);
}
