// Gradient through dropout and ReLU, and the bias gradient behind them, in one pass: dy = active <= 0 ? 0 : g * keep * scale where active is
// what the ReLU gave and keep the mask (0 or 1) that dropout drew, db += column sums of dy.  The products and the comparison are
// torch's (native_dropout_backward, threshold_backward), so a NaN or an infinity goes where it goes there: a NaN activation passes
// its gradient, a dropped element of an infinite gradient is NaN.
// The output h behind both tells nearly always: h > 0 was kept, and where h = 0 a finite gradient ends whichever of the two made it
// zero.  Only a NaN in h, or a NaN or infinite gradient where h = 0, takes a look at keep and active.
// As torch operators this is a mask product, a ReLU backward and a vector-matrix product: 36 us for 59,000 x 128 on a B200.
// HBM bound: two matrices in, one out.  A thread keeps four columns for life, so its column sums stay in registers; a CTA adds
// them up in shared memory and to db once.  Elements that need the look are found by two multiply-adds each and put right in a second
// walk, so that the first keeps its 40 registers: 59,000 x 128 19.9 us, 59,392 x 256 37.6 (without the look 19.1 and 36.6; with keep
// and active read for every element 21.5 and 39.9).
#include "common.cuh"

namespace f2c {
namespace {

constexpr int kThreads = 256;
constexpr int kPartCols = 8192;  // columns whose sums a CTA holds; wider rows are cut into parts (grid.y)

struct Masked {
  const float* active;     // null: h itself
  const uint8_t* keep;     // null: all ones
  float scale;
  static __device__ __forceinline__ bool rare(float g, float h) { return h != h || (h == 0.f && !(fabsf(g) < INFINITY)); }
  __device__ __forceinline__ float often(float g, float h) const { return h > 0.f ? g * scale : 0.f; }  // 0 where rare
  __device__ __forceinline__ float look(float g, float h, int64_t at) const {
    if ((active != nullptr ? active[at] : h) <= 0.f) return 0.f;
    return g * (keep != nullptr ? (float)keep[at] : 1.f) * scale;
  }
};

// MASK = false: only the column sums of g
template <bool VEC, bool MASK>
__global__ void __launch_bounds__(kThreads) sage_mask_kernel(const float* __restrict__ g, const float* __restrict__ h, const Masked m,
                                                             float* __restrict__ dy, float* __restrict__ db, int64_t rows, int n) {
  dependency_wait();
  release_dependents();
  constexpr int E = VEC ? 4 : 1;
  extern __shared__ float sums[];
  const int col0 = (int)blockIdx.y * kPartCols;
  const int cols = min(n - col0, kPartCols), units = cols / E;
  for (int i = threadIdx.x; i < cols; i += kThreads) sums[i] = 0.0f;
  __syncthreads();
  const int lanes = units < kThreads ? kThreads / units : 1;  // rows a CTA works on at a time
  const int local = units < kThreads ? (int)threadIdx.x / units : 0;
  const int64_t step = (int64_t)gridDim.x * lanes;
  for (int u = units < kThreads ? (int)threadIdx.x - local * units : (int)threadIdx.x; u < units && local < lanes; u += kThreads) {
    float s[E] = {};
    const int at0 = col0 + u * E;
    const int64_t r0 = (int64_t)blockIdx.x * lanes + local;
    float finite = 0.f;  // NaN once an element was not: two additions of products with zero each
#pragma unroll 4
    for (int64_t r = r0; r < rows; r += step) {
      const int64_t at = r * n + at0;
      if (VEC) {
        float4 v = __ldcs(reinterpret_cast<const float4*>(g + at));
        if (MASK) {
          const float4 b = __ldcs(reinterpret_cast<const float4*>(h + at));
          finite = fmaf(v.x, 0.f, fmaf(v.y, 0.f, fmaf(v.z, 0.f, fmaf(v.w, 0.f, finite))));
          finite = fmaf(b.x, 0.f, fmaf(b.y, 0.f, fmaf(b.z, 0.f, fmaf(b.w, 0.f, finite))));
          v = make_float4(m.often(v.x, b.x), m.often(v.y, b.y), m.often(v.z, b.z), m.often(v.w, b.w));
          *reinterpret_cast<float4*>(dy + at) = v;
        }
        s[0] += v.x; s[E > 1 ? 1 : 0] += v.y; s[E > 2 ? 2 : 0] += v.z; s[E > 3 ? 3 : 0] += v.w;
      } else {
        float v = g[at];
        if (MASK) {
          const float b = h[at];
          finite = fmaf(v, 0.f, fmaf(b, 0.f, finite));
          v = m.often(v, b);
          dy[at] = v;
        }
        s[0] += v;
      }
    }
    if (MASK && finite != 0.f) {  // once more over the thread's elements, apart from the loop so that it costs that one nothing
#pragma unroll 1
      for (int64_t r = r0; r < rows; r += step)
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const int64_t at = r * n + at0 + e;
          const float v = g[at], b = h[at];
          if (Masked::rare(v, b)) s[e] += dy[at] = m.look(v, b, at);
        }
    }
    if (db != nullptr) {
#pragma unroll
      for (int e = 0; e < E; ++e) atomicAdd(sums + u * E + e, s[e]);
    }
    if (units < kThreads) break;
  }
  if (db == nullptr) return;
  __syncthreads();
  for (int i = threadIdx.x; i < cols; i += kThreads) atomicAdd(db + col0 + i, sums[i]);
}

}  // namespace
}  // namespace f2c

using namespace f2c;

extern "C" int f2c_sage_mask_dropout(const float* g, const float* h, const float* active, const uint8_t* keep, float scale, float* dy, float* db,
                                     int64_t rows, int64_t n, void* stream) {
  const char* op = "sage_mask";
  F2C_REQUIRE(rows >= 0 && n >= 0 && n <= 1 << 28, F2C_ERR_LIMIT, "%s: bad shape", op);
  if (rows * n == 0) return F2C_OK;
  F2C_REQUIRE(g && (h != nullptr ? dy != nullptr : db != nullptr), F2C_ERR_INVALID, "%s: null pointer", op);
  const bool vec = n % 4 == 0 && aligned(g, 16) && aligned(h, 16) && aligned(dy, 16);
  const int cols = (int)(n < kPartCols ? n : kPartCols), units = vec ? cols / 4 : cols;
  const int lanes = units < kThreads ? kThreads / units : 1;
  int64_t grid = ceil_div(rows, (int64_t)lanes * 4);
  if (grid > 8 * current_sm_count()) grid = 8 * current_sm_count();
  auto kern = h != nullptr ? (vec ? sage_mask_kernel<true, true> : sage_mask_kernel<false, true>)
                           : (vec ? sage_mask_kernel<true, false> : sage_mask_kernel<false, false>);
  launch_dependent(kern, dim3((unsigned)grid, (unsigned)ceil_div(n, kPartCols)), kThreads, (size_t)cols * 4, (cudaStream_t)stream, g, h,
                   Masked{active, keep, scale}, dy, db, rows, (int)n);
  return check_launch(op);
}

extern "C" int f2c_sage_mask(const float* g, const float* h, float scale, float* dy, float* db, int64_t rows, int64_t n, void* stream) {
  return f2c_sage_mask_dropout(g, h, nullptr, nullptr, scale, dy, db, rows, n, stream);
}

namespace f2c {
namespace {

constexpr int kMaxRanges = 32;
struct Ranges {
  uint32_t* at[kMaxRanges];
  int64_t words[kMaxRanges];
  int count;
};

__global__ void __launch_bounds__(256) zero_ranges_kernel(const Ranges r) {
  dependency_wait();
  release_dependents();
  for (int i = 0; i < r.count; ++i)
    for (int64_t w = (int64_t)blockIdx.x * 256 + threadIdx.x; w < r.words[i]; w += (int64_t)gridDim.x * 256) r.at[i][w] = 0u;
}

}  // namespace
}  // namespace f2c

extern "C" int f2c_zero_ranges(void* const* ranges_host, const int64_t* bytes_host, int count, void* stream) {
  const char* op = "zero_ranges";
  F2C_REQUIRE(count >= 0 && count <= kMaxRanges && (count == 0 || (ranges_host && bytes_host)), F2C_ERR_INVALID, "%s: at most %d ranges", op,
              kMaxRanges);
  Ranges r{};
  int64_t most = 0;
  for (int i = 0; i < count; ++i) {
    F2C_REQUIRE(bytes_host[i] >= 0 && bytes_host[i] % 4 == 0 && (bytes_host[i] == 0 || (ranges_host[i] && aligned(ranges_host[i], 4))),
                F2C_ERR_INVALID, "%s: ranges are whole, aligned words", op);
    if (bytes_host[i] == 0) continue;
    r.at[r.count] = (uint32_t*)ranges_host[i];
    r.words[r.count++] = bytes_host[i] / 4;
    if (bytes_host[i] / 4 > most) most = bytes_host[i] / 4;
  }
  if (r.count == 0) return F2C_OK;
  int64_t grid = ceil_div(most, 1024);
  if (grid > 2 * current_sm_count()) grid = 2 * current_sm_count();
  launch_dependent(zero_ranges_kernel, (unsigned)grid, 256, 0, (cudaStream_t)stream, r);
  return check_launch(op);
}
