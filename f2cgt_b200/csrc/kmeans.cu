// K-means distance matrix and assignment in fp32 CUDA cores
// (reference operators pairwise_distance / KMeans.predict, src/kmeans.cu:77-118, which wrap RAFT
// 23.10; semantics as restated by the reference in examples/my_kmeans.py:43-64,116-125):
//   L2      dist[i,c] = sum_t (x[i,t] - y[c,t])^2           (no square root)
//   cosine  dist[i,c] = 1 - <x_i, y_c> / (|x_i| |y_c|)      (1 when a norm is zero)
//   label[i] = first argmin_c dist[i,c]; a NaN distance counts as 1 (examples/my_kmeans.py:92-94)
//
// Two mappings:
//  * warp-per-point (any d, any k): lanes stride over the centres, x_i is broadcast; writes the
//    distance matrix with coalesced rows and/or reduces the argmin in the warp.  pairwise_distance is
//    bound by its n*k*4-byte output.
//  * thread-per-point (d <= 128): x_i lives in registers, centres are broadcast from shared memory
//    with 128-bit reads, four FMAs per read.  This is the exact fp32 scorer; the points whose best two
//    candidates are too close to call for the tensor-core kernel (kmeans_tc.cu) go through
//    kmeans_listed_kernel, which computes the same distances.
#include "kmeans_fit.cuh"

namespace f2c {

// ---------------------------------------------------------------- warp per point
template <int METRIC, bool WRITE_DIST, bool WRITE_LABEL>
__global__ void __launch_bounds__(256) kmeans_warp_kernel(const float* __restrict__ x, const float* __restrict__ y,
                                                          float* __restrict__ dist, int64_t* __restrict__ labels, int64_t n,
                                                          int k, int d, const int32_t* done) {
  dependency_wait();
  release_dependents();
  if (done != nullptr && *(volatile const int32_t*)done != 0) return;
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t i = warp; i < n; i += n_warps) {
    const float* xi = x + i * d;
    float xx = 0.0f;
    if (METRIC == F2C_COSINE)
      for (int t = 0; t < d; ++t) { float a = __ldg(xi + t); xx = fmaf(a, a, xx); }
    float best = INFINITY;
    int best_c = 0x7fffffff;
    for (int c = lane; c < k; c += 32) {
      const float* yc = y + (int64_t)c * d;
      float v;
      if (METRIC == F2C_L2) {
        float acc = 0.0f;
        for (int t = 0; t < d; ++t) { float df = __ldg(xi + t) - __ldg(yc + t); acc = fmaf(df, df, acc); }
        v = acc;
      } else {
        float dot = 0.0f, cc = 0.0f;
        for (int t = 0; t < d; ++t) { float a = __ldg(xi + t), b = __ldg(yc + t); dot = fmaf(a, b, dot); cc = fmaf(b, b, cc); }
        v = finish_cosine(dot, xx, cc);
      }
      if (WRITE_DIST) dist[i * k + c] = v;
      if (WRITE_LABEL) {
        if (v != v) v = 1.0f;
        if (v < best) { best = v; best_c = c; }
      }
    }
    if (WRITE_LABEL) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        float ob = __shfl_xor_sync(0xffffffffu, best, o);
        int oc = __shfl_xor_sync(0xffffffffu, best_c, o);
        if (ob < best || (ob == best && oc < best_c)) { best = ob; best_c = oc; }
      }
      if (lane == 0) labels[i] = best_c == 0x7fffffff ? 0 : best_c;
    }
  }
}

// ---------------------------------------------------------------- thread per point
// Centres are staged KC at a time as [KC][DMAX] (zero padded) plus their squared norms.
template <int DMAX, int METRIC>
__global__ void __launch_bounds__(256) kmeans_thread_kernel(const float* __restrict__ x, const float* __restrict__ y,
                                                            int64_t* __restrict__ labels, int64_t n, int k, int d, int kc,
                                                            const int32_t* done) {
  dependency_wait();
  release_dependents();
  if (done != nullptr && *(volatile const int32_t*)done != 0) return;  // a fit that has converged (kmeans_fit.cu)
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* yc_s = reinterpret_cast<float*>(smem_raw);  // [kc][DMAX]
  float* cc_s = yc_s + (size_t)kc * DMAX;            // [kc]
  for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < n; base += (int64_t)gridDim.x * blockDim.x) {
  const int64_t i = base + threadIdx.x;
  const bool valid = i < n;
  float xr[DMAX];
  float xx = 0.0f;
#pragma unroll
  for (int t = 0; t < DMAX; ++t) {
    xr[t] = (valid && t < d) ? __ldg(x + i * d + t) : 0.0f;
    if (METRIC == F2C_COSINE) xx = fmaf(xr[t], xr[t], xx);
  }
  float best = INFINITY;
  int best_c = 0;
  for (int c0 = 0; c0 < k; c0 += kc) {
    const int nc = min(kc, k - c0);
    __syncthreads();
    for (int e = threadIdx.x; e < nc * DMAX; e += blockDim.x) {
      int c = e / DMAX, t = e - c * DMAX;
      yc_s[e] = t < d ? __ldg(y + (int64_t)(c0 + c) * d + t) : 0.0f;
    }
    __syncthreads();
    if (METRIC == F2C_COSINE) {
      for (int c = threadIdx.x; c < nc; c += blockDim.x) {
        float cc = 0.0f;
        for (int t = 0; t < DMAX; ++t) cc = fmaf(yc_s[c * DMAX + t], yc_s[c * DMAX + t], cc);
        cc_s[c] = cc;
      }
      __syncthreads();
    }
    for (int c = 0; c < nc; ++c) {
      const float4* yc4 = reinterpret_cast<const float4*>(yc_s + (size_t)c * DMAX);
      float acc = 0.0f;
#pragma unroll
      for (int q = 0; q < DMAX / 4; ++q) {
        float4 b = yc4[q];
        if (METRIC == F2C_L2) {
          float d0 = xr[4 * q] - b.x, d1 = xr[4 * q + 1] - b.y, d2 = xr[4 * q + 2] - b.z, d3 = xr[4 * q + 3] - b.w;
          acc = fmaf(d0, d0, acc); acc = fmaf(d1, d1, acc); acc = fmaf(d2, d2, acc); acc = fmaf(d3, d3, acc);
        } else {
          acc = fmaf(xr[4 * q], b.x, acc); acc = fmaf(xr[4 * q + 1], b.y, acc);
          acc = fmaf(xr[4 * q + 2], b.z, acc); acc = fmaf(xr[4 * q + 3], b.w, acc);
        }
      }
      float v = METRIC == F2C_L2 ? acc : finish_cosine(acc, xx, cc_s[c]);
      if (v != v) v = 1.0f;
      if (v < best) { best = v; best_c = c0 + c; }
    }
  }
  if (valid) labels[i] = best_c;
  }
}

// ---------------------------------------------------------------- listed points
// Exact scores of the points the tensor-core kernel left undecided: a list whose length only the device knows, usually a
// few hundred points.  The centres are staged once per CTA (rows padded by 16 bytes: eight lanes that read one 16-byte
// piece of eight different centres touch eight bank groups).  A short list is worked one warp per point, lanes over the
// centres, so that its latency is k / 32 centres instead of k (256 centres of 32 dimensions: 17 us of dependent FMAs in one
// thread before); a list longer than the grid's warps could take in kShortRounds rounds goes one thread per point, where a
// centre is read once for 32 points.  Both add a centre's terms in the order of kmeans_thread_kernel: same distances.
constexpr int kListThreads = 256;
constexpr int kShortRounds = 32;

template <int DMAX, int METRIC>
__global__ void __launch_bounds__(kListThreads) kmeans_listed_kernel(const float* __restrict__ x, const float* __restrict__ y,
                                                                     int64_t* __restrict__ labels, const int32_t* __restrict__ list,
                                                                     const int32_t* __restrict__ count_dev, const int32_t* __restrict__ all_dev,
                                                                     int64_t max_count, int k, int d, int kc, int y_vec4, int y_settled) {
  constexpr int STRIDE = DMAX + 4;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* yc_s = reinterpret_cast<float*>(smem_raw);  // [kc][STRIDE]
  float* cc_s = yc_s + (size_t)kc * STRIDE;          // [kc]
  auto stage = [&](int c0, int nc) {
    if (y_vec4) {  // d % 4 == 0; eight 16-byte loads in flight per thread (single floats: 15 us for 256 x 64, now 8)
#pragma unroll 8
      for (int e = threadIdx.x; e < nc * (DMAX / 4); e += kListThreads) {
        const int c = e / (DMAX / 4), t = 4 * (e - c * (DMAX / 4));
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (t < d) v = __ldg(reinterpret_cast<const float4*>(y + (int64_t)(c0 + c) * d + t));
        *reinterpret_cast<float4*>(yc_s + c * STRIDE + t) = v;
      }
    } else {
#pragma unroll 8
      for (int e = threadIdx.x; e < nc * DMAX; e += kListThreads) {
        const int c = e / DMAX, t = e - c * DMAX;
        yc_s[c * STRIDE + t] = t < d ? __ldg(y + (int64_t)(c0 + c) * d + t) : 0.0f;
      }
    }
    __syncthreads();
    if (METRIC == F2C_COSINE) {
      for (int c = threadIdx.x; c < nc; c += kListThreads) {
        float cc = 0.0f;
#pragma unroll
        for (int t = 0; t < DMAX; ++t) cc = fmaf(yc_s[c * STRIDE + t], yc_s[c * STRIDE + t], cc);
        cc_s[c] = cc;
      }
      __syncthreads();
    }
  };
  if (kc >= k && y_settled) stage(0, k);  // while the kernel before, which makes the list, still runs
  dependency_wait();
  release_dependents();
  if (kc >= k && !y_settled) stage(0, k);
  const bool all = all_dev != nullptr && *all_dev != 0;  // every point instead of the listed ones
  const int64_t cnt = !all && *count_dev < max_count ? *count_dev : max_count;
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * kListThreads + threadIdx.x) >> 5, n_warps = ((int64_t)gridDim.x * kListThreads) >> 5;
  const bool by_warp = cnt <= n_warps * kShortRounds && kc >= k;
  if (by_warp ? (int64_t)blockIdx.x * (kListThreads / 32) >= cnt : (int64_t)blockIdx.x * kListThreads >= cnt) return;
  auto distance = [&](const float (&xr)[DMAX], float xx, int c) {
    const float4* yc4 = reinterpret_cast<const float4*>(yc_s + (size_t)c * STRIDE);
    float acc = 0.0f;
#pragma unroll
    for (int q = 0; q < DMAX / 4; ++q) {
      const float4 b = yc4[q];
      if (METRIC == F2C_L2) {
        const float d0 = xr[4 * q] - b.x, d1 = xr[4 * q + 1] - b.y, d2 = xr[4 * q + 2] - b.z, d3 = xr[4 * q + 3] - b.w;
        acc = fmaf(d0, d0, acc); acc = fmaf(d1, d1, acc); acc = fmaf(d2, d2, acc); acc = fmaf(d3, d3, acc);
      } else {
        acc = fmaf(xr[4 * q], b.x, acc); acc = fmaf(xr[4 * q + 1], b.y, acc);
        acc = fmaf(xr[4 * q + 2], b.z, acc); acc = fmaf(xr[4 * q + 3], b.w, acc);
      }
    }
    const float v = METRIC == F2C_L2 ? acc : finish_cosine(acc, xx, cc_s[c]);
    return v != v ? 1.0f : v;
  };
  float xr[DMAX];
  float xx = 0.0f;
  auto load_point = [&](int64_t i) {
    xx = 0.0f;
#pragma unroll
    for (int t = 0; t < DMAX; ++t) {
      xr[t] = (i >= 0 && t < d) ? __ldg(x + i * d + t) : 0.0f;
      if (METRIC == F2C_COSINE) xx = fmaf(xr[t], xr[t], xx);
    }
  };
  if (by_warp) {
    for (int64_t s = warp; s < cnt; s += n_warps) {
      const int64_t i = all ? s : (int64_t)list[s];
      load_point(i);
      float best = INFINITY;
      int best_c = 0x7fffffff;
      for (int c = lane; c < k; c += 32) {
        const float v = distance(xr, xx, c);
        if (v < best) { best = v; best_c = c; }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oc = __shfl_xor_sync(0xffffffffu, best_c, o);
        if (ob < best || (ob == best && oc < best_c)) { best = ob; best_c = oc; }
      }
      if (lane == 0) labels[i] = best_c == 0x7fffffff ? 0 : best_c;
    }
    return;
  }
  for (int64_t base = (int64_t)blockIdx.x * kListThreads; base < cnt; base += (int64_t)gridDim.x * kListThreads) {
    const int64_t s = base + threadIdx.x;
    const int64_t i = s < cnt ? (all ? s : (int64_t)list[s]) : -1;
    load_point(i);
    float best = INFINITY;
    int best_c = 0;
    for (int c0 = 0; c0 < k; c0 += kc) {
      const int nc = min(kc, k - c0);
      if (kc < k) {
        __syncthreads();
        stage(c0, nc);
      }
      for (int c = 0; c < nc; ++c) {
        const float v = distance(xr, xx, c);
        if (v < best) { best = v; best_c = c0 + c; }
      }
    }
    if (i >= 0) labels[i] = best_c;
  }
}

template <int DMAX>
static int launch_listed(const float* x, const float* y, int64_t* labels, const int32_t* list, const int32_t* count_dev, const int32_t* all_dev,
                         int64_t max_count, int64_t k, int64_t d, int metric, bool y_settled, cudaStream_t st) {
  int kc = (int)k;
  while ((size_t)kc * (DMAX + 5) * sizeof(float) > 96 * 1024) kc = (kc + 1) / 2;
  const size_t smem = (size_t)kc * (DMAX + 5) * sizeof(float);
  auto kern = metric == F2C_COSINE ? kmeans_listed_kernel<DMAX, F2C_COSINE> : kmeans_listed_kernel<DMAX, F2C_L2>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return set_error(F2C_ERR_CUDA, "kmeans_assign: %s", cudaGetErrorString(e));
  int64_t grid = ceil_div(max_count, kListThreads / 32);
  if (grid > 2 * current_sm_count()) grid = 2 * current_sm_count();
  launch_dependent(kern, (unsigned)grid, kListThreads, smem, st, x, y, labels, list, count_dev, all_dev, max_count, (int)k, (int)d, kc,
                   d % 4 == 0 && aligned(y, 16) ? 1 : 0, y_settled ? 1 : 0);
  return check_launch("kmeans_assign");
}

template <int DMAX>
static int launch_thread_assign(const float* x, const float* y, int64_t* labels, int64_t n, int64_t k, int64_t d, int metric, cudaStream_t st,
                                const int32_t* done) {
  int kc = (int)k;
  const size_t budget = 96 * 1024;
  while ((size_t)kc * (DMAX + 1) * sizeof(float) > budget) kc = (kc + 1) / 2;
  size_t smem = (size_t)kc * (DMAX + 1) * sizeof(float);
  unsigned grid = (unsigned)ceil_div(n, 256);
  cudaError_t e;
  if (metric == F2C_COSINE) {
    auto kern = kmeans_thread_kernel<DMAX, F2C_COSINE>;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) launch_dependent(kern, grid, 256, smem, st, x, y, labels, n, (int)k, (int)d, kc, done);
  } else {
    auto kern = kmeans_thread_kernel<DMAX, F2C_L2>;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) launch_dependent(kern, grid, 256, smem, st, x, y, labels, n, (int)k, (int)d, kc, done);
  }
  if (e != cudaSuccess) return set_error(F2C_ERR_CUDA, "kmeans_assign: %s", cudaGetErrorString(e));
  return check_launch("kmeans_assign");
}

// Exact fp32 assignment of all points.
int kmeans_assign_exact(const float* x, const float* y, int64_t* labels, int64_t n, int64_t k, int64_t d, int metric, cudaStream_t st,
                        const int32_t* done) {
  if (n == 0) return F2C_OK;
  if (d <= 8) return launch_thread_assign<8>(x, y, labels, n, k, d, metric, st, done);
  if (d <= 16) return launch_thread_assign<16>(x, y, labels, n, k, d, metric, st, done);
  if (d <= 32) return launch_thread_assign<32>(x, y, labels, n, k, d, metric, st, done);
  if (d <= 64) return launch_thread_assign<64>(x, y, labels, n, k, d, metric, st, done);
  if (d <= 128) return launch_thread_assign<128>(x, y, labels, n, k, d, metric, st, done);
  int64_t blocks = ceil_div(n, 8);
  if (blocks > current_sm_count() * 32) blocks = current_sm_count() * 32;
  if (metric == F2C_COSINE)
    launch_dependent(kmeans_warp_kernel<F2C_COSINE, false, true>, (unsigned)blocks, 256, 0, st, x, y, nullptr, labels, n, (int)k, (int)d, done);
  else
    launch_dependent(kmeans_warp_kernel<F2C_L2, false, true>, (unsigned)blocks, 256, 0, st, x, y, nullptr, labels, n, (int)k, (int)d, done);
  return check_launch("kmeans_assign");
}

// Exact assignment of the points listed in `list`; their number sits in device memory (*count_dev <= max_count).  Of all
// max_count points instead when all_dev is set and *all_dev is not 0.  y_settled: the kernel launched before this one on the stream has
// dependency_wait() as its first statement and does not write y, so what y holds then is what it holds now, and the centres are staged
// before that kernel is done.
int kmeans_assign_exact_listed(const float* x, const float* y, int64_t* labels, const int32_t* list, const int32_t* count_dev,
                               const int32_t* all_dev, int64_t max_count, int64_t k, int64_t d, int metric, bool y_settled, cudaStream_t st) {
  if (max_count == 0) return F2C_OK;
  if (d <= 8) return launch_listed<8>(x, y, labels, list, count_dev, all_dev, max_count, k, d, metric, y_settled, st);
  if (d <= 16) return launch_listed<16>(x, y, labels, list, count_dev, all_dev, max_count, k, d, metric, y_settled, st);
  if (d <= 32) return launch_listed<32>(x, y, labels, list, count_dev, all_dev, max_count, k, d, metric, y_settled, st);
  if (d <= 64) return launch_listed<64>(x, y, labels, list, count_dev, all_dev, max_count, k, d, metric, y_settled, st);
  return set_error(F2C_ERR_UNSUPPORTED, "kmeans_assign: listed re-scoring needs d <= 64");
}

bool kmeans_tc_supported(int64_t n, int64_t k, int64_t d);
int64_t kmeans_tc_workspace(int64_t n);
int kmeans_assign_tc(const float* x, const float* y, int64_t* labels, int64_t n, int64_t k, int64_t d, int metric, void* workspace,
                     cudaStream_t st);

static int validate_km(const char* op, int64_t n, int64_t k, int64_t d, int metric) {
  F2C_REQUIRE(n >= 0 && k >= 1 && d >= 1, F2C_ERR_INVALID, "%s: bad shape n=%lld k=%lld d=%lld", op, (long long)n, (long long)k,
              (long long)d);
  F2C_REQUIRE(metric == F2C_L2 || metric == F2C_COSINE, F2C_ERR_INVALID, "%s: unknown metric", op);
  F2C_REQUIRE(k < (1ll << 24) && d < (1ll << 20), F2C_ERR_LIMIT, "%s: k or d too large", op);
  return F2C_OK;
}

}  // namespace f2c

using namespace f2c;

extern "C" int f2c_pairwise_distance(const float* x, const float* y, float* dist, int64_t n, int64_t k, int64_t d, int metric,
                                     void* stream) {
  int rc = validate_km("pairwise_distance", n, k, d, metric);
  if (rc) return rc;
  if (n == 0) return F2C_OK;
  F2C_REQUIRE(x && y && dist, F2C_ERR_INVALID, "pairwise_distance: null pointer");
  int64_t blocks = ceil_div(n, 8);
  if (blocks > current_sm_count() * 32) blocks = current_sm_count() * 32;
  cudaStream_t st = (cudaStream_t)stream;
  if (metric == F2C_COSINE)
    launch_dependent(kmeans_warp_kernel<F2C_COSINE, true, false>, (unsigned)blocks, 256, 0, st, x, y, dist, nullptr, n, (int)k, (int)d, nullptr);
  else
    launch_dependent(kmeans_warp_kernel<F2C_L2, true, false>, (unsigned)blocks, 256, 0, st, x, y, dist, nullptr, n, (int)k, (int)d, nullptr);
  return check_launch("pairwise_distance");
}

extern "C" int64_t f2c_kmeans_assign_workspace(int64_t n, int64_t k, int64_t d) {
  return kmeans_tc_supported(n, k, d) ? kmeans_tc_workspace(n) : 0;
}

extern "C" int f2c_kmeans_assign(const float* x, const float* centers, int64_t* labels, int64_t n, int64_t k, int64_t d,
                                 int metric, void* workspace, void* stream) {
  const int scorer = metric & (F2C_SCORER_EXACT | F2C_SCORER_TENSOR);  // per-call choice of the scorer (tests, benchmarks)
  metric &= ~(F2C_SCORER_EXACT | F2C_SCORER_TENSOR);
  int rc = validate_km("kmeans_assign", n, k, d, metric);
  if (rc) return rc;
  if (n == 0) return F2C_OK;
  F2C_REQUIRE(x && centers && labels, F2C_ERR_INVALID, "kmeans_assign: null pointer");
  // tensor-core path when a scratch buffer is supplied and the shape fits; the exact fp32 scorer otherwise, and below four
  // dimensions, where many points' best two centres are too close for the split product (2,449,029 x 4 against 256 centres:
  // exact scorer 982 us, tensor cores 104)
  const bool prefer_tc = d >= 4 || scorer == F2C_SCORER_TENSOR;
  if (workspace != nullptr && kmeans_tc_supported(n, k, d) && prefer_tc && scorer != F2C_SCORER_EXACT && aligned(workspace, 16))
    return kmeans_assign_tc(x, centers, labels, n, k, d, metric, workspace, (cudaStream_t)stream);
  return kmeans_assign_exact(x, centers, labels, n, k, d, metric, (cudaStream_t)stream, nullptr);
}
