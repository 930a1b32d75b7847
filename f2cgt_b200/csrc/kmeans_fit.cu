// Lloyd iterations of KMeans.fit (reference: RAFT kmeans::fit behind src/kmeans.cu:61-75, and the torch loop of
// examples/my_kmeans.py:73-113) queued on the device without a host read per iteration.
//
// Shapes of the tensor cores (up to 256 centres, 4 to 64 dimensions): kmeans_fit_tc.cu, a kernel for many iterations.  All others, here:
// one iteration = the exact assignment (kmeans.cu) + ONE kernel that sums every cluster's points and, in the CTA that finishes last,
// replaces the centres, measures their shift and raises the `done` word.  All kernels return at once when that word is set, so the
// caller queues several iterations ahead and looks at the word every few of them; iterations queued behind the converged one change
// nothing.
//
//  * Sums are exact and independent of the order of the additions: a value becomes a fixed-point integer (43 fraction bits
//    below the largest magnitude of its column, fewer when more than 2^18 points could overflow 63 bits), and integers
//    commute.  A fit is therefore reproducible bit for bit, as it was with the sorted float64 prefix sums this replaces,
//    and at least as accurate.
//  * Inside a CTA the integers are added in shared memory as two 22-bit limbs with 32-bit atomics without a result (the
//    64-bit ones are a compare-and-swap loop); at most 1023 points can be added before a limb could overflow, so a CTA
//    takes chunks of at most 1000 points and adds the touched clusters to the 64-bit sums in global memory.
#include "kmeans_fit.cuh"

namespace f2c {

bool kmeans_tc_supported(int64_t n, int64_t k, int64_t d);
int kmeans_fit_tc(const float* x, float* centers, int64_t n, int64_t k, int64_t d, int metric, double tol, int iterations, FitState* state, long long* sums,
                  uint32_t* counts, const uint32_t* maxima, uint16_t* labels, double* shifts, int32_t* error, cudaStream_t st, int flags);
int kmeans_assign_exact(const float* x, const float* y, int64_t* labels, int64_t n, int64_t k, int64_t d, int metric, cudaStream_t st,
                        const int32_t* done);

namespace fit {

constexpr int kThreads = 512;
constexpr int kChunk = 1000;                 // points whose limbs cannot overflow 32 bits
constexpr size_t kSmemLimit = 200 * 1024;

// Largest |x| of every column as float bits.  `threads` is a multiple of d, so that a thread stays in its column; d above the grid's
// threads: every thread walks over columns.
__global__ void __launch_bounds__(256) max_abs_kernel(const float* __restrict__ x, int64_t numel, int d, int64_t threads, uint32_t* __restrict__ maxima) {
  dependency_wait();
  release_dependents();
  extern __shared__ uint32_t max_s[];
  const int64_t me = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool shared = threads > 0 && d <= 4096;
  if (shared) {
    for (int j = threadIdx.x; j < d; j += blockDim.x) max_s[j] = 0u;
    __syncthreads();
  }
  if (threads > 0) {
    uint32_t m = 0;
    if (me < threads)
      for (int64_t i = me; i < numel; i += threads) m = max(m, __float_as_uint(__ldg(x + i)) & 0x7fffffffu);  // NaN has larger bits than inf
    if (m != 0u) atomicMax(shared ? max_s + me % d : maxima + me % d, m);
  } else {
    for (int64_t j = me; j < d; j += (int64_t)gridDim.x * blockDim.x) {
      uint32_t m = 0;
      for (int64_t i = j; i < numel; i += d) m = max(m, __float_as_uint(__ldg(x + i)) & 0x7fffffffu);
      maxima[j] = m;
    }
  }
  if (shared) {
    __syncthreads();
    for (int j = threadIdx.x; j < d; j += blockDim.x)
      if (max_s[j] != 0u) atomicMax(maxima + j, max_s[j]);
  }
}

__global__ void begin_kernel(const uint32_t* __restrict__ maxima, int d, FitState* st) {
  dependency_wait();
  release_dependents();
  for (int j = threadIdx.x; j < d; j += blockDim.x)
    if (maxima[j] >= 0x7f800000u) { st->not_finite = 1; st->done = 1; }
}

// Centres <- sums / counts (clusters without points keep theirs), sums and counts <- 0, shift, done.  One CTA.
// scale_of(j): what column j's values were multiplied with, a power of two.
template <typename Scale>
__device__ void finish_iteration(float* __restrict__ centers, long long* sums, unsigned int* counts, int k, int d, Scale scale_of, double tol,
                                 FitState* st) {
  __shared__ double part[kThreads / 32];
  double shift = 0.0;
  // this CTA alone works now: the loads of eight entries are in flight together (one at a time: 11 of 23 us for 256 x 32)
  constexpr int U = 8;
  for (int i0 = threadIdx.x; i0 < k * d; i0 += U * kThreads) {
    unsigned int cnt[U];
    int col[U];
    long long sum[U];
    float old[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * kThreads;
      const int c = i / d;
      cnt[u] = 0u;
      col[u] = i - c * d;
      if (i < k * d) { cnt[u] = __ldcg(counts + c); sum[u] = __ldcg(sums + i); old[u] = centers[i]; }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * kThreads;
      if (cnt[u] != 0u) {  // sums of clusters without points are zero
        sums[i] = 0;
        const double unit = __hiloint2double((2046 << 20) - __double2hiint(scale_of(col[u])), 0);  // 1 / scale
        const float next = (float)((double)sum[u] * unit) / (float)cnt[u];
        const float diff = next - old[u];
        shift += (double)(diff * diff);
        centers[i] = next;
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) shift += __shfl_xor_sync(0xffffffffu, shift, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = shift;
  __syncthreads();
  for (int i = threadIdx.x; i < k; i += kThreads) counts[i] = 0u;
  if (threadIdx.x == 0) {
    double total = 0.0;
    for (int w = 0; w < kThreads / 32; ++w) total += part[w];
    st->shift = total;
    st->iterations += 1;
    st->arrived = 0u;
    if ((double)(float)total <= tol) st->done = 1;
  }
}

// SHARED: k * d entries fit in shared memory as two limbs; otherwise every value is one 64-bit atomic in global memory.
template <bool SHARED>
__global__ void __launch_bounds__(kThreads) accumulate_kernel(const float* __restrict__ x, const int64_t* __restrict__ labels,
                                                              float* __restrict__ centers, long long* sums, unsigned int* counts,
                                                              const uint32_t* __restrict__ maxima, int64_t n, int k, int d, double tol,
                                                              FitState* st) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int kd = k * d;
  double* scales = reinterpret_cast<double*>(smem);  // of the columns
  uint32_t* lo = reinterpret_cast<uint32_t*>(scales + (SHARED ? d : 0));
  int32_t* hi = reinterpret_cast<int32_t*>(lo + (SHARED ? kd : 0));
  uint32_t* cnt = reinterpret_cast<uint32_t*>(hi + (SHARED ? kd : 0));
  uint16_t* lab = reinterpret_cast<uint16_t*>(cnt + (SHARED ? k : 0));  // labels of the chunk (k <= 65535 here)
  __shared__ bool last;
  const int tid = (int)threadIdx.x;
  if (SHARED)  // while the kernel before still runs
    for (int i = tid; i < 2 * kd + k; i += kThreads) lo[i] = 0u;
  dependency_wait();
  release_dependents();
  const int bits = fraction_bits(n);
  auto scale_of = [&](int j) { return SHARED ? scales[j] : power2(bits - exponent(__ldg(maxima + j))); };
  if (SHARED)
    for (int i = tid; i < d; i += kThreads) scales[i] = power2(bits - exponent(__ldg(maxima + i)));
  if (*(volatile int32_t*)&st->done != 0) return;

  // chunks are dealt so that every CTA gets almost the same number of points
  const int64_t rounds = (n + (int64_t)gridDim.x * kChunk - 1) / ((int64_t)gridDim.x * kChunk);
  const int64_t per = (n + rounds * gridDim.x - 1) / (rounds * gridDim.x);
  if (SHARED) __syncthreads();
  for (int64_t r = 0; r < rounds; ++r) {
    const int64_t p0 = (r * gridDim.x + blockIdx.x) * per;
    const int pts = (int)max((int64_t)0, min(per, n - p0));
    if (SHARED) {
      for (int i = tid; i < pts; i += kThreads) {
        const int l = (int)labels[p0 + i];
        lab[i] = (uint16_t)l;
        atomicAdd(cnt + l, 1u);
      }
      __syncthreads();
    }
    const float* __restrict__ base = x + p0 * d;
    const int total = pts * d;
    int p = tid / d, j = tid - p * d;
    const int dp = kThreads / d, dj = kThreads - dp * d;
    for (int t = tid; t < total; t += kThreads) {
      const long long v = __double2ll_rn((double)__ldg(base + t) * scale_of(j));
      if (SHARED) {
        const int at = (int)lab[p] * d + j;
        atomicAdd(lo + at, (uint32_t)v & 0x3fffffu);
        atomicAdd(hi + at, (int32_t)(v >> 22));
      } else {
        const int64_t l = labels[p0 + p];
        atomicAdd(reinterpret_cast<unsigned long long*>(sums + l * d + j), (unsigned long long)v);
        if (j == 0) atomicAdd(counts + l, 1u);
      }
      p += dp; j += dj;
      if (j >= d) { j -= d; ++p; }
    }
    if (SHARED) {
      __syncthreads();
      for (int i = tid; i < kd; i += kThreads) {
        if (cnt[i / d] == 0u) continue;
        const long long v = ((long long)hi[i] << 22) + (long long)lo[i];
        lo[i] = 0u; hi[i] = 0;
        atomicAdd(reinterpret_cast<unsigned long long*>(sums + i), (unsigned long long)v);
      }
      __syncthreads();
      for (int i = tid; i < k; i += kThreads)
        if (cnt[i] != 0u) { atomicAdd(counts + i, cnt[i]); cnt[i] = 0u; }
      __syncthreads();
    }
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) last = atomicAdd(&st->arrived, 1u) == gridDim.x - 1;
  __syncthreads();
  if (last) {
    __threadfence();
    finish_iteration(centers, sums, counts, k, d, scale_of, tol, st);
  }
}

struct Layout { size_t sums, counts, labels, assign, maxima, shifts, total; };

static Layout plan(int64_t n, int64_t k, int64_t d) {
  auto up = [](size_t v) { return (v + 255) & ~(size_t)255; };
  Layout w{};
  size_t at = 256;
  w.sums = at; at += up((size_t)k * d * 8);
  w.counts = at; at += up((size_t)k * 4);
  w.labels = at; at += up((size_t)n * 8);
  w.assign = at; at += 256;  // second word: code of a bounded wait of the tensor-core kernel that ran out
  w.maxima = at; at += up((size_t)d * 4);
  w.shifts = at; at += up((size_t)kFitMaxCtas * 8);
  w.total = at;
  return w;
}

static int validate(const char* op, int64_t n, int64_t k, int64_t d) {
  F2C_REQUIRE(n >= 1 && k >= 1 && d >= 1, F2C_ERR_INVALID, "%s: bad shape n=%lld k=%lld d=%lld", op, (long long)n, (long long)k,
              (long long)d);
  F2C_REQUIRE(n < (1ll << 31) && k < (1ll << 24) && k * d < (1ll << 31), F2C_ERR_LIMIT, "%s: n, k or k * d too large", op);
  return F2C_OK;
}

}  // namespace fit
}  // namespace f2c

using namespace f2c;

extern "C" int64_t f2c_kmeans_fit_workspace(int64_t n, int64_t k, int64_t d) {
  return n >= 1 && k >= 1 && d >= 1 ? (int64_t)fit::plan(n, k, d).total : 0;
}

extern "C" int f2c_kmeans_fit_begin(const float* x, int64_t n, int64_t k, int64_t d, void* workspace, void* stream) {
  const char* op = "kmeans_fit_begin";
  int rc = fit::validate(op, n, k, d);
  if (rc) return rc;
  F2C_REQUIRE(x && workspace && aligned(workspace, 256), F2C_ERR_INVALID, "%s: null or misaligned pointer", op);
  cudaStream_t st = (cudaStream_t)stream;
  const fit::Layout w = fit::plan(n, k, d);
  cudaError_t e = cudaMemsetAsync(workspace, 0, w.labels, st);  // state, sums and counts
  if (e == cudaSuccess) e = cudaMemsetAsync((unsigned char*)workspace + w.assign, 0, w.shifts - w.assign, st);  // error, maxima
  if (e == cudaSuccess && kmeans_tc_supported(n, k, d)) e = cudaMemsetAsync((uint16_t*)((unsigned char*)workspace + w.labels) + n, 0xff, (size_t)n * 2, st);  // summed: none
  if (e != cudaSuccess) return set_error(F2C_ERR_CUDA, "%s: %s", op, cudaGetErrorString(e));
  FitState* state = (FitState*)workspace;
  int64_t blocks = ceil_div(n * d, 256 * 8);
  if (blocks > 8 * current_sm_count()) blocks = 8 * current_sm_count();
  uint32_t* maxima = (uint32_t*)((unsigned char*)workspace + w.maxima);
  launch_dependent(fit::max_abs_kernel, (unsigned)blocks, 256, d <= 4096 ? (size_t)d * 4 : 0, st, x, n * d, (int)d, blocks * 256 / d * d, maxima);
  launch_dependent(fit::begin_kernel, 1, 256, 0, st, maxima, (int)d, state);
  return check_launch(op);
}

extern "C" int f2c_kmeans_fit_iterate(const float* x, float* centers, int64_t n, int64_t k, int64_t d, int metric, double tol,
                                      int iterations, void* workspace, void* stream) {
  const char* op = "kmeans_fit_iterate";
  int rc = fit::validate(op, n, k, d);
  if (rc) return rc;
  const int flags = metric & F2C_NO_WAITS;
  metric &= ~F2C_NO_WAITS;
  F2C_REQUIRE(metric == F2C_L2 || metric == F2C_COSINE, F2C_ERR_INVALID, "%s: unknown metric", op);
  F2C_REQUIRE(x && centers && workspace && aligned(workspace, 256) && iterations >= 0, F2C_ERR_INVALID, "%s: bad argument", op);
  cudaStream_t st = (cudaStream_t)stream;
  const fit::Layout w = fit::plan(n, k, d);
  unsigned char* ws = (unsigned char*)workspace;
  FitState* state = (FitState*)ws;
  long long* sums = (long long*)(ws + w.sums);
  unsigned int* counts = (unsigned int*)(ws + w.counts);
  int64_t* labels = (int64_t*)(ws + w.labels);
  // the line is that of the assignment (kmeans.cu)
  if (kmeans_tc_supported(n, k, d) && d >= 4) {
    if (iterations == 0) return F2C_OK;
    return kmeans_fit_tc(x, centers, n, k, d, metric, tol, iterations, state, sums, counts, (const uint32_t*)(ws + w.maxima), (uint16_t*)labels,
                         (double*)(ws + w.shifts), (int32_t*)(ws + w.assign) + 1, st, flags);
  }
  const size_t smem = (size_t)d * 8 + ((size_t)2 * k * d + k) * 4 + fit::kChunk * 2;
  const uint32_t* maxima = (const uint32_t*)(ws + w.maxima);
  const bool shared = smem <= fit::kSmemLimit && k <= 65535;
  auto kern = shared ? fit::accumulate_kernel<true> : fit::accumulate_kernel<false>;
  if (shared) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return set_error(F2C_ERR_CUDA, "%s: %s", op, cudaGetErrorString(e));
  }
  // every CTA adds its clusters to the global sums once per chunk: few points per CTA would make that the bigger part
  int64_t grid = shared ? ceil_div(n, 256) : ceil_div(n * d, fit::kThreads);
  if (grid > current_sm_count()) grid = current_sm_count();
  for (int it = 0; it < iterations; ++it) {
    rc = kmeans_assign_exact(x, centers, labels, n, k, d, metric, st, &state->done);
    if (rc) return rc;
    launch_dependent(kern, (unsigned)grid, fit::kThreads, shared ? smem : 0, st, x, labels, centers, sums, counts, maxima, n, (int)k, (int)d, tol,
                     state);
    rc = check_launch(op);
    if (rc) return rc;
  }
  return F2C_OK;
}
