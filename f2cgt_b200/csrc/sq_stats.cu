// Codebook statistics of the scalar compressor (reference: examples/process_compress.py:43-68): four order statistics of |x|
// over a sample of one column slice - the neighbours of the 0.5 and 99.5 percentiles - and the mean of |x|.
//
// The reference sorts the sample (250,000 rows x slice).  Only four ranks are wanted, so this selects them by radix: the
// 31-bit magnitude is split 13 + 12 + 6 bits and three passes over the sample each narrow the ranks to one bin.  The sampled
// rows are read where they lie (no gathered copy); a pass moves the sample once, from L2 where it fits.  Histograms are kept
// in shared memory (pass 1 twice, by warp parity, because features crowd into a few dozen bins) and the CTA that finishes
// last scans the merged histogram, so a pass is one launch and the host reads nothing in between.  Pass 2 also lists the
// values that share the first 13 bits with a wanted rank - pass 1 has counted them - and pass 3 reads only that list, unless
// it would be longer than a million values (features that are mostly zero): then it reads the sample again.
#include <stddef.h>

#include "common.cuh"

namespace f2c {
namespace sqstat {

constexpr int kThreads = 512;
constexpr int kBins1 = 8192, kBins2 = 4096, kBins3 = 64;
constexpr int kInFlight = 8;  // loads in flight per lane
constexpr int kShift1 = 18, kShift2 = 6;
constexpr int kMaxCtas = 1024;
constexpr uint32_t kListMax = 1u << 20;
constexpr uint32_t kNear = 4096;  // candidates one CTA keeps in shared memory (more go to the list one by one)

struct Work {                 // zeroed before the first pass
  uint32_t hist[4 * kBins2];  // pass 1 uses 8192 entries, pass 2 4 x 4096, pass 3 4 x 64
  uint32_t arrived[4];
  uint32_t prefix[4];         // bits fixed so far of each wanted rank
  unsigned long long rank[4]; // rank inside the bin
  double sum[kMaxCtas];
  uint32_t listed;            // candidates appended in pass 2
  uint32_t fits;              // pass 1: all candidates fit the list
  uint32_t list[kListMax];    // magnitudes that share the first 13 bits with a wanted rank
};

struct Args {
  const float* x;
  const int64_t* rows;  // sampled rows, or null: rows 0 .. n_rows - 1
  int64_t ld, col, n_rows;
  int width;
  unsigned long long rank[4];
  Work* work;
  double* out;          // [5]: the four order statistics, the mean
};

struct Found { uint32_t bin[4], count[4]; unsigned long long inside[4]; };

// For each wanted rank the bin of its histogram that holds it, the rank inside the bin and the bin's count.  H histograms of NB
// bins; rank r lies in histogram owner[r].  One trip to memory for all of them: the CTA that does this works alone.
template <int H, int NB>
__device__ void locate(const uint32_t* __restrict__ hist, const int (&owner)[4], const unsigned long long (&rank)[4], Found* found) {
  constexpr int PER = NB >= kThreads ? NB / kThreads : 1;
  __shared__ unsigned long long warp_sum[H][kThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  uint32_t v[H][PER];
  unsigned long long before[H];
#pragma unroll
  for (int h = 0; h < H; ++h)
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int b = tid * PER + i;
      v[h][i] = b < NB ? __ldcg(hist + h * NB + b) : 0u;
    }
#pragma unroll
  for (int h = 0; h < H; ++h) {
    unsigned long long mine = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) mine += v[h][i];
    unsigned long long inc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) warp_sum[h][wid] = inc;
    before[h] = inc - mine;
  }
  __syncthreads();
#pragma unroll
  for (int h = 0; h < H; ++h) {
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) before[h] += w < wid ? warp_sum[h][w] : 0ull;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      if (owner[r] != h) continue;
      unsigned long long at = before[h];
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        if (rank[r] >= at && rank[r] < at + v[h][i]) { found->bin[r] = (uint32_t)(tid * PER + i); found->inside[r] = rank[r] - at; found->count[r] = v[h][i]; }
        at += v[h][i];
      }
    }
  }
  __syncthreads();
}

// A value that shares the fixed bits with wanted rank r (rare, so one copy of the code, and nothing captured by it).
template <int PASS>
__device__ __noinline__ void near_value(uint32_t key, int r, uint32_t* hist, bool keep, uint32_t* near_s, uint32_t* n_near, Work* w) {
  const uint32_t bin = PASS == 2 ? (key >> kShift2) & (kBins2 - 1) : key & (kBins3 - 1);
  atomicAdd(hist + r * (PASS == 2 ? kBins2 : kBins3) + bin, 1u);
  if (PASS == 2 && keep) {
    const uint32_t at = atomicAdd(n_near, 1u);
    if (at < kNear) near_s[at] = key; else w->list[atomicAdd(&w->listed, 1u)] = key;
  }
}

// PASS 1, 2, 3; VEC = 4: rows and columns allow 16-byte loads
template <int PASS, int VEC>
__global__ void __launch_bounds__(kThreads, 2) select_kernel(const Args a) {
  dependency_wait();
  release_dependents();
  extern __shared__ __align__(16) uint32_t hist_s[];
  __shared__ bool last;
  __shared__ double warp_total[kThreads / 32];
  __shared__ uint32_t n_near, list_at;  // this CTA's candidates, appended to the list in one piece
  uint32_t* near_s = hist_s + 4 * kBins2;
  constexpr int kShared = PASS == 1 ? 2 * kBins1 : PASS == 2 ? 4 * kBins2 : 4 * kBins3;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  Work* w = a.work;
  for (int i = tid; i < kShared; i += kThreads) hist_s[i] = 0u;
  if (tid == 0) n_near = 0u;
  // distinct prefixes of the wanted ranks (the lowest rank owns the histogram of a shared one)
  uint32_t prefix[4], want[4];
  int owner[4] = {0, 0, 0, 0};
  if (PASS > 1) {
#pragma unroll
    for (int r = 0; r < 4; ++r) prefix[r] = __ldcg(&w->prefix[r]);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      owner[r] = r;
#pragma unroll
      for (int q = r - 1; q >= 0; --q)
        if (prefix[q] == prefix[r]) owner[r] = q;
      want[r] = owner[r] == r ? prefix[r] : 0xffffffffu;
    }
  }
  __syncthreads();
  double sum = 0.0;
  const bool keep = PASS > 1 && __ldcg(&w->fits) != 0u;
  uint32_t* mine = hist_s + (PASS == 1 ? (wid & 1) * kBins1 : 0);
  auto count = [&](float f) {
    const uint32_t key = __float_as_uint(f) & 0x7fffffffu;
    if (PASS == 1) {
      sum += (double)fabsf(f);
      atomicAdd(mine + (key >> kShift1), 1u);
    } else {
      const uint32_t pf = PASS == 2 ? key >> kShift1 : key >> kShift2;
      if (pf == want[0] || pf == want[1] || pf == want[2] || pf == want[3])
        near_value<PASS>(key, pf == want[0] ? 0 : pf == want[1] ? 1 : pf == want[2] ? 2 : 3, mine, keep, near_s, &n_near, w);
    }
  };
  if (PASS == 3 && keep) {
    const uint32_t n = min(__ldcg(&w->listed), kListMax);
    for (uint32_t i = blockIdx.x * kThreads + tid; i < n; i += gridDim.x * kThreads) count(__uint_as_float(__ldcg(w->list + i)));
  }
  // a warp takes 32 rows at a time: one row number per lane, then the lanes sweep the rows' pieces
  const int pieces = a.width / VEC;  // VEC == 1: every column
  const uint32_t magic = 0xffffffffu / (uint32_t)pieces + 1u;  // item / pieces for item < 32 * pieces (pieces < 2^13)
  const int64_t groups = PASS == 3 && keep ? 0 : (a.n_rows + 31) / 32;
  for (int64_t g = (int64_t)blockIdx.x * (kThreads / 32) + wid; g < groups; g += (int64_t)gridDim.x * (kThreads / 32)) {
    const int64_t r0 = g * 32;
    const int live = (int)min((int64_t)32, a.n_rows - r0);
    int64_t row = 0;
    if (lane < live) row = a.rows != nullptr ? __ldg(a.rows + r0 + lane) : r0 + lane;
    const int items = 32 * pieces;
    for (int t = lane; t < items; t += 32 * kInFlight) {
      float4 v[kInFlight];
      bool on[kInFlight];
#pragma unroll
      for (int u = 0; u < kInFlight; ++u) {
        const int it = t + 32 * u;
        const int r = pieces == 1 ? it : (int)__umulhi((uint32_t)it, magic);
        const int64_t src = __shfl_sync(0xffffffffu, row, r & 31);
        on[u] = it < items && r < live;
        v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (on[u]) {
          const float* q = a.x + src * a.ld + a.col + (int64_t)(it - r * pieces) * VEC;
          if (VEC == 4) v[u] = __ldg(reinterpret_cast<const float4*>(q)); else v[u].x = __ldg(q);
        }
      }
#pragma unroll
      for (int u = 0; u < kInFlight; ++u)
        if (on[u]) {
          count(v[u].x);
          if (VEC == 4) { count(v[u].y); count(v[u].z); count(v[u].w); }
        }
    }
  }
  if (PASS == 1) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) warp_total[wid] = sum;
  }
  __syncthreads();
  if (PASS == 1) {
    if (tid == 0) {
      double t = 0.0;
      for (int i = 0; i < kThreads / 32; ++i) t += warp_total[i];
      w->sum[blockIdx.x] = t;
    }
    for (int i = tid; i < kBins1; i += kThreads) {
      const uint32_t c = hist_s[i] + hist_s[kBins1 + i];
      if (c != 0u) atomicAdd(w->hist + i, c);
    }
  } else {
    if (PASS == 2) {
      const uint32_t n = min(n_near, kNear);
      if (tid == 0) list_at = n != 0u ? atomicAdd(&w->listed, n) : 0u;
      __syncthreads();
      for (uint32_t i = tid; i < n; i += kThreads) w->list[list_at + i] = near_s[i];
    }
    for (int i = tid; i < kShared; i += kThreads)
      if (hist_s[i] != 0u) atomicAdd(w->hist + i, hist_s[i]);
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) last = atomicAdd(&w->arrived[PASS - 1], 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  // ---- the last CTA: which bin holds each wanted rank
  // (it works alone, so its trips to memory count: one after the other they were 30 of the 37 us of the first pass over 3.2 M values)
  __shared__ Found found;
  __shared__ double cta_sum[PASS == 1 ? kMaxCtas : 1];
  unsigned long long rank[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) rank[r] = PASS == 1 ? a.rank[r] : __ldcg(&w->rank[r]);
  if (PASS == 1)
    for (int i = tid; i < (int)gridDim.x; i += kThreads) cta_sum[i] = __ldcg(&w->sum[i]);
  locate<PASS == 1 ? 1 : 4, PASS == 1 ? kBins1 : PASS == 2 ? kBins2 : kBins3>(w->hist, owner, rank, &found);
  if (PASS < 3)
    for (int i = tid; i < 4 * kBins2; i += kThreads) w->hist[i] = 0u;
  if (tid < 4) {
    const uint32_t pf = PASS == 1 ? 0u : tid == 0 ? prefix[0] : tid == 1 ? prefix[1] : tid == 2 ? prefix[2] : prefix[3];
    if (PASS < 3) {
      w->prefix[tid] = PASS == 1 ? found.bin[tid] : pf << 12 | found.bin[tid];
      w->rank[tid] = found.inside[tid];
    } else {
      a.out[tid] = (double)__uint_as_float(pf << 6 | found.bin[tid]);
    }
  }
  if (PASS == 1 && tid == 0) {
    unsigned long long candidates = 0;
    for (int r = 0; r < 4; ++r) {
      bool seen = false;
      for (int q = 0; q < r; ++q) seen |= found.bin[q] == found.bin[r];
      if (!seen) candidates += found.count[r];
    }
    w->fits = candidates <= kListMax ? 1u : 0u;
    double t = 0.0;
    for (int i = 0; i < (int)gridDim.x; ++i) t += cta_sum[i];
    a.out[4] = t / ((double)a.n_rows * (double)a.width);
  }
}

template <int PASS, int VEC>
static cudaError_t launch(const Args& a, int grid, cudaStream_t st) {
  constexpr int smem = 4 * (PASS == 1 ? 2 * kBins1 : PASS == 2 ? 4 * kBins2 + (int)kNear : 4 * kBins3);
  auto kern = select_kernel<PASS, VEC>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
  }
  launch_dependent(kern, (unsigned)grid, kThreads, smem, st, a);
  return cudaGetLastError();
}

template <int VEC>
static cudaError_t launch_all(const Args& a, int grid, cudaStream_t st) {
  cudaError_t e = launch<1, VEC>(a, grid, st);
  if (e == cudaSuccess) e = launch<2, VEC>(a, grid, st);
  if (e == cudaSuccess) e = launch<3, VEC>(a, grid, st);
  return e;
}

}  // namespace sqstat
}  // namespace f2c

using namespace f2c;

extern "C" int64_t f2c_sq_statistics_workspace(void) { return (int64_t)sizeof(sqstat::Work); }

extern "C" int f2c_sq_statistics(const float* x, int64_t ld, const int64_t* rows, int64_t n_rows, int64_t col, int64_t width,
                                 const int64_t* ranks_host, double* out, void* workspace, void* stream) {
  const char* op = "sq_statistics";
  F2C_REQUIRE(x && out && workspace && ranks_host && aligned(workspace, 16), F2C_ERR_INVALID, "%s: null or misaligned pointer", op);
  F2C_REQUIRE(n_rows >= 1 && width >= 1 && col >= 0 && ld >= col + width, F2C_ERR_INVALID, "%s: bad shape", op);
  F2C_REQUIRE(width < (1 << 13) && n_rows * width < (1ll << 31), F2C_ERR_LIMIT, "%s: sample too large", op);
  sqstat::Args a{};
  a.x = x; a.rows = rows; a.ld = ld; a.col = col; a.n_rows = n_rows; a.width = (int)width; a.work = (sqstat::Work*)workspace; a.out = out;
  for (int r = 0; r < 4; ++r) {
    F2C_REQUIRE(ranks_host[r] >= 0 && ranks_host[r] < n_rows * width, F2C_ERR_INVALID, "%s: rank out of range", op);
    a.rank[r] = (unsigned long long)ranks_host[r];
  }
  cudaStream_t st = (cudaStream_t)stream;
  cudaError_t e = cudaMemsetAsync(workspace, 0, offsetof(sqstat::Work, list), st);
  // two 64 KB histograms per SM; a CTA's 16 warps should have a few groups of 32 rows each before it pays for its histogram
  int64_t grid = ceil_div(n_rows, 32 * 16);
  if (grid > 2 * current_sm_count()) grid = 2 * current_sm_count();
  if (grid > sqstat::kMaxCtas) grid = sqstat::kMaxCtas;
  const bool vec = width % 4 == 0 && col % 4 == 0 && ld % 4 == 0 && aligned(x, 16);
  if (e == cudaSuccess) e = vec ? sqstat::launch_all<4>(a, (int)grid, st) : sqstat::launch_all<1>(a, (int)grid, st);
  if (e != cudaSuccess) return set_error(F2C_ERR_CUDA, "%s: %s", op, cudaGetErrorString(e));
  return F2C_OK;
}
