// A whole minibatch - every hop of neighbour sampling and relabelling - in ONE cooperative kernel (the loop of the
// reference's loader, examples/dataloader.py:167-182, whose operators live in its absent ShmTensor submodule).  Same draws
// and same numbering as one sample_block call per hop; what changes is
//  * the host reads once per minibatch instead of once per hop: the number of seeds of a hop stays on the device;
//  * no hash table.  The graph has one 64-bit word per node, 20 MB for 2.4 M nodes and so in L2 (0.9 GB at 111 M nodes): the
//    high half is the complement of the minibatch's number, so that words of earlier minibatches always lose an atomic
//    minimum and nothing is ever cleared; the low half is the node's new number or, while a hop is being built, bit 31 and
//    the first position at which the node occurred.  An occurrence is one reduction without a result, where the table cost
//    its clearing, a compare-and-swap chain and two more probe chains;
//  * numbers carry over: the seeds of a hop are the nodes numbered so far, so only sampled ids are looked at (in the first hop
//    the seeds are positions like any other, because they may repeat);
//  * a group of 8, 16 or 32 lanes draws for one seed: each lane makes one draw of Floyd's subset algorithm, a short loop of
//    shuffles settles repeated draws in order, and the reads of the neighbour ids go out together.
// Per hop and barrier: A degrees, scanned per warp and CTA | B offsets, draws, first positions | C which occurrences are
// first, ranked | D numbers.  Every warp owns a contiguous run of seeds (A, B) and of positions (C), so prefix sums are
// warp prefix + CTA prefix + one array of CTA totals.
//
// Latency bound: chains of dependent reads between grid barriers.  Measured on B200, 1024 seeds, fan-out 12,12,12 on 2.4 M
// nodes (708,000 edges in the last hop): 86 us against 37 + 49 + 123 us for the three sample_block kernels, and one host
// read instead of three; a minibatch of the loader 368 -> 93 us.
#include <cooperative_groups.h>

#include <mutex>
#include <type_traits>

#include "block_build.cuh"

namespace cg = cooperative_groups;

namespace f2c {
namespace mb {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxCtas = 512;  // one thread of a CTA per CTA total
constexpr uint32_t kPending = 0x80000000u;

template <typename IdxT>
struct Params {
  const IdxT* indptr;
  const IdxT* indices;
  const IdxT* seeds;
  int64_t n_nodes;
  int n_seeds, n_hops;
  int pick[F2C_MAX_HOPS];
  IdxT* sub_indptr[F2C_MAX_HOPS];
  IdxT* ids[F2C_MAX_HOPS];
  IdxT* local[F2C_MAX_HOPS];
  IdxT* unique;
  unsigned long long* node_map;
  unsigned long long stamp;  // complement of the minibatch's number, in the high half
  uint32_t* val;             // per position: what the node's word said
  uint32_t* rank;            // per first occurrence: rank inside the warp's run
  uint32_t* warp_prefix;     // per warp: first occurrences of the CTA's warps before it
  uint32_t* cta_sum;         // [2 * kMaxCtas]
  int32_t* error;
  int64_t* header;           // [2 * n_hops + 1], host memory: edges and distinct nodes per hop, error
  uint64_t rng_seed, rng_offset;
};

__device__ __forceinline__ uint32_t warp_exclusive(uint32_t v, uint32_t* total) {
  const int lane = threadIdx.x & 31;
  uint32_t inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  *total = __shfl_sync(0xffffffffu, inc, 31);
  return inc - v;
}

// totals of this CTA's warps -> exclusive prefix per warp (returned to every lane of it) and the CTA's total in *sum
__device__ __forceinline__ uint32_t cta_exclusive(uint32_t warp_total, uint32_t* smem, uint32_t* sum) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) smem[wid] = warp_total;
  __syncthreads();
  uint32_t total;
  const uint32_t ex = warp_exclusive(lane < kWarps ? smem[lane] : 0u, &total);
  *sum = total;
  return __shfl_sync(0xffffffffu, ex, wid);
}

// exclusive prefix of the CTA totals into shared memory; returns the grand total to every thread
__device__ __forceinline__ uint32_t scan_totals(const uint32_t* totals, int n_cta, uint32_t* prefix, uint32_t* smem) {
  const uint32_t v = (int)threadIdx.x < n_cta ? __ldcg(totals + threadIdx.x) : 0u;
  uint32_t warp_total, sum;
  const uint32_t ex = warp_exclusive(v, &warp_total);
  const uint32_t before = cta_exclusive(warp_total, smem, &sum);
  prefix[threadIdx.x] = before + ex;
  __syncthreads();
  return sum;
}

// Draws of one seed by a group of W lanes (num_pick <= W): offset of this lane's neighbour inside the seed's list, -1 for
// lanes without one.  All lanes of the warp call; d = in-degree, below 2^32.
template <int W>
__device__ __forceinline__ int64_t draw(uint32_t d, int num_pick, int64_t position, uint64_t rng_seed, uint64_t rng_offset) {
  const int s = threadIdx.x & (W - 1);
  const bool all = d <= (uint32_t)num_pick;
  uint32_t chosen = 0xffffffffu, t = 0u, j = 0u;
  if (!all && s < num_pick) {
    const uint4 r = Philox(rng_seed, rng_offset)((uint64_t)position * (kMaxPick / 2) + (uint64_t)(s >> 1));
    const uint64_t bits = (s & 1) == 0 ? ((uint64_t)r.x << 32 | r.y) : ((uint64_t)r.z << 32 | r.w);
    j = d - (uint32_t)num_pick + (uint32_t)s;
    t = (uint32_t)__umul64hi(bits, (uint64_t)j + 1u);
  }
  // Floyd: draw s is t_s unless an earlier draw was t_s, then j_s.  Lane s knows after step s - 1 whether t_s is taken.
  bool taken = false;
  for (int q = 0; q < num_pick; ++q) {
    if (s == q) chosen = taken ? j : t;
    const uint32_t c = __shfl_sync(0xffffffffu, chosen, q, W);
    if (q < s) taken |= c == t;
  }
  if (all) return s < (int)d ? s : -1;
  return s < num_pick ? (int64_t)chosen : -1;
}

template <typename IdxT>
__global__ void __launch_bounds__(kThreads) minibatch_kernel(const Params<IdxT> p) {
  cg::grid_group grid = cg::this_grid();
  __shared__ uint32_t smem[kWarps];
  __shared__ uint32_t prefix[kThreads];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, cta = blockIdx.x, n_cta = gridDim.x;
  const uint32_t gwarp = cta * kWarps + wid, n_warps = n_cta * kWarps;
  const uint32_t gtid = cta * kThreads + tid;
  uint32_t n = (uint32_t)p.n_seeds;

  for (int hop = 0; hop < p.n_hops; ++hop) {
    const IdxT* seeds = hop == 0 ? p.seeds : p.unique;
    const int pick = p.pick[hop];
    IdxT* sub_indptr = p.sub_indptr[hop];
    IdxT* ids = p.ids[hop];
    auto note = [&](int64_t id, uint32_t pos) {  // an occurrence of `id` at position pos
      if (id < 0 || id >= p.n_nodes) { *(volatile int32_t*)p.error = id < 0 ? 2 : 3; return; }
      atomicMin(p.node_map + id, p.stamp | kPending | pos);
    };

    // ---- A: degrees of this warp's seeds, offsets inside its run
    const uint32_t per_warp = (n + n_warps - 1) / n_warps;
    const uint32_t s_lo = min(gwarp * per_warp, n), s_hi = min(s_lo + per_warp, n);
    uint32_t run = 0;
    for (uint32_t base = s_lo; base < s_hi; base += 32) {
      const uint32_t i = base + lane;
      uint32_t deg = 0;
      if (i < s_hi) {
        const int64_t v = (int64_t)__ldcg(seeds + i);
        if (hop == 0) note(v, i);
        if (v >= 0 && v < p.n_nodes) {
          const int64_t d = (int64_t)__ldg(p.indptr + v + 1) - (int64_t)__ldg(p.indptr + v);
          deg = d < pick ? (uint32_t)d : (uint32_t)pick;
        }
      }
      uint32_t total;
      const uint32_t ex = warp_exclusive(deg, &total);
      if (i < s_hi) sub_indptr[i] = (IdxT)(run + ex);
      run += total;
    }
    uint32_t cta_total;
    const uint32_t my_prefix = cta_exclusive(run, smem, &cta_total);
    if (tid == 0) p.cta_sum[cta] = cta_total;
    grid.sync();

    // ---- B: offsets, draws, first positions
    const uint32_t n_edges = scan_totals(p.cta_sum, n_cta, prefix, smem);
    const uint32_t base_off = prefix[cta] + my_prefix;
    auto sample = [&](auto width) {
      constexpr int W = decltype(width)::value;
      constexpr int G = 32 / W;
      const int grp = lane / W, s = lane & (W - 1);
      // the next seed's list is looked up while the current one is drawn
      auto look = [&](uint32_t i, int64_t& begin, uint32_t& d, uint32_t& off) {
        begin = 0; d = 0; off = 0;
        if (i < s_hi) {
          const int64_t v = (int64_t)__ldcg(seeds + i);
          off = (uint32_t)sub_indptr[i] + base_off;  // this warp wrote it
          if (v >= 0 && v < p.n_nodes) {
            begin = (int64_t)__ldg(p.indptr + v);
            d = (uint32_t)((int64_t)__ldg(p.indptr + v + 1) - begin);
          }
        }
      };
      int64_t begin; uint32_t d, off;
      look(s_lo + grp, begin, d, off);
      for (uint32_t base = s_lo; base < s_hi; base += G) {
        const uint32_t i = base + grp;
        int64_t begin2; uint32_t d2, off2;
        look(i + G, begin2, d2, off2);
        const int64_t o = draw<W>(d, pick, (int64_t)i, p.rng_seed, p.rng_offset + (uint64_t)hop);
        __syncwarp();
        if (i < s_hi) {
          if (s == 0) sub_indptr[i] = (IdxT)off;
          if (o >= 0) {
            const IdxT id = __ldg(p.indices + begin + o);
            ids[off + s] = id;
            note((int64_t)id, n + off + s);
          }
        }
        begin = begin2; d = d2; off = off2;
      }
    };
    if (pick <= 8) sample(std::integral_constant<int, 8>());
    else if (pick <= 16) sample(std::integral_constant<int, 16>());
    else if (pick <= 32) sample(std::integral_constant<int, 32>());
    else {
      for (uint32_t i = s_lo + lane; i < s_hi; i += 32) {
        const uint32_t off = (uint32_t)sub_indptr[i] + base_off;
        sub_indptr[i] = (IdxT)off;
        const int64_t v = (int64_t)__ldcg(seeds + i);
        if (v < 0 || v >= p.n_nodes) continue;
        sample_one_seed(p.indptr, p.indices, v, (int64_t)i, ids + off, pick, p.rng_seed, p.rng_offset + (uint64_t)hop);
        const int64_t d = (int64_t)p.indptr[v + 1] - (int64_t)p.indptr[v];
        for (int k = 0; k < (d < pick ? (int)d : pick); ++k) note((int64_t)ids[off + k], n + off + k);
      }
    }
    if (gtid == 0) sub_indptr[n] = (IdxT)n_edges;
    grid.sync();

    // ---- C: first occurrences among the positions [start, n + n_edges), ranked inside the warp's run
    const uint32_t start = hop == 0 ? 0u : n, stop = n + n_edges;
    const uint32_t run_len = max(((stop - start + n_warps - 1) / n_warps + 31u) & ~31u, 32u);
    const uint32_t k_lo = min(start + gwarp * run_len, stop), k_hi = min(k_lo + run_len, stop);
    uint32_t firsts = 0;
    for (uint32_t base = k_lo; base < k_hi; base += 32) {
      const uint32_t k = base + lane;
      bool first = false;
      if (k < k_hi) {
        const int64_t id = (int64_t)(k < n ? __ldcg(seeds + k) : __ldcg(ids + (k - n)));
        uint32_t v = 0u;
        if (id >= 0 && id < p.n_nodes) v = (uint32_t)__ldcg(p.node_map + id);
        p.val[k] = v;
        first = v == (kPending | k);
      }
      const uint32_t mask = __ballot_sync(0xffffffffu, first);
      if (first) p.rank[k] = firsts + __popc(mask & ((1u << lane) - 1u));
      firsts += __popc(mask);
    }
    const uint32_t before = cta_exclusive(firsts, smem, &cta_total);
    if (lane == 0) p.warp_prefix[gwarp] = before;
    if (tid == 0) p.cta_sum[kMaxCtas + cta] = cta_total;
    grid.sync();

    // ---- D: numbers
    const uint32_t fresh = scan_totals(p.cta_sum + kMaxCtas, n_cta, prefix, smem);
    for (uint32_t k = start + gtid; k < stop; k += n_cta * kThreads) {
      uint32_t v = __ldcg(p.val + k);
      if ((v & kPending) != 0u) {
        const uint32_t pos = v & ~kPending;
        const uint32_t w = (pos - start) / run_len;
        v = start + __ldcg(p.rank + pos) + __ldcg(p.warp_prefix + w) + prefix[w / kWarps];
        if (pos == k) {
          const IdxT id = k < n ? __ldcg(seeds + k) : __ldcg(ids + (k - n));
          p.unique[v] = id;
          p.node_map[(int64_t)id] = p.stamp | v;
        }
      }
      if (k >= n) p.local[hop][k - n] = (IdxT)v;
    }
    n = start + fresh;
    if (gtid == 0) {
      p.header[2 * hop] = (int64_t)n_edges;
      p.header[2 * hop + 1] = (int64_t)n;
    }
    if (hop + 1 < p.n_hops) grid.sync();
  }
  if (gtid == 0) {
    p.header[2 * p.n_hops] = (int64_t)*(volatile int32_t*)p.error;
    *p.error = 0;  // for the next minibatch
    __threadfence_system();
  }
}

struct Scratch { size_t val, rank, warp_prefix, cta_sum, error, total; };

static Scratch plan(int64_t max_positions) {
  auto up = [](size_t v) { return (v + 255) & ~(size_t)255; };
  Scratch w{};
  size_t at = 0;
  w.error = at; at += 256;
  w.val = at; at += up((size_t)max_positions * 4);
  w.rank = at; at += up((size_t)max_positions * 4);
  w.warp_prefix = at; at += up((size_t)kMaxCtas * kWarps * 4);
  w.cta_sum = at; at += up((size_t)2 * kMaxCtas * 4);
  w.total = at;
  return w;
}

// CTAs the device keeps resident, queried once per device
template <typename IdxT>
static int resident_ctas(int dev) {
  static std::mutex m;
  static int cached[64] = {};
  std::lock_guard<std::mutex> lock(m);
  int& slot = cached[dev & 63];
  if (slot == 0) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, minibatch_kernel<IdxT>, kThreads, 0) != cudaSuccess || per_sm < 1) per_sm = 1;
    if (per_sm > 2) per_sm = 2;
    const int n = per_sm * sm_count(dev);
    slot = n > kMaxCtas ? kMaxCtas : n;
  }
  return slot;
}

template <typename IdxT>
static int launch(const f2c_minibatch* a, int64_t max_positions, cudaStream_t st) {
  const char* op = "sample_minibatch";
  unsigned char* ws = (unsigned char*)a->workspace;
  const Scratch w = plan(max_positions);
  Params<IdxT> p;
  p.indptr = (const IdxT*)a->indptr; p.indices = (const IdxT*)a->indices; p.seeds = (const IdxT*)a->seeds;
  p.n_nodes = a->n_nodes; p.n_seeds = (int)a->n_seeds; p.n_hops = a->n_hops;
  for (int h = 0; h < F2C_MAX_HOPS; ++h) {
    const bool on = h < a->n_hops;
    p.pick[h] = on ? a->num_pick[h] : 0;
    p.sub_indptr[h] = on ? (IdxT*)a->sub_indptr[h] : nullptr;
    p.ids[h] = on ? (IdxT*)a->ids[h] : nullptr;
    p.local[h] = on ? (IdxT*)a->local[h] : nullptr;
  }
  p.unique = (IdxT*)a->unique;
  p.node_map = (unsigned long long*)a->node_map;
  p.stamp = (unsigned long long)(0xffffffffu - a->epoch) << 32;
  p.val = (uint32_t*)(ws + w.val); p.rank = (uint32_t*)(ws + w.rank); p.warp_prefix = (uint32_t*)(ws + w.warp_prefix);
  p.cta_sum = (uint32_t*)(ws + w.cta_sum); p.error = (int32_t*)(ws + w.error);
  p.header = a->header;
  p.rng_seed = a->rng_seed; p.rng_offset = a->rng_offset;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) dev = 0;
  int grid = resident_ctas<IdxT>(dev);
  // few seeds: fewer CTAs make cheaper barriers, as long as the last hop's positions still fill them
  const int64_t tiles = ceil_div(max_positions, kThreads);
  if (grid > tiles) grid = (int)tiles;
  void* args[] = {(void*)&p};
  cudaError_t e = cudaLaunchCooperativeKernel((const void*)minibatch_kernel<IdxT>, dim3((unsigned)grid), dim3(kThreads), args, 0, st);
  if (e != cudaSuccess) return set_error(F2C_ERR_CUDA, "%s: cooperative launch: %s", op, cudaGetErrorString(e));
  return check_launch(op);
}

// largest number of positions (seeds + sampled ids) of any hop; -1 when a size limit is exceeded
static int64_t most_positions(int64_t n_nodes, int64_t n_seeds, int n_hops, const int* num_pick) {
  int64_t rows = n_seeds, most = 0;
  for (int h = 0; h < n_hops; ++h) {
    const int64_t positions = rows * (num_pick[h] + 1);
    if (positions >= (1ll << 31) - 1) return -1;
    if (positions > most) most = positions;
    rows = positions < n_nodes ? positions : n_nodes;
  }
  return most;
}

}  // namespace mb
}  // namespace f2c

using namespace f2c;

extern "C" int64_t f2c_sample_minibatch_workspace(int64_t n_nodes, int64_t n_seeds, int n_hops, const int* num_pick_host) {
  if (n_nodes < 1 || n_seeds < 1 || n_hops < 1 || n_hops > F2C_MAX_HOPS || num_pick_host == nullptr) return 0;
  for (int h = 0; h < n_hops; ++h)
    if (num_pick_host[h] < 1 || num_pick_host[h] > kMaxPick) return 0;
  const int64_t most = mb::most_positions(n_nodes, n_seeds, n_hops, num_pick_host);
  return most < 0 ? 0 : (int64_t)mb::plan(most).total;
}

extern "C" int f2c_sample_minibatch(const f2c_minibatch* a, void* stream) {
  const char* op = "sample_minibatch";
  F2C_REQUIRE(a != nullptr, F2C_ERR_INVALID, "%s: null pointer", op);
  F2C_REQUIRE(is_index_dtype(a->index_dtype), F2C_ERR_UNSUPPORTED, "%s: ids must be int32 or int64", op);
  F2C_REQUIRE(a->n_nodes >= 1 && a->n_seeds >= 1 && a->n_hops >= 1 && a->n_hops <= F2C_MAX_HOPS, F2C_ERR_INVALID, "%s: bad sizes", op);
  F2C_REQUIRE(a->indptr && a->seeds && a->unique && a->node_map && a->header && a->workspace && aligned(a->workspace, 256),
              F2C_ERR_INVALID, "%s: null or misaligned pointer", op);
  for (int h = 0; h < a->n_hops; ++h) {
    F2C_REQUIRE(a->num_pick[h] >= 1 && a->num_pick[h] <= kMaxPick, F2C_ERR_LIMIT, "%s: num_pick must be in [1, %d]", op, kMaxPick);
    F2C_REQUIRE(a->sub_indptr[h] && a->ids[h] && a->local[h], F2C_ERR_INVALID, "%s: null pointer", op);
  }
  const int64_t most = mb::most_positions(a->n_nodes, a->n_seeds, a->n_hops, a->num_pick);
  F2C_REQUIRE(most >= 0, F2C_ERR_LIMIT, "%s: at most 2^31 - 2 ids per hop", op);
  F2C_REQUIRE(a->workspace_bytes >= (int64_t)mb::plan(most).total, F2C_ERR_INVALID, "%s: the workspace is too small", op);
  return a->index_dtype == F2C_I32 ? mb::launch<int32_t>(a, most, (cudaStream_t)stream) : mb::launch<int64_t>(a, most, (cudaStream_t)stream);
}
