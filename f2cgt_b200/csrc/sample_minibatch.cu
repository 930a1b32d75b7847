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
//  * a group of 8, 16 or 32 lanes draws for one seed: each lane makes one draw of Floyd's subset algorithm, a match and a vote settle
//    repeated draws, and the reads of the neighbour ids go out together and are waited for behind the next seed's draws;
//  * whoever finds a first occurrence also looks up the node's list for the next hop, whose offsets then come out of the scan
//    that numbers the nodes.
// Per hop and barrier: B draws, first positions | C which occurrences are first, ranked; their lists | D numbers, offsets of the next
// hop.  The first hop's lists (A) take a barrier of their own only when they are many: every CTA scans up to 2048 seeds itself.  Every
// warp owns a contiguous run of seeds (A, B) and of positions (C), so prefix sums are warp prefix + CTA prefix + one array of CTA
// totals.
//
// Latency bound: chains of dependent reads between grid barriers.  Measured on B200, on 2.4 M nodes of mean degree 50, 1024 seeds, fan-out
// 12,12,12 (708,000 edges in the last hop): 75 us against 87 with a phase and a barrier more per hop, for the degrees, and one position
// at a time per thread; 64 seeds, 5,5,5: 35.5 against 39; 8000 seeds, 5,5,12: 108 against 124.  (Three sample_block kernels: 37 + 49 + 123 us
// and three host reads.)
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
constexpr int kSmall = 4;  // seeds per thread up to which every CTA scans the first hop's lists itself
constexpr int kBatch = 4;  // positions per thread whose chains of reads go on side by side

// neighbours of a seed: where its list begins, its degree, where its samples go
struct __align__(16) List {
  int64_t begin;
  uint32_t degree, offset;
};

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
  unsigned long long* warp_prefix;  // per warp: first occurrences of the CTA's warps before it, and in the upper half their samples in the next hop
  unsigned long long* cta_sum;      // [2 * kMaxCtas]
  List* lists;               // per seed of the hop
  List* found;               // per first occurrence: offset inside the warp's run
  int32_t* error;
  int64_t* header;           // [2 * n_hops + 1], host memory: edges and distinct nodes per hop, error
  uint64_t rng_seed, rng_offset;
};

template <typename T>
__device__ __forceinline__ T warp_exclusive(T v, T* total) {
  const int lane = threadIdx.x & 31;
  T inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  *total = __shfl_sync(0xffffffffu, inc, 31);
  return inc - v;
}

// totals of this CTA's warps -> exclusive prefix per warp (returned to every lane of it) and the CTA's total in *sum
template <typename T>
__device__ __forceinline__ T cta_exclusive(T warp_total, T* smem, T* sum) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) smem[wid] = warp_total;
  __syncthreads();
  T total;
  const T ex = warp_exclusive(lane < kWarps ? smem[lane] : (T)0, &total);
  *sum = total;
  return __shfl_sync(0xffffffffu, ex, wid);
}

// exclusive prefix of the CTA totals into shared memory; returns the grand total to every thread
template <typename T>
__device__ __forceinline__ T scan_totals(const T* totals, int n_cta, T* prefix, T* smem) {
  const T v = (int)threadIdx.x < n_cta ? __ldcg(totals + threadIdx.x) : (T)0;
  T warp_total, sum;
  const T ex = warp_exclusive(v, &warp_total);
  const T before = cta_exclusive(warp_total, smem, &sum);
  prefix[threadIdx.x] = before + ex;
  __syncthreads();
  return sum;
}

// Draws of one seed by a group of W lanes (num_pick <= W): offset of this lane's neighbour inside the seed's list, -1 for
// lanes without one.  All lanes of the warp call; d = in-degree, below 2^32.
// Floyd: draw s is t_s unless t_s was drawn before, then j_s = d - num_pick + s.  What was drawn before holds t_s if an earlier t is the same
// number, or if an earlier draw q took its j_q and that is t_s - which only q = t_s - (d - num_pick) can have.  So one match and
// a vote or two settle all draws at once (a loop over the draws, one shuffle each, was a chain of num_pick of them).
template <int W>
__device__ __forceinline__ int64_t draw(uint32_t d, int num_pick, int64_t position, uint64_t rng_seed, uint64_t rng_offset) {
  const int lane = threadIdx.x & 31, s = lane & (W - 1), group = lane - s;
  const bool all = d <= (uint32_t)num_pick, on = !all && s < num_pick;
  uint32_t t = 0xffffffffu, j = 0u;  // t < j + 1 <= d, so no draw is 0xffffffff
  bool chained = false;
  int from = 0;
  if (on) {
    const uint4 r = Philox(rng_seed, rng_offset)((uint64_t)position * (kMaxPick / 2) + (uint64_t)(s >> 1));
    const uint64_t bits = (s & 1) == 0 ? ((uint64_t)r.x << 32 | r.y) : ((uint64_t)r.z << 32 | r.w);
    const uint32_t low = d - (uint32_t)num_pick;
    j = low + (uint32_t)s;
    t = (uint32_t)__umul64hi(bits, (uint64_t)j + 1u);
    chained = t >= low && t < j;
    from = chained ? (int)(t - low) : 0;
  }
  const uint32_t same = __match_any_sync(0xffffffffu, t);
  const bool repeated = on && ((same >> group) & ((1u << s) - 1u)) != 0u;
  uint32_t taken = __ballot_sync(0xffffffffu, repeated);
  for (uint32_t before = 0u; before != taken;) {  // ends after num_pick rounds at the latest: a draw only hangs on earlier ones
    before = taken;
    taken = __ballot_sync(0xffffffffu, repeated || (chained && ((before >> (group + from)) & 1u) != 0u));
  }
  if (all) return s < (int)d ? s : -1;
  return s < num_pick ? (int64_t)((taken >> lane) & 1u ? j : t) : -1;
}

// 56 registers: two CTAs of the kernel leave an eighth of an SM's registers to the consumer's kernels, so that the next minibatch starts while
// they run (64: it waits for them, 109 us a minibatch instead of 90; one CTA per SM with 96: 112).
template <typename IdxT>
__global__ void __maxnreg__(56) minibatch_kernel(const Params<IdxT> p) {
  cg::grid_group grid = cg::this_grid();
  __shared__ unsigned long long smem[kWarps];
  __shared__ unsigned long long prefix[kThreads];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, cta = blockIdx.x, n_cta = gridDim.x;
  const uint32_t gwarp = cta * kWarps + wid, n_warps = n_cta * kWarps;
  const uint32_t gtid = cta * kThreads + tid;
  uint32_t n = (uint32_t)p.n_seeds;
  uint32_t n_edges = 0;   // of this hop
  uint32_t base_off = 0;  // what the offsets in p.lists still lack
  auto note = [&](int64_t id, uint32_t pos) {  // an occurrence of `id` at position pos
    if (id < 0 || id >= p.n_nodes) { *(volatile int32_t*)p.error = id < 0 ? 2 : 3; return; }
    atomicMin(p.node_map + id, p.stamp | kPending | pos);
  };
  auto list_of = [&](int64_t v, int pick, int64_t& begin, uint32_t& d) -> uint32_t {  // number of neighbours that are sampled
    begin = 0; d = 0;
    if (v < 0 || v >= p.n_nodes) return 0u;
    begin = (int64_t)__ldg(p.indptr + v);
    d = (uint32_t)((int64_t)__ldg(p.indptr + v + 1) - begin);
    return d < (uint32_t)pick ? d : (uint32_t)pick;
  };

  // ---- A: the first hop's lists
  {
    const uint32_t per_warp = (n + n_warps - 1) / n_warps;
    if (n <= kSmall * kThreads) {
      // few seeds: every CTA scans all of them, which costs it the same chain of reads and no barrier
      const uint32_t lo = cta * kWarps * per_warp, hi = lo + kWarps * per_warp;
      int64_t v[kSmall], begin[kSmall];
      uint32_t d[kSmall], deg[kSmall];
#pragma unroll
      for (int c = 0; c < kSmall; ++c) { const uint32_t i = c * kThreads + tid; v[c] = i < n ? (int64_t)__ldg(p.seeds + i) : -1; }
#pragma unroll
      for (int c = 0; c < kSmall; ++c) deg[c] = list_of(v[c], p.pick[0], begin[c], d[c]);
#pragma unroll
      for (int c = 0; c < kSmall; ++c) {
        const uint32_t i = c * kThreads + tid;
        if (c * kThreads < n) {  // CTA uniform
          uint32_t warp_total;
          unsigned long long sum;
          const uint32_t ex = warp_exclusive(deg[c], &warp_total);
          const uint32_t off = n_edges + (uint32_t)cta_exclusive((unsigned long long)warp_total, smem, &sum) + ex;
          if (i >= lo && i < hi && i < n) {
            note(v[c], i);
            p.lists[i] = List{begin[c], d[c], off};
          }
          n_edges += (uint32_t)sum;
        }
      }
      __syncthreads();
    } else {
      const uint32_t s_lo = min(gwarp * per_warp, n), s_hi = min(s_lo + per_warp, n);
      uint32_t run = 0;
      for (uint32_t base = s_lo; base < s_hi; base += 32) {
        const uint32_t i = base + lane;
        int64_t begin;
        uint32_t d, deg = 0, total;
        if (i < s_hi) {
          const int64_t v = (int64_t)__ldg(p.seeds + i);
          note(v, i);
          deg = list_of(v, p.pick[0], begin, d);
        }
        const uint32_t ex = warp_exclusive(deg, &total);
        if (i < s_hi) p.lists[i] = List{begin, d, run + ex};
        run += total;
      }
      unsigned long long cta_total;
      const uint32_t my_prefix = (uint32_t)cta_exclusive((unsigned long long)run, smem, &cta_total);
      if (tid == 0) p.cta_sum[cta] = cta_total;
      grid.sync();
      n_edges = (uint32_t)scan_totals(p.cta_sum, n_cta, prefix, smem);
      base_off = (uint32_t)prefix[cta] + my_prefix;
    }
  }

  for (int hop = 0; hop < p.n_hops; ++hop) {
    const IdxT* seeds = hop == 0 ? p.seeds : p.unique;
    const int pick = p.pick[hop];
    const bool last = hop + 1 == p.n_hops;
    IdxT* sub_indptr = p.sub_indptr[hop];
    IdxT* ids = p.ids[hop];

    // ---- B: draws, first positions
    const uint32_t per_warp = (n + n_warps - 1) / n_warps;
    const uint32_t s_lo = min(gwarp * per_warp, n), s_hi = min(s_lo + per_warp, n);
    auto sample = [&](auto width) {
      constexpr int W = decltype(width)::value;
      constexpr int G = 32 / W;
      const int grp = lane / W, s = lane & (W - 1);
      auto look = [&](uint32_t i) {
        int4 w = make_int4(0, 0, 0, 0);
        if (i < s_hi) w = __ldcg(reinterpret_cast<const int4*>(p.lists + i));
        return w;
      };
      // The next seed's list is looked up while the current one is drawn, and an id is waited for after the next draw.
      int4 list = look(s_lo + grp);
      IdxT id = 0;
      uint32_t slot = 0xffffffffu;
      auto keep = [&]() {
        if (slot != 0xffffffffu) {
          ids[slot] = id;
          note((int64_t)id, n + slot);
        }
      };
      for (uint32_t base = s_lo; base < s_hi; base += G) {
        const uint32_t i = base + grp;
        const int4 next = look(i + G);
        const int64_t o = draw<W>((uint32_t)list.z, pick, (int64_t)i, p.rng_seed, p.rng_offset + (uint64_t)hop);
        __syncwarp();
        keep();
        slot = 0xffffffffu;
        if (i < s_hi) {
          const uint32_t off = (uint32_t)list.w + base_off;
          if (s == 0) sub_indptr[i] = (IdxT)off;
          if (o >= 0) {
            const int64_t begin = (int64_t)((uint64_t)(uint32_t)list.y << 32 | (uint32_t)list.x);
            id = __ldg(p.indices + begin + o);
            slot = off + s;
          }
        }
        list = next;
      }
      keep();
    };
    if (pick <= 8) sample(std::integral_constant<int, 8>());
    else if (pick <= 16) sample(std::integral_constant<int, 16>());
    else if (pick <= 32) sample(std::integral_constant<int, 32>());
    else {
      for (uint32_t i = s_lo + lane; i < s_hi; i += 32) {
        const uint32_t off = (uint32_t)__ldcg(reinterpret_cast<const int4*>(p.lists + i)).w + base_off;
        sub_indptr[i] = (IdxT)off;
        const int64_t v = (int64_t)__ldcg(seeds + i);
        if (v < 0 || v >= p.n_nodes) continue;
        sample_one_seed(p.indptr, p.indices, v, (int64_t)i, ids + off, pick, p.rng_seed, p.rng_offset + (uint64_t)hop);
        const int64_t d = (int64_t)p.indptr[v + 1] - (int64_t)p.indptr[v];
        for (int k = 0; k < (d < pick ? (int)d : pick); ++k) note((int64_t)ids[off + k], n + off + k);
      }
    }
    base_off = 0;
    if (gtid == 0) sub_indptr[n] = (IdxT)n_edges;
    grid.sync();

    // ---- C: first occurrences among the positions [start, n + n_edges), ranked inside the warp's run.  Where another hop follows, their lists
    // too; then the seeds, whose numbers carry over, are positions as well.
    const uint32_t start = hop == 0 || !last ? 0u : n, stop = n + n_edges;
    const uint32_t run_len = max(((stop - start + n_warps - 1) / n_warps + 31u) & ~31u, 32u);
    const uint32_t k_lo = min(start + gwarp * run_len, stop), k_hi = min(k_lo + run_len, stop);
    const uint32_t old = hop == 0 ? 0u : n;  // positions below: nodes numbered in an earlier hop
    uint32_t firsts = 0, edges = 0;
    for (uint32_t base = k_lo; base < k_hi; base += 32 * kBatch) {
      int64_t id[kBatch];
      uint32_t v[kBatch];
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
        const uint32_t k = base + 32 * b + lane;
        id[b] = k < k_hi && k >= old ? (int64_t)(k < n ? __ldcg(seeds + k) : __ldcg(ids + (k - n))) : -1;
      }
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
        const uint32_t k = base + 32 * b + lane;
        v[b] = k < old ? (kPending | k) : 0u;
        if (id[b] >= 0 && id[b] < p.n_nodes) v[b] = (uint32_t)__ldcg(p.node_map + id[b]);
      }
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
        const uint32_t k = base + 32 * b + lane;
        if (base + 32 * b >= k_hi) break;  // warp uniform
        const bool first = k < k_hi && v[b] == (kPending | k);
        if (k < k_hi) p.val[k] = v[b];
        const uint32_t mask = __ballot_sync(0xffffffffu, first);
        if (first) p.rank[k] = firsts + __popc(mask & ((1u << lane) - 1u));
        firsts += __popc(mask);
        if (!last) {
          int64_t begin = 0;
          uint32_t d = 0, deg = 0, total;
          if (first && k < old) {
            const int4 w = __ldcg(reinterpret_cast<const int4*>(p.lists + k));
            begin = (int64_t)((uint64_t)(uint32_t)w.y << 32 | (uint32_t)w.x);
            d = (uint32_t)w.z;
            deg = min(d, (uint32_t)p.pick[hop + 1]);
          } else if (first) {
            deg = list_of(id[b], p.pick[hop + 1], begin, d);
          }
          const uint32_t ex = warp_exclusive(deg, &total);
          if (first) p.found[k] = List{begin, d, edges + ex};
          edges += total;
        }
      }
    }
    unsigned long long cta_total;
    const unsigned long long before = cta_exclusive((unsigned long long)edges << 32 | firsts, smem, &cta_total);
    if (lane == 0) p.warp_prefix[gwarp] = before;
    if (tid == 0) p.cta_sum[kMaxCtas + cta] = cta_total;
    grid.sync();

    // ---- D: numbers; the next hop's lists.  The upper half of the prefixes counts edges, the lower half nodes (both below 2^31).
    const unsigned long long fresh = scan_totals(p.cta_sum + kMaxCtas, n_cta, prefix, smem);
    const uint32_t step = n_cta * kThreads;
    for (uint32_t base = start + gtid; base < stop; base += step * kBatch) {
      uint32_t v[kBatch], rank[kBatch];
      unsigned long long ahead[kBatch];
#pragma unroll
      for (int b = 0; b < kBatch; ++b) v[b] = stop - base > b * step ? __ldcg(p.val + base + b * step) : 0u;
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
        rank[b] = 0u;
        ahead[b] = 0ull;
        if ((v[b] & kPending) != 0u) {
          const uint32_t pos = v[b] & ~kPending, w = (pos - start) / run_len;
          rank[b] = __ldcg(p.rank + pos);
          ahead[b] = __ldcg(p.warp_prefix + w) + prefix[w / kWarps];
        }
      }
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
        const uint32_t k = base + b * step;
        if (stop - base <= b * step) break;
        uint32_t number = v[b];
        if ((v[b] & kPending) != 0u) {
          number = start + rank[b] + (uint32_t)ahead[b];
          if ((v[b] & ~kPending) == k) {
            if (k >= old) {
              const IdxT id = k < n ? __ldcg(seeds + k) : __ldcg(ids + (k - n));
              p.unique[number] = id;
              p.node_map[(int64_t)id] = p.stamp | number;
            }
            if (!last) {
              const int4 w = __ldcg(reinterpret_cast<const int4*>(p.found + k));
              *reinterpret_cast<int4*>(p.lists + number) = make_int4(w.x, w.y, w.z, w.w + (int)(uint32_t)(ahead[b] >> 32));
            }
          }
        }
        if (k >= n) p.local[hop][k - n] = (IdxT)number;
      }
    }
    const uint32_t sampled = n_edges;
    n = start + (uint32_t)fresh;
    n_edges = (uint32_t)(fresh >> 32);
    if (gtid == 0) {
      p.header[2 * hop] = (int64_t)sampled;
      p.header[2 * hop + 1] = (int64_t)n;
    }
    if (!last) grid.sync();
  }
  if (gtid == 0) {
    p.header[2 * p.n_hops] = (int64_t)*(volatile int32_t*)p.error;
    *p.error = 0;  // for the next minibatch
    __threadfence_system();
  }
}

struct Scratch { size_t val, rank, warp_prefix, cta_sum, lists, found, error, total; };

// max_seeds, max_found: seeds of any hop, and positions of any hop that another one follows
static Scratch plan(int64_t max_positions, int64_t max_seeds, int64_t max_found) {
  auto up = [](size_t v) { return (v + 255) & ~(size_t)255; };
  Scratch w{};
  size_t at = 0;
  w.error = at; at += 256;
  w.val = at; at += up((size_t)max_positions * 4);
  w.rank = at; at += up((size_t)max_positions * 4);
  w.warp_prefix = at; at += up((size_t)kMaxCtas * kWarps * 8);
  w.cta_sum = at; at += up((size_t)2 * kMaxCtas * 8);
  w.lists = at; at += up((size_t)max_seeds * sizeof(List));
  w.found = at; at += up((size_t)max_found * sizeof(List));
  w.total = at;
  return w;
}

// largest numbers of positions (seeds + sampled ids) and of seeds of any hop; positions = -1 when a size limit is exceeded
struct Sizes {
  int64_t positions, seeds, found;  // found: positions of any hop but the last
  size_t workspace() const { return plan(positions, seeds, found).total; }
};
static Sizes most(int64_t n_nodes, int64_t n_seeds, int n_hops, const int* num_pick) {
  int64_t rows = n_seeds;
  Sizes m{0, 0, 0};
  for (int h = 0; h < n_hops; ++h) {
    const int64_t positions = rows * (num_pick[h] + 1);
    if (positions >= (1ll << 31) - 1) return Sizes{-1, 0, 0};
    if (rows > m.seeds) m.seeds = rows;
    if (positions > m.positions) m.positions = positions;
    if (h + 1 < n_hops && positions > m.found) m.found = positions;
    rows = positions < n_nodes ? positions : n_nodes;
  }
  return m;
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
static int launch(const f2c_minibatch* a, const Sizes& sizes, cudaStream_t st) {
  const char* op = "sample_minibatch";
  unsigned char* ws = (unsigned char*)a->workspace;
  const Scratch w = plan(sizes.positions, sizes.seeds, sizes.found);
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
  p.val = (uint32_t*)(ws + w.val); p.rank = (uint32_t*)(ws + w.rank);
  p.warp_prefix = (unsigned long long*)(ws + w.warp_prefix); p.cta_sum = (unsigned long long*)(ws + w.cta_sum);
  p.lists = (List*)(ws + w.lists); p.found = (List*)(ws + w.found); p.error = (int32_t*)(ws + w.error);
  p.header = a->header;
  p.rng_seed = a->rng_seed; p.rng_offset = a->rng_offset;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) dev = 0;
  int grid = resident_ctas<IdxT>(dev);
  // few seeds: fewer CTAs make cheaper barriers, as long as the last hop's positions still fill them
  const int64_t tiles = ceil_div(sizes.positions, kThreads);
  if (grid > tiles) grid = (int)tiles;
  void* args[] = {(void*)&p};
  cudaError_t e = cudaLaunchCooperativeKernel((const void*)minibatch_kernel<IdxT>, dim3((unsigned)grid), dim3(kThreads), args, 0, st);
  if (e != cudaSuccess) return set_error(F2C_ERR_CUDA, "%s: cooperative launch: %s", op, cudaGetErrorString(e));
  return check_launch(op);
}

}  // namespace mb
}  // namespace f2c

using namespace f2c;

extern "C" int64_t f2c_sample_minibatch_workspace(int64_t n_nodes, int64_t n_seeds, int n_hops, const int* num_pick_host) {
  if (n_nodes < 1 || n_seeds < 1 || n_hops < 1 || n_hops > F2C_MAX_HOPS || num_pick_host == nullptr) return 0;
  for (int h = 0; h < n_hops; ++h)
    if (num_pick_host[h] < 1 || num_pick_host[h] > kMaxPick) return 0;
  const mb::Sizes sizes = mb::most(n_nodes, n_seeds, n_hops, num_pick_host);
  return sizes.positions < 0 ? 0 : (int64_t)sizes.workspace();
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
  const mb::Sizes sizes = mb::most(a->n_nodes, a->n_seeds, a->n_hops, a->num_pick);
  F2C_REQUIRE(sizes.positions >= 0, F2C_ERR_LIMIT, "%s: at most 2^31 - 2 ids per hop", op);
  F2C_REQUIRE(a->workspace_bytes >= (int64_t)sizes.workspace(), F2C_ERR_INVALID, "%s: the workspace is too small", op);
  return a->index_dtype == F2C_I32 ? mb::launch<int32_t>(a, sizes, (cudaStream_t)stream) : mb::launch<int64_t>(a, sizes, (cudaStream_t)stream);
}
