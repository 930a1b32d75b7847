// K-means assignment on the 5th-generation tensor cores (tcgen05, TMEM accumulators).
// Reference operator: KMeans.predict (src/kmeans.cu:77-98, RAFT kmeans_predict), i.e.
// labels[i] = first argmin_c dist(x_i, y_c) with dist = squared L2 or cosine distance.
//
// The n*k*d contraction S = X * Y^T is the only dense GEMM on the path, so it runs as tcgen05.mma.kind::f16 with M = 128
// points per tile, N = all (<= 256) centres, fp32 accumulators in TMEM, operands in shared memory in the canonical
// no-swizzle K-major layout.
//
//  * Accuracy.  A value is split into two f16 numbers, x = h1 + h2 + (rest below 2^-22 |x|, or 2^-25 where h2 is subnormal),
//    and the products h1*g1 + h2*g1 + h1*g2 are obtained in ONE GEMM by concatenating along K:
//    A' = [x1 | x2 | x1], B' = [y1 | y1 | y2] (K = 3d).  f16 has five exponent bits, so operands are scaled by powers of two
//    first: the rows of X each by their own largest value (a common factor of a point's scores does not change its arg-max;
//    squared L2: only rows that lie further out than the centres), the rows of Y by their norm (cosine) or by the largest
//    norm of all (squared L2).  (Two f16 carry 22 bits where 3 x tf32 carried 21 at half the rate and twice the bytes, and
//    3 x bf16 16, which sent several per cent of 64-dimensional points to the exact scorer.)
//  * The whole score comes out of the GEMM.  argmin_c |y_c|^2 - 2 x.y_c = argmax_c (x.y_c - |y_c|^2 / 2): one more chunk of K
//    carries powers of two on the point side and three f16 pieces of -|y_c|^2/2 on the centre side, so the epilogue is a pure
//    arg-max.  A column that is padding carries -65504 in that chunk.
//  * The epilogue reads the 128 x 256 scores with tcgen05.ld (one point per thread) and finds the best score and whether it is
//    the only one within the error bound of the product.  A point where it is not goes to a list of the CTA, whose warps give it
//    the label of the exact fp32 scorer (kmeans.cu) at the end, so every label equals the label of that kernel.  (Squared distances of points
//    that lie some 10^3 times further out than the centres differ by less than their own fp32 rounding; there the score, which leaves |x|^2
//    out, still decides, for the nearer centre.)
//  * Overlap.  A CTA has 22 warps with fixed roles: three groups of four epilogue warps, two of four producer warps, which have their
//    points' rows copied to shared memory ahead, split them and store them into a ring of A tiles, and two warps whose first lanes issue the
//    MMAs, each into its pair of accumulators of 128 columns.  They meet at mbarriers only: a half of the columns is made while the epilogue
//    reads another, and a group ends a tile while the two others read theirs.
//    What bounds it: up to 16 dimensions the maxima (one per point and centre and direction, two cycles per three-operand instruction: ALU
//    pipe 68 % busy) and the latency of the chain accumulator free - MMAs - accumulator full; more dimensions: no unit alone (61 % at 32, 45 % at 64),
//    warps wait for accumulators and rows and, at 64, for instructions.
//    Measured, 2,449,029 points against 256 centres, whole call between two events, L2 flushed (before, calls in a row: sixteen warps that all
//    loaded, split, waited and searched, one barrier per tile, 3 x tf32 or 3 x bf16, undecided points in a second kernel): 8 dimensions 153 ->
//    107 us (102 in a row), 16: 193 -> 119, 24: 227 -> 148, 32: 265 -> 160, 64: 400 -> 318; 100 centres of 8 dimensions 118 -> 79, of 64: 357 ->
//    240.  Two epilogue groups instead of three: 8 dimensions 9 more.  Few points: 5000 x 8 20 -> 14, 40,000 x 8 20 -> 16, 149,000 x 32 37 -> 31
//    (the events alone are 3 of these); slower: 149,000 x 64 47 -> 48 in a row.
//    Every wait on an mbarrier is bounded; on expiry an error code is recorded, no further wait is made and no copy started, and the exact
//    scorer assigns all points of the CTA.  Rows that were asked for may still arrive then, so it works where no copy is aimed, over the operands.
//    The copies and MMAs are waited for at the common exit, in front of the freeing of the TMEM.
#pragma once
#include <cooperative_groups.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "kmeans_fit.cuh"

namespace f2c {

namespace tc {

constexpr int kTileM = 128;
constexpr int kMaxN = 256;
constexpr uint32_t kWaitLimit = 1u << 18, kWaitHint = 4000;  // tries, and nanoseconds that one may take: about a second
constexpr int kEpilogueGroups = 3, kEpilogueWarps = 4 * kEpilogueGroups, kProducerWarps = 8;
constexpr int kMmaWarp = kEpilogueWarps + kProducerWarps, kMmaWarps = 2;  // one per pair of accumulators of 128 columns
constexpr int kThreads = 32 * (kMmaWarp + kMmaWarps);
constexpr int kList = 1024;    // undecided points that a CTA keeps in shared memory
constexpr float kTiny = 0x1p-100f;  // squared lengths below: the exact scorer's products run out of exponent, and a score says nothing of its labels
constexpr int kBoundRing = 8;  // tiles whose error bounds are kept; more than the A ring and the two accumulators hold together

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor, K-major, no swizzle: element (row r, 16-byte K chunk c) lives at
// start + (r % 8) * 16 + (r / 8) * SBO + c * LBO.
__device__ __forceinline__ uint64_t make_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  uint32_t lo = ((addr & 0x3FFFFu) >> 4) | ((lbo >> 4) << 16);
  uint32_t hi = (sbo >> 4) | (1u << 14);  // bits 46-47: descriptor version 1 (sm_100); layout type 0 = no swizzle
  return ((uint64_t)hi << 32) | lo;
}

__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t"
      "}\n" ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u)
      : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}

__device__ __forceinline__ void mbar_init(uint32_t mbar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t mbar) {
  asm volatile("{\n\t.reg .b64 s;\n\tmbarrier.arrive.shared::cta.b64 s, [%0];\n\t}" ::"r"(mbar) : "memory");
}

// A role's waits.  One that runs out is reported (code = 1 + tiles done) and no later one waits.
struct Waiter {
  int32_t* error;
  bool gave_up;
  __device__ __forceinline__ bool operator()(uint32_t mbar, uint32_t parity, int code) {
    if (gave_up) return false;
    for (uint32_t it = 0; it < kWaitLimit; ++it) {
      uint32_t done;
      asm volatile(
          "{\n\t.reg .pred p;\n\t"
          "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t}\n"
          : "=r"(done) : "r"(mbar), "r"(parity), "r"(kWaitHint) : "memory");
      if (done) return true;
    }
    gave_up = true;
    atomicExch(error, code);
    return false;
  }
};

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}

// The loads issued so far are complete; naming the registers keeps their uses behind the wait.
__device__ __forceinline__ void tmem_wait(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                 "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])::"memory");
}

struct Params {
  const float* x;
  const float* y;
  int64_t* labels;
  int32_t* undecided;  // how many points the exact scorer assigned
  int32_t* error;      // non-zero when a bounded wait expired
  int64_t n;
  int k, d;
  int metric;
  int x_aligned;       // x starts on a 16-byte boundary
  int x_wide, y_wide;  // rows can be read as float4
  uint32_t never;      // ~0, which the kernel does not know: see arrived()
  float eps;   // relative error bound of one score
};

// What a fit needs beside them (kmeans_fit_tc.cu): labels, list and count above are unused then.
struct FitParams : Params {
  FitState* state;
  float* centers;              // = y
  uint16_t* labels16;          // kUndecided until the exact scorer has been there
  uint16_t* summed16;          // the labels that sums and counts hold; kUndecided: none yet
  long long* sums;             // [k][d] fixed-point sums of the clusters
  uint32_t* counts;            // [k] and how many points they have
  const uint32_t* maxima;      // [d] largest |x| of a column, as float bits
  double* shifts;              // [CTA] squared shift of the centres that it replaced
  int iterations;
  double tol;
};
constexpr uint32_t kUndecided = 0xffffu;

__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// True once `any`, a maximum over magnitudes that were read, is there: its bits are never `never`.  The compiler does not know that, so whoever
// branches on it waits for the reads.  (any >= 0 in its place is folded to a constant, and with it goes the wait.)
__device__ __forceinline__ bool arrived(float any, uint32_t never) { return __float_as_uint(any) != never; }

__device__ __forceinline__ float sqrt_approx(float v) {
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ void add_if_ge(int& sum, float a, float b, int add) {
  asm("{\n\t.reg .pred q;\n\tsetp.ge.f32 q, %1, %2;\n\t@q add.s32 %0, %0, %3;\n\t}" : "+r"(sum) : "f"(a), "f"(b), "r"(add));
}

__device__ __forceinline__ float power2f(int e) { return __int_as_float((127 + e) << 23); }  // -127 < e < 128
// |v| < 2^e for the largest such v; 0 for v = 0 and for what is not finite
__device__ __forceinline__ int exponent_above(float v) {
  const int b = (int)((__float_as_uint(v) & 0x7fffffffu) >> 23);
  return b == 0 || b == 255 ? 0 : b - 126;
}

// v = c1 + c2 + rest: eight values -> two 16-byte chunks of f16
__device__ __forceinline__ void split8(const float (&v)[8], uint4& c1, uint4& c2) {
  uint32_t w1[4], w2[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const __half2 a = __floats2half2_rn(v[2 * e], v[2 * e + 1]);
    const float2 f = __half22float2(a);
    const __half2 b = __floats2half2_rn(v[2 * e] - f.x, v[2 * e + 1] - f.y);
    w1[e] = *reinterpret_cast<const uint32_t*>(&a);
    w2[e] = *reinterpret_cast<const uint32_t*>(&b);
  }
  c1 = make_uint4(w1[0], w1[1], w1[2], w1[3]);
  c2 = make_uint4(w2[0], w2[1], w2[2], w2[3]);
}

// Eight values of a row from column t on; zeros behind its end and where !on.  They come from L2: in a fit other SMs have written them.
__device__ __forceinline__ void load8(const float* row, int t, int d, bool wide, bool on, float (&v)[8]) {
  if (wide) {  // d % 4 == 0
    const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const float4 a = on && t < d ? __ldcg(reinterpret_cast<const float4*>(row + t)) : none;
    const float4 b = on && t + 4 < d ? __ldcg(reinterpret_cast<const float4*>(row + t + 4)) : none;
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = on && t + e < d ? __ldcg(row + t + e) : 0.0f;
  }
}

// How a warp reads rows of C chunks of eight columns: lane = (row of R, chunk of CL), chunk fastest.  PAD bytes between the operands'
// chunks make the eight lanes of a 16-byte store touch eight bank groups.
template <int C>
struct Lanes {
  static constexpr int CL = C <= 2 ? C : C <= 4 ? 4 : 8;  // lanes per row
  static constexpr int R = 32 / CL;                       // rows of one read
  static constexpr int PAD = CL == 1 ? 0 : 128 / CL;
  // A producer warp's rows of a tile come in PARTS of ROWS rows, one bulk copy each.
  static constexpr int ROWS = C <= 4 ? 32 : 16, PARTS = 32 / ROWS, READS = ROWS / R;
  static constexpr int PART_BYTES = ROWS * C * 32;
};

// Which 16-byte chunks the operands of the concatenated GEMM take.  Along K: [x1 | x2 | x1 | norm] against [y1 | y1 | y2 | norm], C
// chunks each and one (C even: two, the second zero) for the norm; one MMA takes two neighbours of that sequence, whose distance
// in shared memory a descriptor states.  So x1 is stored once, and y1 where no pair starts in one copy of it and ends in the next.
template <int C>
struct Operands {
  static constexpr int steps = (3 * C + 2) / 2;
  static constexpr int zero = C % 2 == 0 ? 1 : 0;  // a zero chunk behind the norm chunk
  static constexpr int a_chunks = 2 * C + 1 + zero, b_chunks = C % 2 == 0 ? 2 * C + 2 : 3 * C + 1;
  static constexpr int a_norm = 2 * C, b_norm = C % 2 == 0 ? 2 * C : 3 * C, b_low = C % 2 == 0 ? C : 2 * C;  // where norm and y2 start
  static constexpr int a(int q) { return q < 2 * C ? q : q < 3 * C ? q - 2 * C : q - C; }
  static constexpr int b(int q) { return C % 2 != 0 || q < C ? q : q - C; }
};

// What shared memory holds: A tiles in the ring, and parts of rows in flight per producer warp: 32 to 64 KB per SM (the DRAM's latency
// holds about 35 at its full rate).  Tiles go to two producer groups and two MMA threads in turn, so with an odd number of stages a stage
// changes hands; its barriers, of which each side has to see every phase, are then those of t % (2 * stages).
template <int C, int NB>
struct Ring {
  static constexpr int stages = C >= 7 && NB == 8 ? 3 : 4, turns = stages % 2 ? 2 * stages : stages;
  static constexpr int slots = C == 1 ? 8 : C == 2 ? 4 : C >= 7 ? 1 : 2;
  static constexpr size_t bytes = (size_t)Operands<C>::b_chunks * (NB * 512 + Lanes<C>::PAD) + (size_t)Operands<C>::a_chunks * stages * (kTileM * 16 + Lanes<C>::PAD) +
                                  (size_t)kProducerWarps * slots * Lanes<C>::PART_BYTES + kMaxN * 4 + kBoundRing * kTileM * 4 +
                                  8 * (2 * turns + 4 * kEpilogueGroups + 6 + kProducerWarps * slots) + 16 + 4 * kList;
  static_assert(bytes <= 227 * 1024, "shared memory of a CTA");
};

// ---------------------------------------------------------------- points that the tensor cores leave undecided
// Shared memory, behind the assignment, of a list of undecided points (numbered inside the CTA: 128 * tile + row) and of their labels.
// Bytes of what the second half of an assignment, or of a Lloyd iteration, keeps in shared memory beside the centres.
template <int C>
constexpr size_t kListsPlace = 20480 + 1024 * C;
constexpr int kFew = 8;     // points up to which the centres are not staged for them
constexpr int kMany = 400;  // points from which on a thread scores one
struct Scores {
  unsigned long long nearest[kFew];
  uint16_t label[kList];
};

// Labels of the listed points by exact distances, term by term those of kmeans.cu's kernels; called by all threads.
//  * A few points: a warp scores one of them against 32 centres where these lie; the smallest distance, then the smallest index.  (Staging
//    the centres for them took 7 to 28 thousand cycles, and in a fit all other CTAs waited for the few that had such points.)
//  * More: the centres are staged in a_ring, rows padded so that eight lanes touch eight bank groups, and a warp scores a point.
//  * Many, as where rows are zero: a thread scores a point, a centre is read once for 32 of them.
template <int C>
__device__ __noinline__ void score_exactly(const Params& p, const uint32_t* list, int count, Scores* out, unsigned char* a_ring, float* points, bool& staged) {
  constexpr int DP = 8 * C, STRIDE = DP + 4, kWarps = kThreads / 32;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool cosine = p.metric == F2C_COSINE;
  auto point = [&](int w) {
    const int at = (int)list[w];
    return p.x + (((int64_t)blockIdx.x + (int64_t)(at >> 7) * gridDim.x) * kTileM + (at & 127)) * p.d;
  };
  auto distance = [&](float acc, float x_norm, float c_norm) {  // finish_cosine() with the square roots taken before
    const float den = x_norm * c_norm, v = !cosine ? acc : den > 0.0f ? 1.0f - acc / den : 1.0f;
    return v != v ? 1.0f : v;
  };
  if (count <= kFew) {
    if (tid < kFew) out->nearest[tid] = ~0ull;
    for (int e = tid; e < count * DP; e += kThreads) points[e] = e % DP < p.d ? __ldg(point(e / DP) + e % DP) : 0.0f;
    __syncthreads();
    const int blocks = (p.k + 31) / 32;
    for (int w = warp; w < count * blocks; w += kWarps) {
      const int c = w % blocks * 32 + lane;
      const float* xs = points + w / blocks * DP;
      const float* yc = p.y + min(c, p.k - 1) * p.d;
      float acc = 0.0f, xx = 0.0f, cc = 0.0f;
#pragma unroll 1
      for (int b = 0; b < DP; b += 32) {
        constexpr int IN_FLIGHT = C < 4 ? C : 4;
        float y[IN_FLIGHT][8];
#pragma unroll
        for (int q = 0; q < IN_FLIGHT; ++q) load8(yc, b + 8 * q, p.d, p.y_wide, true, y[q]);
#pragma unroll
        for (int q = 0; q < IN_FLIGHT; ++q) {
          if (b + 8 * q >= DP) break;
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const float a = xs[b + 8 * q + e];
            if (cosine) {
              acc = fmaf(a, y[q][e], acc);
              xx = fmaf(a, a, xx);
              cc = fmaf(y[q][e], y[q][e], cc);
            } else {
              const float df = a - y[q][e];
              acc = fmaf(df, df, acc);
            }
          }
        }
      }
      const uint32_t bits = __float_as_uint(distance(acc, sqrtf(xx), sqrtf(cc))), order = bits ^ ((int32_t)bits < 0 ? 0xffffffffu : 0x80000000u);
      if (c < p.k) atomicMin(out->nearest + w / blocks, (unsigned long long)order << 32 | (uint32_t)c);
    }
    __syncthreads();
    if (tid < count) out->label[tid] = (uint16_t)out->nearest[tid];
    __syncthreads();
    return;
  }
  float* yc = reinterpret_cast<float*>(a_ring);
  float* norm = yc + p.k * STRIDE;
  if (!staged) {
#pragma unroll 12
    for (int e = tid; e < p.k * DP; e += kThreads) {  // many reads in flight
      const int c = e / DP, t = e - c * DP;
      yc[c * STRIDE + t] = t < p.d ? __ldcg(p.y + c * p.d + t) : 0.0f;
    }
    __syncthreads();
    for (int c = tid; c < p.k; c += kThreads) {
      float s = 0.0f;
      for (int t = 0; t < DP; ++t) s = fmaf(yc[c * STRIDE + t], yc[c * STRIDE + t], s);
      norm[c] = sqrtf(s);
    }
    __syncthreads();
    staged = true;
  }
  if (count < kMany) {
    float* xs = points + warp * DP;
    for (int w = warp; w < count; w += kWarps) {
      const float* xi = point(w);
      __syncwarp();
      for (int t = lane; t < DP; t += 32) xs[t] = t < p.d ? __ldg(xi + t) : 0.0f;
      __syncwarp();
      float xx = 0.0f, best = INFINITY;
      int best_c = 0x7fffffff;
      if (cosine)
        for (int t = 0; t < DP; ++t) xx = fmaf(xs[t], xs[t], xx);
      const float x_norm = sqrtf(xx);
      for (int c = lane; c < p.k; c += 32) {
        float acc = 0.0f;
#pragma unroll
        for (int t = 0; t < DP; t += 4) {
          const float4 a = *reinterpret_cast<const float4*>(xs + t), b = *reinterpret_cast<const float4*>(yc + c * STRIDE + t);
          if (!cosine) {
            const float d0 = a.x - b.x, d1 = a.y - b.y, d2 = a.z - b.z, d3 = a.w - b.w;
            acc = fmaf(d0, d0, acc); acc = fmaf(d1, d1, acc); acc = fmaf(d2, d2, acc); acc = fmaf(d3, d3, acc);
          } else {
            acc = fmaf(a.x, b.x, acc); acc = fmaf(a.y, b.y, acc); acc = fmaf(a.z, b.z, acc); acc = fmaf(a.w, b.w, acc);
          }
        }
        const float v = distance(acc, x_norm, norm[c]);
        if (v < best) { best = v; best_c = c; }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oc = __shfl_xor_sync(0xffffffffu, best_c, o);
        if (ob < best || (ob == best && oc < best_c)) { best = ob; best_c = oc; }
      }
      if (lane == 0) out->label[w] = (uint16_t)(best_c == 0x7fffffff ? 0 : best_c);
    }
  } else {
    for (int w = tid; w < count; w += kThreads) {
      const float* xi = point(w);
      float xr[DP], xx = 0.0f, best = INFINITY;
      int best_c = 0;
#pragma unroll
      for (int t = 0; t < DP; ++t) {
        xr[t] = t < p.d ? __ldg(xi + t) : 0.0f;
        xx = fmaf(xr[t], xr[t], xx);
      }
      const float x_norm = sqrtf(xx);
#pragma unroll 1
      for (int c = 0; c < p.k; ++c) {
        float acc = 0.0f;
#pragma unroll
        for (int t = 0; t < DP; t += 4) {
          const float4 b = *reinterpret_cast<const float4*>(yc + c * STRIDE + t);
          if (!cosine) {
            const float d0 = xr[t] - b.x, d1 = xr[t + 1] - b.y, d2 = xr[t + 2] - b.z, d3 = xr[t + 3] - b.w;
            acc = fmaf(d0, d0, acc); acc = fmaf(d1, d1, acc); acc = fmaf(d2, d2, acc); acc = fmaf(d3, d3, acc);
          } else {
            acc = fmaf(xr[t], b.x, acc); acc = fmaf(xr[t + 1], b.y, acc); acc = fmaf(xr[t + 2], b.z, acc); acc = fmaf(xr[t + 3], b.w, acc);
          }
        }
        const float v = distance(acc, x_norm, norm[c]);
        if (v < best) { best = v; best_c = c; }
      }
      out->label[w] = (uint16_t)best_c;
    }
  }
  __syncthreads();
}

// What an assignment does with its undecided points: the CTA's list holds the first kList of them; if there are more, or a wait has run out (lost),
// they are found by their labels, -1, and scored as many at a time as there are threads.
template <int C>
__device__ __noinline__ void settle(const Params& p, int turns, bool lost, const uint32_t* open_list, uint32_t* counter, unsigned char* a_ring, unsigned char* rows) {
  Scores* scores = reinterpret_cast<Scores*>(rows);
  uint32_t* list = reinterpret_cast<uint32_t*>(scores + 1);  // [2 * kThreads]
  float* points = reinterpret_cast<float*>(list + 2 * kThreads);
  static_assert(sizeof(Scores) % 16 == 0 && kThreads <= kList && sizeof(Scores) + 8 * kThreads + kThreads / 32 * 8 * C * 4 <= kListsPlace<C>,
                "fits");
  const int tid = threadIdx.x;
  const uint32_t open = *counter;
  bool staged = false;
  auto index_of = [&](uint32_t at) { return ((int64_t)blockIdx.x + (int64_t)(at >> 7) * gridDim.x) * kTileM + (at & 127u); };
  auto score = [&](const uint32_t* which, int count) {
    score_exactly<C>(p, which, count, scores, a_ring, points, staged);
    for (int w = tid; w < count; w += kThreads) p.labels[index_of(which[w])] = scores->label[w];
    __syncthreads();
  };
  uint32_t total = open;
  if (!lost && open <= (uint32_t)kList) {
    if (open == 0u) return;
    score(open_list, (int)open);
  } else {
    total = 0u;
    __syncthreads();
    if (tid == 0) *counter = 0u;
    for (int first = 0; first < turns * kTileM; first += kThreads) {
      __syncthreads();
      const uint32_t at = (uint32_t)(first + tid);
      const int64_t i = index_of(at);
      if (first + tid < turns * kTileM && i < p.n && (lost || __ldcg(p.labels + i) < 0)) list[atomicAdd(counter, 1u)] = at;
      __syncthreads();
      int count = (int)*counter;
      const bool last = first + kThreads >= turns * kTileM;
      for (int from = 0; count >= kThreads || (last && count > 0); from += kThreads, count -= min(count, kThreads)) {
        score(list + from, min(count, kThreads));
        total += (uint32_t)min(count, kThreads);
        if (count < kThreads) break;
        if (count - kThreads < kThreads && !last) {  // the rest moves to the front
          const uint32_t rest = tid < count - kThreads ? list[from + kThreads + tid] : 0u;
          __syncthreads();
          if (tid < count - kThreads) list[tid] = rest;
          if (tid == 0) *counter = (uint32_t)(count - kThreads);
          break;
        }
      }
    }
  }
  if (tid == 0) atomicAdd(p.undecided, (int32_t)total);
}

// ---------------------------------------------------------------- the second half of a Lloyd iteration
// Behind the labels of this CTA's points: those that are still undecided, the clusters' sums, and, all CTAs together, the new centres.
// Returns whether the fit has converged.  `number`: of this iteration; a_ring, rows: shared memory that the assignment has done with; `instead`: if
// not null, a wait of this CTA has run out and this is where nothing may still arrive.
//  * The sums are integers and exact, so they are kept from iteration to iteration, and only points that have changed their cluster are
//    taken off one sum and added to another.  From the second iteration on these are few: an iteration of 149,000 x 32 that added up
//    everything anew took 40 us, 35 with this (a 64-bit reduction per cluster, column and CTA; L2 does about a hundred of them a cycle).
//  * A CTA sorts its changes by cluster (a counting sort of up to 1024 points' at a time), and 8, 16 or 32 lanes walk a part of them, hold
//    their columns' sums in registers and add them to the global ones where the cluster changes.
template <int C>
__device__ __noinline__ bool end_of_iteration(const FitParams& p, int number, int turns, unsigned char* instead, unsigned char* a_ring, unsigned char* rows) {
  if (instead != nullptr) { rows = instead; a_ring = instead + kListsPlace<C>; }
  namespace cg = cooperative_groups;
  constexpr int DP = 8 * C, kWarps = kThreads / 32;
  constexpr int kChunkTiles = 8, kChunk = kChunkTiles * kTileM, kShares = (kChunk / 32 + kWarps - 1) / kWarps;
  constexpr int W = C == 1 ? 8 : C == 2 ? 16 : 32, CPL = C > 4 ? 2 : 1;  // lanes per point, columns per lane
  uint2* sorted = reinterpret_cast<uint2*>(rows);  // cluster and, where it lost the point, kLost; where the point's row starts behind the chunk's first
  constexpr uint32_t kLost = 1u << 16;
  uint32_t* hist = reinterpret_cast<uint32_t*>(sorted + 2 * kChunk);
  uint32_t* start = hist + kMaxN;  // [257]
  int32_t* gained = reinterpret_cast<int32_t*>(start + kMaxN + 4);
  float* point = reinterpret_cast<float*>(gained + kMaxN);  // one per warp
  double* part = reinterpret_cast<double*>(point + kWarps * DP);
  static_assert((4 * kChunk + 3 * kMaxN + 4 + kWarps * DP + 2 * kWarps) * 4 <= kListsPlace<C>, "fits");
  static_assert(kMaxN * (DP + 5) * 4 <= Ring<C, 8>::stages * Operands<C>::a_chunks * (kTileM * 16 + Lanes<C>::PAD), "fits the A ring's place");
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool all = instead != nullptr || *(volatile const int32_t*)p.error != 0;  // a wait has run out, here or in another CTA: score every point exactly
  auto index_of = [&](int t, int row) { return ((int64_t)blockIdx.x + (int64_t)t * gridDim.x) * kTileM + row; };
  bool staged = false;
  const int bits = fraction_bits(p.n);
  // A value's fixed-point integer, round(x * 2^(bits - e)), in two parts with fp32 alone: hi = round(x * 2^(21 - e)), lo = round of what is left
  // times 2^(bits - 21), each in the low bits of a float to which 1.5 * 2^23 was added.  All steps but the last rounding are exact, and sums of
  // the floats' bit patterns, of a walker's 94 values at most, fit 32 bits once the pattern of 1.5 * 2^23 is taken off.  (Conversions through
  // double: 1.7 values a cycle and SM, 19,000 of an iteration's 90,000 cycles at 147,000 x 32.)
  constexpr float kMagic = 12582912.0f;
  constexpr uint32_t kMagicBits = 0x4B400000u;
  static_assert((2 * kChunk + kWarps - 1) / kWarps < (1 << 9), "hi: up to 2^21 each");
  const float low_unit = (float)(1 << (bits - 21));
  float up[CPL], rest[CPL];  // 2^(21 - e), as two factors that fp32 holds
#pragma unroll
  for (int q = 0; q < CPL; ++q) {
    const int j = lane % W + 32 * q;
    const int to = 21 - (j < p.d ? exponent(__ldg(p.maxima + j)) : 0);
    up[q] = power2f(min(to, 100));
    rest[q] = power2f(to - min(to, 100));
  }

  for (int t0 = 0; t0 < turns; t0 += kChunkTiles) {
    const int shares = 4 * min(kChunkTiles, turns - t0);  // of 32 points
    for (int c = tid; c < kMaxN; c += kThreads) { hist[c] = 0u; gained[c] = 0; }
    if (tid == 0) start[0] = 0u;  // length of the list of open points
    uint32_t label[kShares], before[kShares], rank[kShares], rank_before[kShares];
    bool open = false;
#pragma unroll
    for (int s = 0; s < kShares; ++s) {
      const int g = warp + kWarps * s;
      const int64_t i = index_of(t0 + (g >> 2), (g & 3) * 32 + lane);
      label[s] = g < shares && i < p.n ? __ldcg(p.labels16 + i) : kUndecided + 1u;
      open |= label[s] == kUndecided;
    }
    if (__syncthreads_or(open || all)) {
      uint32_t* list = reinterpret_cast<uint32_t*>(rows);
      Scores* scores = reinterpret_cast<Scores*>(rows + kChunk * 4);
      static_assert(kChunk <= kList && kChunk * 4 + sizeof(Scores) <= 2 * kChunk * sizeof(uint2), "in the place of the sorted changes");
      int entry[kShares];
#pragma unroll
      for (int s = 0; s < kShares; ++s) {
        entry[s] = -1;
        if (label[s] == kUndecided || (all && label[s] < kUndecided)) {
          entry[s] = (int)atomicAdd(start, 1u);
          list[entry[s]] = (uint32_t)(t0 * kTileM + (warp + kWarps * s) * 32 + lane);
        }
      }
      __syncthreads();
      score_exactly<C>(p, list, (int)start[0], scores, a_ring, point, staged);
#pragma unroll
      for (int s = 0; s < kShares; ++s)
        if (entry[s] >= 0) label[s] = scores->label[entry[s]];
      __syncthreads();  // the sorted changes take their place
    }
    bool any = false;
#pragma unroll
    for (int s = 0; s < kShares; ++s) {
      const int g = warp + kWarps * s;
      const int64_t i = index_of(t0 + (g >> 2), (g & 3) * 32 + lane);
      before[s] = label[s] < kUndecided ? __ldcg(p.summed16 + i) : label[s];
      if (label[s] == before[s]) continue;
      any = true;
      __stcg(p.summed16 + i, (uint16_t)label[s]);
      rank[s] = atomicAdd(hist + label[s], 1u);
      atomicAdd(gained + label[s], 1);
      if (before[s] != kUndecided) {
        rank_before[s] = atomicAdd(hist + before[s], 1u);
        atomicAdd(gained + before[s], -1);
      }
    }
    if (!__syncthreads_or(any)) continue;
    if (warp == 0) {
      uint32_t own[kMaxN / 32], sum = 0u;
#pragma unroll
      for (int q = 0; q < kMaxN / 32; ++q) { own[q] = sum; sum += hist[lane * (kMaxN / 32) + q]; }
      uint32_t before = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, before, o);
        if (lane >= o) before += v;
      }
      before -= sum;
#pragma unroll
      for (int q = 0; q < kMaxN / 32; ++q) start[lane * (kMaxN / 32) + q] = before + own[q];
      if (lane == 31) start[kMaxN] = before + sum;
    }
    __syncthreads();
#pragma unroll
    for (int s = 0; s < kShares; ++s)
      if (label[s] != before[s]) {
        const int g = warp + kWarps * s;
        const uint32_t row = (uint32_t)(((int64_t)(g >> 2) * gridDim.x * kTileM + (g & 3) * 32 + lane) * p.d);
        sorted[start[label[s]] + rank[s]] = make_uint2(label[s], row);
        if (before[s] != kUndecided) sorted[start[before[s]] + rank_before[s]] = make_uint2(before[s] | kLost, row);
      }
    for (int c = tid; c < p.k; c += kThreads)
      if (gained[c] != 0) atomicAdd(p.counts + c, (uint32_t)gained[c]);
    __syncthreads();
    const int points = (int)start[kMaxN], walkers = kWarps * (32 / W);
    const int run = (points + walkers - 1) / walkers, walker = warp * (32 / W) + lane / W;
    const int lo = min(walker * run, points), hi = min(lo + run, points);
    // Four changes a turn, the next four's rows on their way: a short loop, since warps that run through long unrolled code wait for instructions.
    constexpr int U = 4;
    const float* first = p.x + index_of(t0, 0) * p.d + lane % W;
    uint32_t next_label[U];
    float next_v[U][CPL];
    auto look = [&](int s) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint2 entry = sorted[max(min(s + u, hi - 1), 0)];
        next_label[u] = entry.x;
#pragma unroll
        for (int q = 0; q < CPL; ++q) next_v[u][q] = s + u < hi && lane % W + 32 * q < p.d ? __ldg(first + entry.y + 32 * q) : 0.0f;
      }
    };
    look(lo);
    uint32_t sum_hi[CPL] = {}, sum_lo[CPL] = {};
#pragma unroll 1
    for (int s = lo; s < hi; s += U) {
      uint32_t label[U];
      float v[U][CPL];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        label[u] = next_label[u];
#pragma unroll
        for (int q = 0; q < CPL; ++q) v[u][q] = next_v[u][q];
      }
      look(s + U);
#pragma unroll
      for (int u = 0; u < U; ++u) {
#pragma unroll
        for (int q = 0; q < CPL; ++q) {
          const float t = v[u][q] * up[q] * ((label[u] & kLost) != 0u ? -rest[q] : rest[q]), hi = t + kMagic;
          sum_hi[q] += __float_as_uint(hi) - kMagicBits;
          sum_lo[q] += __float_as_uint(fmaf(t - (hi - kMagic), low_unit, kMagic)) - kMagicBits;
        }
        const uint32_t then = u + 1 < U ? label[u + 1 < U ? u + 1 : 0] : next_label[0];
        if (s + u + 1 >= hi || (uint16_t)then != (uint16_t)label[u]) {  // the last point of its cluster in this run
          if (s + u < hi) {
#pragma unroll
            for (int q = 0; q < CPL; ++q)
              if (lane % W + 32 * q < p.d)
                atomicAdd(reinterpret_cast<unsigned long long*>(p.sums) + (label[u] & 0xffffu) * p.d + lane % W + 32 * q,
                          (unsigned long long)((long long)(int32_t)sum_hi[q] * (1ll << (bits - 21)) + (int32_t)sum_lo[q]));
          }
#pragma unroll
          for (int q = 0; q < CPL; ++q) sum_hi[q] = sum_lo[q] = 0u;
        }
      }
    }
    __syncthreads();  // the next chunk takes the lists' place
  }
  cg::this_grid().sync();

  // ---- centres <- sums / counts; clusters without points keep theirs ----
  const int kd = p.k * p.d, share = (kd + (int)gridDim.x - 1) / (int)gridDim.x;
  double shift = 0.0;
  for (int i = blockIdx.x * share + tid; i < min(((int)blockIdx.x + 1) * share, kd); i += kThreads) {
    const int c = i / p.d, j = i - c * p.d;
    const uint32_t cnt = __ldcg(p.counts + c);
    if (cnt != 0u) {
      const float next = (float)((double)__ldcg(p.sums + i) * power2(exponent(__ldg(p.maxima + j)) - bits)) / (float)cnt;
      const float diff = next - __ldcg(p.centers + i);
      __stcg(p.centers + i, next);
      shift += (double)(diff * diff);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) shift += __shfl_xor_sync(0xffffffffu, shift, o);
  if (lane == 0) part[warp] = shift;
  __syncthreads();
  if (tid == 0) {
    double total = 0.0;
    for (int w = 0; w < kWarps; ++w) total += part[w];
    __stcg(p.shifts + blockIdx.x, total);
    if (blockIdx.x == 0) {
      // after a wait that ran out the labels are the exact scorer's, so the iteration counts and the next one starts afresh
      const int32_t error = *(volatile const int32_t*)p.error;
      if (error != 0) { p.state->assign_error = error; *p.error = 0; }
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // copies and MMAs have the shared memory next
  cg::this_grid().sync();
  // every warp of the grid adds the same numbers in the same order
  double total = 0.0;
  for (int b0 = 0; b0 < (int)gridDim.x; b0 += 256) {
    double from[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) from[q] = b0 + 32 * q + lane < (int)gridDim.x ? __ldcg(p.shifts + b0 + 32 * q + lane) : 0.0;
#pragma unroll
    for (int q = 0; q < 8; ++q) total += from[q];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
  const bool converged = (double)(float)total <= p.tol;
  if (blockIdx.x == 0 && tid == 0) {
    p.state->shift = total;
    p.state->iterations = number + 1;
    if (converged) p.state->done = 1;
  }
  return converged;
}

// Shared memory: [B tile][A ring][rows in flight][norms 256 floats][bounds kBoundRing x 128 floats][mbarriers, tmem slot, count and list of undecided points]
// C: chunks of eight dimensions of a row (1 to 8); NB: blocks of 32 columns (4: up to 128 centres, 8: up to 256).
// NO_WAITS: every wait runs out at once, for tests of what follows.
// P = Params: one assignment.  FitParams: Lloyd iterations, by CTAs that are all resident (kmeans_fit_tc.cu); tiles are then counted on
// from iteration to iteration, so that the barriers' phases go on.
template <int C, int NB, bool NO_WAITS, typename P>
__device__ __forceinline__ void run(const P& p) {
  constexpr bool FIT = std::is_same<P, FitParams>::value;
  using L = Lanes<C>;
  using O = Operands<C>;
  using Q = Ring<C, NB>;
  constexpr int N = 32 * NB;
  constexpr uint32_t lbo_b = N * 16 + L::PAD, lbo_a = kTileM * 16 + L::PAD, sbo = 128;
  extern __shared__ __align__(128) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr uint32_t a_bytes = O::a_chunks * lbo_a;
  unsigned char* b_tile = smem;
  unsigned char* a_ring = smem + O::b_chunks * lbo_b;
  unsigned char* rows = a_ring + Q::stages * a_bytes;
  float* norms = reinterpret_cast<float*>(rows + kProducerWarps * Q::slots * L::PART_BYTES);
  float* bounds = norms + kMaxN;
  uint64_t* mbars = reinterpret_cast<uint64_t*>(bounds + kBoundRing * kTileM);
  // a_full[turns], a_free[turns], acc_full[kFull][HALVES], acc_free[4], drained[2], row_full[producer warp][slots].  A wait names the parity of a
  // phase only, so whoever waits has to have seen the phase before, and the next one must not end before it has looked.  That an accumulator
  // has become full is therefore a matter of its tile, t % kFull, where t + kFull has the same accumulator and the same epilogue group: its
  // MMAs wait for those of all tiles between that have this accumulator, t among them, to have been read.
  constexpr int HALVES = NB / 4, kFull = 4 * kEpilogueGroups / HALVES;
  const uint32_t a_full = smem_u32(mbars), a_free = a_full + 8 * Q::turns, acc_full = a_free + 8 * Q::turns, acc_free = acc_full + 8 * kFull * HALVES,
                 drained = acc_free + 32, row_full = drained + 16;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mbars + 2 * Q::turns + 6 + kFull * HALVES + kProducerWarps * Q::slots);
  uint32_t* open_count = tmem_slot + 1;  // undecided points of this CTA, the first kList of them in the list
  uint32_t* open_list = tmem_slot + 4;

  const int64_t n_tiles = (p.n + kTileM - 1) / kTileM;
  const int turns = (int)((n_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x);  // tiles of this CTA: blockIdx.x + t * gridDim.x
  Waiter wait{p.error, false};

  const int group = warp >= kEpilogueWarps ? (warp - kEpilogueWarps) >> 2 : warp >> 2;
  const bool l2 = p.metric == F2C_L2;
  const int row_l = lane / L::CL, chunk_l = lane % L::CL;
  const bool producer = warp >= kEpilogueWarps && warp < kMmaWarp;
  const int own = producer ? warp - kEpilogueWarps : 0;
  unsigned char* own_rows = rows + own * (Q::slots * L::PART_BYTES);
  const uint32_t own_full = row_full + (uint32_t)own * (8 * Q::slots);
  // rows of part q of this warp's share of tile t: how many there are, and whether one bulk copy fetches them
  auto part_base = [&](int t, int q) { return ((int64_t)blockIdx.x + (int64_t)t * gridDim.x) * kTileM + (warp & 3) * 32 + q * L::ROWS; };
  auto part_bulk = [&](int64_t base) { return p.x_aligned && base + L::ROWS <= p.n; };
  uint32_t fetched = 0;  // lane 0: bit s, slot s has had a bulk copy; bit 8 + s, the parity of its last one's phase
  auto fetch = [&](int t, int q, int slot) {
    if (t < turns && !wait.gave_up) {
      const int64_t base = part_base(t, q);
      const float* src = p.x + base * p.d;
      const uint32_t dst = smem_u32(own_rows + slot * L::PART_BYTES);
      if (part_bulk(base)) {
        if (lane == 0) {
          fetched = (fetched ^ (((fetched >> slot) & 1u) << (8 + slot))) | (1u << slot);
          const uint32_t bytes = (uint32_t)(L::ROWS * 4 * p.d), full = own_full + 8u * slot;
          asm volatile("{\n\t.reg .b64 s;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 s, [%0], %1;\n\t}" ::"r"(full), "r"(bytes) : "memory");
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(full)
                       : "memory");
        }
      } else {  // the last rows of x, or an x that starts off a 16-byte boundary
        const int some = (int)max((int64_t)0, min((int64_t)L::ROWS, p.n - base)) * p.d;
        for (int e = lane; e < some; e += 32) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 4u * e), "l"(src + e) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  // ---- one-time setup: mbarriers, TMEM (all 512 columns), centre tile ----
  if (threadIdx.x == 32 * kMmaWarp) {
    *open_count = 0u;
    for (int s = 0; s < Q::turns; ++s) { mbar_init(a_full + 8 * s, 4); mbar_init(a_free + 8 * s, 1); }
    for (int u = 0; u < kFull * HALVES; ++u) mbar_init(acc_full + 8 * u, 1);
    for (int u = 0; u < 4; ++u) mbar_init(acc_free + 8 * u, 4);
    for (int g = 0; g < 2; ++g) mbar_init(drained + 8 * g, 1);
    for (int u = 0; u < kProducerWarps * Q::slots; ++u) mbar_init(row_full + 8 * u, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  constexpr int kStagers = 16;  // warps that stage the centres; the last of the producers prepare the A ring
  constexpr int STEPS = (N / kStagers + L::R - 1) / L::R;  // reads that make a warp's share of the centres
  static_assert(N / kStagers % L::R == 0 || STEPS == 1, "shares of whole reads");
  const int c0 = warp * (STEPS * L::R);  // C = 1: the first N / 32 warps have 32 centres each
  constexpr bool KEEP = STEPS <= 4;  // in registers between the two passes; more than 32 dimensions are read twice
  float yv[KEEP ? STEPS : 1][8];
  auto load_centres = [&](int s, float (&v)[8]) {
    const int c = c0 + s * L::R + row_l;
    load8(p.y + (int64_t)c * p.d, 8 * chunk_l, p.d, p.y_wide, c < p.k, v);
  };
  int iterations = 1, done_before = 0;
  if constexpr (FIT) { iterations = p.iterations; done_before = p.state->iterations; }
  uint32_t phases = 0;  // bit s: parity of the phase that slot s's next copy completes
  int unit = 0;         // parts that this producer warp has taken
  bool lost = false;    // a wait of this CTA has run out: from then on the exact scorer alone
  for (int it = 0; it < iterations; ++it) {
    const int base = it * turns;  // the first tile of this iteration
    if (!lost) {
      if (producer) {  // the first rows, on their way while the centres are staged
        const int first = (group ^ base) & 1;
#pragma unroll
        for (int u = 0; u < Q::slots; ++u) fetch(first + 2 * (u / L::PARTS), u % L::PARTS, (unit + u) % Q::slots);
      }
      if (warp < kStagers) {
        if constexpr (KEEP) {
#pragma unroll
          for (int s = 0; s < STEPS; ++s) load_centres(s, yv[s]);
        }
#pragma unroll
        for (int s = 0; s < STEPS; ++s) {
          float (&v)[8] = yv[KEEP ? s : 0];
          if constexpr (!KEEP) load_centres(s, v);
          float nrm = 0.0f;
#pragma unroll
          for (int e = 0; e < 8; ++e) nrm = fmaf(v[e], v[e], nrm);
#pragma unroll
          for (int o = 1; o < L::CL; o <<= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
          if (chunk_l == 0 && c0 + s * L::R + row_l < kMaxN) norms[c0 + s * L::R + row_l] = nrm;
        }
      }
      __syncthreads();
      // largest centre norm (scale and tolerance of the L2 score); a centre that is not finite or (cosine; squared L2: all of them) so short that its
      // squared length has lost bits sends every point to the exact scorer
      float cmax = 0.0f, poison = 0.0f;
#pragma unroll
      for (int c = lane; c < N; c += 32) {
        cmax = fmaxf(cmax, norms[c]);
        poison = fmaf(norms[c], !l2 && norms[c] > 0.0f && norms[c] < kTiny ? INFINITY : 0.0f, poison);  // inf, NaN -> NaN
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        cmax = fmaxf(cmax, __shfl_xor_sync(0xffffffffu, cmax, o));
        poison += __shfl_xor_sync(0xffffffffu, poison, o);
      }
      const bool bad_centres = !(poison == 0.0f) || (l2 && cmax < kTiny);
      const int e_y = l2 ? max(-120, min(120, exponent_above(sqrtf(cmax)))) : 0;  // squared L2: everything times 2^-e_y
      const float scale_y = power2f(-e_y);
      cmax = l2 ? sqrtf(cmax) * scale_y : 1.0f;
      if (warp < kStagers) {
#pragma unroll
        for (int s = 0; s < STEPS; ++s) {
          const int c = c0 + s * L::R + row_l;
          float (&v)[8] = yv[KEEP ? s : 0];
          if constexpr (!KEEP) load_centres(s, v);
          if (c < N) {
            const float nrm = norms[c];
            // cosine: rows of unit length (zero rows stay zero)
            const float f = l2 ? scale_y : (nrm > 0.0f ? 1.0f / sqrtf(nrm) : 0.0f);
            float own_sq = 0.0f;  // squared length of the scaled row, which the norm term takes: |y|^2 itself may overflow
#pragma unroll
            for (int e = 0; e < 8; ++e) { v[e] *= f; own_sq = fmaf(v[e], v[e], own_sq); }
            if (C == L::CL || chunk_l < C) {
              uint4 c1, c2;
              split8(v, c1, c2);
              *reinterpret_cast<uint4*>(b_tile + (size_t)chunk_l * lbo_b + c * 16) = c1;
              if (O::b_low > C) *reinterpret_cast<uint4*>(b_tile + (size_t)(C + chunk_l) * lbo_b + c * 16) = c1;
              *reinterpret_cast<uint4*>(b_tile + (size_t)(O::b_low + chunk_l) * lbo_b + c * 16) = c2;
            }
#pragma unroll
            for (int o = 1; o < L::CL; o <<= 1) own_sq += __shfl_xor_sync(0xffffffffu, own_sq, o);
            if (chunk_l == 0) {
              const float h = l2 && c < p.k ? -0.5f * own_sq : 0.0f;
              const __half h1 = __float2half_rn(h), h2 = __float2half_rn(h - __half2float(h1));
              const __half h3 = __float2half_rn(h - __half2float(h1) - __half2float(h2));
              const __half never = __float2half_rn(c < p.k ? 0.0f : -65504.0f);
              *reinterpret_cast<uint4*>(b_tile + (size_t)O::b_norm * lbo_b + c * 16) =
                  make_uint4((uint32_t)__half_as_ushort(h1) | ((uint32_t)__half_as_ushort(h2) << 16),
                             (uint32_t)__half_as_ushort(h3) | ((uint32_t)__half_as_ushort(never) << 16), 0u, 0u);
              if (O::zero) *reinterpret_cast<uint4*>(b_tile + (size_t)(O::b_norm + 1) * lbo_b + c * 16) = make_uint4(0u, 0u, 0u, 0u);
            }
          }
        }
      } else if (warp < kMmaWarp) {
        // what the norm chunk holds in every A tile (cosine: a one against the padding's number), and the zeros behind it
        for (int i = threadIdx.x - 32 * kStagers; i < Q::stages * kTileM; i += 32 * (kMmaWarp - kStagers)) {
          unsigned char* at = a_ring + (size_t)(i / kTileM) * a_bytes + (size_t)O::a_norm * lbo_a + i % kTileM * 16;
          *reinterpret_cast<uint4*>(at) = make_uint4(0u, 0x3C000000u, 0u, 0u);
          if (O::zero) *reinterpret_cast<uint4*>(at + lbo_a) = make_uint4(0u, 0u, 0u, 0u);
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncthreads();
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t tmem_base = *tmem_slot;
      // Tile t's columns 128 h .. 128 h + 127 are in accumulator (t, h) of four.
      auto accumulator = [](int t, int h) { return 2 * (t & 1) + (NB == 8 ? h : (t >> 1) & 1); };

      if constexpr (NO_WAITS) {  // the first rows are on their way
        wait.gave_up = true;
        if (threadIdx.x == 0) atomicExch(p.error, 1);
      } else if (producer) {
        const float eps = 2.0f * cmax * (bad_centres ? INFINITY : p.eps);  // what two scores may be off by together, per |x|
        for (int t = base + ((group ^ base) & 1); t < base + turns; t += 2) {
          unsigned char* a_tile = a_ring + (size_t)(t % Q::stages) * a_bytes;
          if (t >= Q::stages) wait(a_free + 8 * ((t - Q::stages) % Q::turns), (uint32_t)((t - Q::stages) / Q::turns) & 1u, 1 + t);
#pragma unroll
          for (int q = 0; q < L::PARTS; ++q, ++unit) {
            const int slot = unit % Q::slots;
            asm volatile("cp.async.wait_group %0;" ::"n"(Q::slots - 1) : "memory");
            if (part_bulk(part_base(t - base, q))) {
              wait(own_full + 8 * slot, (phases >> slot) & 1u, 1 + t);
              phases ^= 1u << slot;
            }
            __syncwarp();
            // The reads go through every step side by side: their chains of dependent instructions are what a lone warp waits for.
            float v[L::READS][8], top[L::READS], sum[L::READS], factor[L::READS];
#pragma unroll
            for (int b = 0; b < L::READS; ++b) {
              const float* row = reinterpret_cast<const float*>(own_rows + slot * L::PART_BYTES) + (b * L::R + row_l) * p.d + 8 * chunk_l;
              if (p.x_wide) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                  float4 w = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                  if (8 * chunk_l + 4 * h < p.d) w = *reinterpret_cast<const float4*>(row + 4 * h);
                  v[b][4 * h] = w.x; v[b][4 * h + 1] = w.y; v[b][4 * h + 2] = w.z; v[b][4 * h + 3] = w.w;
                }
              } else {
#pragma unroll
                for (int e = 0; e < 8; ++e) v[b][e] = 8 * chunk_l + e < p.d ? row[e] : 0.0f;
              }
            }
            float any = 0.0f;
#pragma unroll
            for (int b = 0; b < L::READS; ++b) {
              top[b] = max3(max3(fabsf(v[b][0]), fabsf(v[b][1]), fabsf(v[b][2])), max3(fabsf(v[b][3]), fabsf(v[b][4]), fabsf(v[b][5])),
                            fmaxf(fabsf(v[b][6]), fabsf(v[b][7])));
              any = fmaxf(any, top[b]);
            }
            // The slot's next copy may start when all lanes' reads have arrived, not merely been issued: every lane's vote needs what it has read.
            // (A barrier of the warp in its place let rows be overwritten before they were read.  A proxy fence beside the vote adds nothing to that
            // and takes 16 of 178 us of 2,449,029 x 32.)
            if (__all_sync(0xffffffffu, arrived(any, p.never))) fetch(t - base + 2 * ((q + Q::slots) / L::PARTS), (q + Q::slots) % L::PARTS, slot);
            if (l2) {
#pragma unroll
              for (int b = 0; b < L::READS; ++b) {
                top[b] *= scale_y;
#pragma unroll
                for (int e = 0; e < 8; ++e) v[b][e] *= scale_y;
              }
            }
#pragma unroll
            for (int b = 0; b < L::READS; ++b) {
#pragma unroll
              for (int o = 1; o < L::CL; o <<= 1) top[b] = fmaxf(top[b], __shfl_xor_sync(0xffffffffu, top[b], o));
              // |v| < 2^ex.  Squared L2: among the centres the factor stays that of the centres, so that the norm term is not scaled up
              const int biased = min(max(__float_as_int(top[b]) & 0x7f800000, l2 ? 126 << 23 : 0), 252 << 23);
              factor[b] = __int_as_float((253 << 23) - biased);  // 2^-ex, ex = biased - 126
            }
#pragma unroll
            for (int b = 0; b < L::READS; ++b) {
              unsigned char* at = a_tile + (size_t)chunk_l * lbo_a + ((warp & 3) * 32 + q * L::ROWS + b * L::R + row_l) * 16;
              float even = 0.0f, odd = 0.0f;
#pragma unroll
              for (int e = 0; e < 8; e += 2) {
                v[b][e] *= factor[b]; v[b][e + 1] *= factor[b];
                even = fmaf(v[b][e], v[b][e], even); odd = fmaf(v[b][e + 1], v[b][e + 1], odd);
              }
              sum[b] = even + odd;
              uint4 c1, c2;
              split8(v[b], c1, c2);
              if (C == L::CL || chunk_l < C) {
                *reinterpret_cast<uint4*>(at) = c1;
                *reinterpret_cast<uint4*>(at + C * lbo_a) = c2;
              }
            }
#pragma unroll
            for (int b = 0; b < L::READS; ++b)
#pragma unroll
              for (int o = 1; o < L::CL; o <<= 1) sum[b] += __shfl_xor_sync(0xffffffffu, sum[b], o);
            // one lane per row: its error bound, and (squared L2) its part of the norm term: powers of two against the pieces of -|y|^2 / 2 (0 for a
            // point so far out that its own is no f16: the term is below the bound there), a one against the padding's
            float own_sum = sum[0], own_factor = factor[0];
#pragma unroll
            for (int b = 1; b < L::READS; ++b)
              if (chunk_l == b) { own_sum = sum[b]; own_factor = factor[b]; }
            const int row = (warp & 3) * 32 + q * L::ROWS + chunk_l * L::R + row_l;
            const float floor = 2.0f * cmax * (l2 ? fmaxf(0x1p-19f * own_factor, 0x1p-126f) : 0x1p-21f);  // f16 at its lower end, and the norm term
            const float unscale = __int_as_float((254 << 23) - __float_as_int(own_factor)) * power2f(e_y);  // 1 / all that x was multiplied with
            // INFINITY for NaN, for a point whose |x|^2 is more than fp32 holds, and, cosine, for one whose values are all below 2^-51, as kTiny is for
            // centres (the exact scorer may take 0 for its length, all distances are 1 then): the exact scorer's distance says so
            // (-1 for a row of zeros under the cosine metric: all its distances are 1, its label is 0).  (The length in the factor's place: 175 us
            // instead of 162 for 2,449,029 x 32.)
            const float bound = !l2 && own_factor > 0x1p50f ? (own_sum == 0.0f ? -1.0f : INFINITY) : own_sum * unscale * unscale < INFINITY ? fminf(fmaf(eps, sqrt_approx(own_sum), floor), INFINITY) : INFINITY;
            if (chunk_l < L::READS) {
              bounds[(t & (kBoundRing - 1)) * kTileM + row] = bound;
              if (l2) {
                const uint32_t one = (uint32_t)__half_as_ushort(__float2half_rn(own_factor));
                *reinterpret_cast<uint4*>(a_tile + (size_t)O::a_norm * lbo_a + row * 16) = make_uint4(one | (one << 16), one | 0x3C000000u, 0u, 0u);
              }
            }
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(a_full + 8 * (t % Q::turns));
        }
      } else if (warp >= kMmaWarp) {
        // One thread per pair of accumulators, with nothing but constants to add: its instructions follow one another at their full latency (one
        // thread for both, descriptors made in the loop: 740 cycles a tile, more than the epilogue takes; a thread for each of the four: the
        // same at 8 dimensions and 24 us slower at 2,449,029 x 32, whose MMAs then get in each other's way).
        if (lane == 0) {
          // instruction descriptor: fp32 accumulate; A and B f16 (0); 128 columns; M / 16
          constexpr uint32_t idesc = (1u << 4) | ((uint32_t)(128 >> 3) << 17) | ((uint32_t)(kTileM >> 4) << 24);
          const int g = warp - kMmaWarp;
          const uint64_t b_base = make_desc(smem_u32(b_tile), 0, sbo);
          bool on = true;
          for (int t = base + ((g ^ base) & 1); t < base + turns && on; t += 2) {
            const uint64_t a_base = make_desc(smem_u32(a_ring) + (uint32_t)(t % Q::stages) * a_bytes, 0, sbo);
            on = wait(a_full + 8 * (t % Q::turns), (uint32_t)(t / Q::turns) & 1u, 1 + t);
#pragma unroll
            for (int h = 0; h < HALVES; ++h) {  // the epilogue reads one half of the columns while the other is made
              const int a = accumulator(t, h);
              on = on && wait(acc_free + 8 * a, ((uint32_t)(t >> (NB == 8 ? 1 : 2)) & 1u) ^ 1u, 1 + t);
              if (!on) break;
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
              for (int s = 0; s < O::steps; ++s) {  // one MMA consumes 16 f16 = two 16-byte chunks of K
                constexpr auto part = [](int first, int second, uint32_t lbo) { return (uint64_t)((uint32_t)first * lbo >> 4) | (uint64_t)((uint32_t)(second - first) * lbo >> 4) << 16; };
                mma_f16(tmem_base + (uint32_t)a * 128u, a_base + part(O::a(2 * s), O::a(2 * s + 1), lbo_a),
                        b_base + part(O::b(2 * s), O::b(2 * s + 1), lbo_b) + (uint64_t)(h * 128), idesc, s > 0 ? 1u : 0u);
              }
              mma_commit(acc_full + 8 * (HALVES * (t % kFull) + h));
            }
            if (on) mma_commit(a_free + 8 * (t % Q::turns));
          }
        }
        __syncwarp();
      } else {
        // ---- epilogue: TMEM lane pt = point; its thread scans all centres ----
        // Maxima only, one three-operand max per score: of the 16-column groups (row_max) and of the columns with the same number in
        // their group (col_max).  Scores within the bound of the best lie in the crossings of the groups and columns whose maximum does,
        // so the best centre is decided exactly when that is one group and one column - at the crossing.  (A running best, second
        // best and index took five compare instructions per score, which issue at half rate.)
        const int pt = (warp & 3) * 32 + lane;
        const uint32_t lane_addr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
        constexpr int kGroups = 2 * NB;
        for (int t = base + (group + kEpilogueGroups - base % kEpilogueGroups) % kEpilogueGroups; t < base + turns; t += kEpilogueGroups) {
          const uint32_t turn = (uint32_t)t / kEpilogueGroups;  // which of this group's tiles
          float row_max[kGroups], col_max[16], bound = 0.0f;
          uint32_t ra[16], rb[16];  // two 16-column loads alternate: one is consumed while the other is in flight
          auto group_max = [&](const uint32_t (&r)[16]) {
            auto f = [&](int j) { return __uint_as_float(r[j]); };
            const float m0 = max3(f(0), f(1), f(2)), m1 = max3(f(3), f(4), f(5)), m2 = max3(f(6), f(7), f(8)), m3 = max3(f(9), f(10), f(11));
            const float m4 = max3(f(12), f(13), f(14));
            return fmaxf(max3(m0, m1, m2), max3(m3, m4, f(15)));
          };
#pragma unroll
          for (int h = 0; h < HALVES; ++h) {
            constexpr uint32_t laps = kFull / kEpilogueGroups;  // barriers that this group uses in turn
            const int a = accumulator(t, h);
            wait(acc_full + 8 * (HALVES * (group + kEpilogueGroups * (turn % laps)) + h), (turn / laps) & 1u, 1 + t);
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (h == 0) bound = bounds[(t & (kBoundRing - 1)) * kTileM + pt];  // before acc_free: a later tile's takes its place
            const uint32_t addr = lane_addr + (uint32_t)a * 128u;
            tmem_ld16(addr, ra);
#pragma unroll
            for (int q = 0; q < 8; q += 2) {
              tmem_wait(ra);
              tmem_ld16(addr + (uint32_t)(16 * q + 16), rb);
              row_max[8 * h + q] = group_max(ra);
              float own[16];
#pragma unroll
              for (int j = 0; j < 16; ++j) own[j] = __uint_as_float(ra[j]);
              tmem_wait(rb);
              if (q + 2 < 8) {
                tmem_ld16(addr + (uint32_t)(16 * q + 32), ra);
              } else {  // the next MMAs may overwrite the accumulator
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_free + 8 * a);
              }
              row_max[8 * h + q + 1] = group_max(rb);
#pragma unroll
              for (int j = 0; j < 16; ++j)
                col_max[j] = h == 0 && q == 0 ? fmaxf(own[j], __uint_as_float(rb[j])) : max3(col_max[j], own[j], __uint_as_float(rb[j]));
            }
          }
          float best = row_max[0];
#pragma unroll
          for (int q = 1; q + 1 < kGroups; q += 2) best = max3(best, row_max[q], row_max[q + 1]);
          best = fmaxf(best, row_max[kGroups - 1]);
          // hits, each counted as 64 + its number: from 64 to 127 there was one
          const float from = best - bound;
          int rows_hit[2] = {0, 0}, cols_hit[2] = {0, 0};
#pragma unroll
          for (int q = 0; q < kGroups; ++q) add_if_ge(rows_hit[q & 1], row_max[q], from, 64 + q);
#pragma unroll
          for (int j = 0; j < 16; ++j) add_if_ge(cols_hit[j & 1], col_max[j], from, 64 + j);
          const int r_hit = rows_hit[0] + rows_hit[1], c_hit = cols_hit[0] + cols_hit[1];
          const bool zero = bound < 0.0f;
          const int centre = zero ? 0 : 16 * r_hit + c_hit - (16 * 64 + 64);
          const bool decided = zero || ((r_hit >> 6) == 1 && (c_hit >> 6) == 1 && best > -INFINITY);
          const int64_t i = ((int64_t)blockIdx.x + (int64_t)(t - base) * gridDim.x) * kTileM + pt;
          if constexpr (FIT) {
            if (i < p.n) p.labels16[i] = (uint16_t)(decided ? (uint32_t)centre : kUndecided);
          } else {
            const bool undecided = i < p.n && !decided;
            const uint32_t listed = __ballot_sync(0xffffffffu, undecided);
            if (listed != 0u) {
              uint32_t slot = 0;
              if (lane == 0) slot = atomicAdd(open_count, (uint32_t)__popc(listed));
              slot = __shfl_sync(0xffffffffu, slot, 0) + __popc(listed & ((1u << lane) - 1u));
              if (undecided && slot < (uint32_t)kList) open_list[slot] = (uint32_t)(t * kTileM + pt);
            }
            if (i < p.n) p.labels[i] = decided ? centre : -1;
          }
        }
      }
    }
    // Behind a wait that has run out copies may still arrive in `rows`, and MMAs still read the operands: the second half's lists and centres
    // lie over the operands then, which are not used again.
    lost = __syncthreads_or(wait.gave_up) != 0;
    constexpr size_t place = kListsPlace<C>;
    static_assert(place + N * (8 * C + 5) * 4 <= O::b_chunks * lbo_b + Q::stages * a_bytes && place <= kProducerWarps * Q::slots * L::PART_BYTES, "room in both places");
    if constexpr (FIT) {
      if (end_of_iteration<C>(p, done_before + it, turns, lost ? smem : nullptr, a_ring, rows)) break;
    } else {
      settle<C>(p, turns, lost, open_list, open_count, lost ? smem + place : a_ring, lost ? smem : rows);
    }
  }

  // ---- common exit: own copies and MMAs complete (after a wait that ran out nobody else has waited for them) and all TMEM reads
  // retired, then the allocating warp frees the columns ----
  asm volatile("cp.async.wait_all;" ::: "memory");
  Waiter last{p.error, false};
  if (producer && lane == 0 && wait.gave_up)  // one copy per slot at most, since nothing is fetched after such a wait
    for (int slot = 0; slot < Q::slots; ++slot)
      if ((fetched >> slot) & 1u) last(own_full + 8 * slot, (fetched >> (8 + slot)) & 1u, 1);
  if (warp >= kMmaWarp && lane == 0) {
    mma_commit(drained + 8 * (warp - kMmaWarp));
    last(drained + 8 * (warp - kMmaWarp), 0u, 1);
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(*tmem_slot), "r"(512u) : "memory");
  }
}

constexpr size_t kOneCta = 120 * 1024;  // shared memory that keeps a second CTA off the SM: it would only wait for the TMEM columns

inline void describe(Params& p, const float* x, const float* y, int64_t n, int64_t k, int64_t d, int metric) {
  p.x = x; p.y = y; p.n = n; p.k = (int)k; p.d = (int)d; p.metric = metric;
  p.x_aligned = aligned(x, 16);
  p.x_wide = d % 4 == 0;  // of the copy in shared memory
  p.y_wide = d % 4 == 0 && aligned(y, 16);
  p.never = ~0u;
  // relative error bound of one score: the split leaves 3 * 2^-22 of |x||y|, the rest is the sums of up to 13 MMAs of 16 products
  p.eps = d <= 32 ? 1.0f / 65536.0f : 1.0f / 32768.0f;
}

}  // namespace tc
}  // namespace f2c
