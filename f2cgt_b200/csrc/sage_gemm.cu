// Forward product of a GraphSAGE layer on the 5th-generation tensor cores:
//   Y [m, n] = act((X1 W1^T + b) + X2 W2^T)      (fc_self and fc_neigh of examples/conv.py:62-76, act = ReLU or nothing)
//
// What bounds it.  A layer of a minibatch has 10^3 .. 10^5 rows of 64 .. 256 columns: the product reads its rows once and
// computes little, so HBM does (59,000 rows x (128 + 128) columns: 60 MB in, 30 MB out, 14 us).  As two library products and
// a ReLU the output made four more trips (14 + 29 + 8 us).  Here one persistent kernel, one CTA per SM:
//  * a warp brings 128 rows x 32 columns per step with TMA (128-byte swizzle, rounded to tf32 on the way, zero behind the
//    matrix' edges) through a ring of stages; the weights of the CTA's column tile stay in shared memory when they fit beside
//    the ring, else their pieces travel with the rows;
//  * a thread issues the MMAs (128 x up to 128, four per step).  X1 W1^T and X2 W2^T have an accumulator each, and two tiles
//    alternate: 4 x 128 columns of TMEM.  Separate accumulators cost nothing and keep the result the same, bit for bit, as
//    the two products one after the other (a sum in another order moves hidden values by an ulp, tf32 rounding of the next
//    layer's operands turns that into 2^-11, and a ReLU near zero into a different gradient);
//  * four warps add bias and the two sums, apply the ReLU and write 128-byte pieces of rows through shared memory, while the
//    next tile is loaded and multiplied.
// Every wait is bounded: when one runs out the CTA's roles all leave, the rows it has not finished become NaN (whoever uses them
// sees it), the copies and products still in flight are waited for, the error word is raised and TMEM is freed.
#include <cuda.h>

#include <mutex>

#include "common.cuh"

namespace f2c {

int* stream_error_word();

namespace sg {

constexpr int kThreads = 192;            // warp 0: TMA, warp 1: MMA, warps 2-5: epilogue
constexpr int kM = 128, kN = 128, kK = 32;
constexpr int kABytes = kM * kK * 4;     // 16 KB
constexpr int kMaxStages = 6;
constexpr int kEpiFloats = 32 * 36;      // per epilogue warp: 32 rows x 32 columns, rows padded by 16 bytes
constexpr size_t kSmemLimit = 227 * 1024;
constexpr uint32_t kWaitLimit = 1u << 22;

struct Params {
  float* y;
  const float* bias;
  int64_t m;
  int n, k;
  int relu;
  int stages, resident;    // stages of the ring; 1: the weights stay in shared memory
  int b_rows;              // rows of a weight piece (column tile), a multiple of 16
  int tiles;               // row tiles
  int* error;
};

struct Bars {
  uint64_t full[kMaxStages], empty[kMaxStages], weights, drain, acc_full[2], acc_empty[2];
  uint32_t tmem;
  int failed;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// K-major, 128-byte swizzle: rows of 128 bytes, atoms of 8 rows (1024 bytes)
__device__ __forceinline__ uint64_t make_desc(uint32_t addr) {
  const uint32_t lo = ((addr & 0x3FFFFu) >> 4) | (1u << 16);
  const uint32_t hi = (1024u >> 4) | (1u << 14) | (2u << 29);
  return ((uint64_t)hi << 32) | lo;
}

__device__ __forceinline__ void mma_tf32(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}\n" ::"r"(d_tmem), "l"(a), "l"(b), "r"(idesc),
      "r"(accumulate), "r"(0u)
      : "memory");
}

__device__ __forceinline__ void commit(const uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void init_bar(const uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void arrive(const uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void expect(const uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// false when the limit ran out or another role has given up
__device__ __forceinline__ bool wait_bar(const uint64_t* bar, uint32_t parity, volatile int* failed) {
  uint32_t done = 0;
  for (uint32_t it = 0; it < kWaitLimit; ++it) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    if (done) return true;
    if ((it & 255u) == 255u && *failed) return false;
  }
  *failed = 1;
  return false;
}

__device__ __forceinline__ void tma_load(const CUtensorMap* map, uint32_t dst, const uint64_t* bar, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
               "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}

__global__ void __launch_bounds__(kThreads, 1) sage_forward_kernel(const __grid_constant__ CUtensorMap x1, const __grid_constant__ CUtensorMap x2,
                                                                   const __grid_constant__ CUtensorMap w1, const __grid_constant__ CUtensorMap w2,
                                                                   const Params p) {
  dependency_wait();
  release_dependents();
  extern __shared__ unsigned char smem_raw[];
  __shared__ Bars bars;
  __shared__ __align__(16) float epi_s[4 * kEpiFloats];
  __shared__ float bias_s[kN];
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
  const int per_segment = (p.k + kK - 1) / kK, steps = 2 * per_segment;
  const int col0 = (int)blockIdx.y * kN;
  const int tile_cols = min(kN, p.n - col0);
  const uint32_t b_bytes = (uint32_t)p.b_rows * kK * 4;
  // shared memory: resident weights (one piece per step), then the ring
  unsigned char* weights = smem;
  unsigned char* ring = smem + (p.resident ? (size_t)steps * b_bytes : 0);
  const uint32_t stage_bytes = kABytes + (p.resident ? 0u : b_bytes);
  volatile int* failed = &bars.failed;

  if (wid == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars.tmem)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int s = 0; s < p.stages; ++s) { init_bar(bars.full + s, 1); init_bar(bars.empty + s, 1); }
    init_bar(&bars.weights, 1);
    init_bar(&bars.drain, 1);
    for (int b = 0; b < 2; ++b) { init_bar(bars.acc_full + b, 1); init_bar(bars.acc_empty + b, 4); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    bars.failed = 0;
  }
  if (tid < kN) bias_s[tid] = p.bias != nullptr && col0 + tid < p.n ? __ldg(p.bias + col0 + tid) : 0.0f;
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = bars.tmem;
  int s = 0;  // loading thread: stage and round of its next load
  uint32_t round = 0;

  if (wid == 0) {
    // ================= loads
    if (lane == 0) {
      if (p.resident) {
        expect(&bars.weights, (uint32_t)steps * b_bytes);
        for (int i = 0; i < steps; ++i)
          tma_load(i < per_segment ? &w1 : &w2, smem_u32(weights + (size_t)i * b_bytes), &bars.weights, (i % per_segment) * kK, col0);
      }
      for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x) {
        for (int i = 0; i < steps; ++i) {
          if (round > 0 && !wait_bar(bars.empty + s, (round - 1) & 1, failed)) { tile = p.tiles; break; }
          unsigned char* stage = ring + (size_t)s * stage_bytes;
          const int x = (i % per_segment) * kK;
          expect(bars.full + s, stage_bytes);
          tma_load(i < per_segment ? &x1 : &x2, smem_u32(stage), bars.full + s, x, tile * kM);
          if (!p.resident) tma_load(i < per_segment ? &w1 : &w2, smem_u32(stage + kABytes), bars.full + s, x, col0);
          if (++s == p.stages) { s = 0; ++round; }
        }
      }
    }
  } else if (wid == 1) {
    // ================= MMAs
    if (lane == 0) {
      // fp32 accumulate, tf32 operands, N / 8, M / 16
      const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(p.b_rows >> 3) << 17) | ((uint32_t)(kM >> 4) << 24);
      bool ok = !p.resident || wait_bar(&bars.weights, 0, failed);
      uint32_t t = 0;
      for (int tile = blockIdx.x; ok && tile < p.tiles; tile += gridDim.x, ++t) {
        const uint32_t buf = t & 1u;
        if (t >= 2) ok = wait_bar(bars.acc_empty + buf, ((t >> 1) - 1) & 1, failed);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int i = 0; ok && i < steps; ++i) {
          ok = wait_bar(bars.full + s, round & 1, failed);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a_addr = smem_u32(ring + (size_t)s * stage_bytes);
          const uint32_t b_addr = p.resident ? smem_u32(weights + (size_t)i * b_bytes) : a_addr + kABytes;
          const int seg = i >= per_segment;
          const uint32_t acc = tmem + buf * 256u + (uint32_t)seg * 128u;
#pragma unroll
          for (int q = 0; q < kK / 8; ++q)
            mma_tf32(acc, make_desc(a_addr + q * 32), make_desc(b_addr + q * 32), idesc, (i - seg * per_segment) + q != 0 ? 1u : 0u);
          commit(bars.empty + s);
          if (++s == p.stages) { s = 0; ++round; }
        }
        if (ok) commit(bars.acc_full + buf);
      }
    }
  } else {
    // ================= epilogue: warp w owns the TMEM lanes of its quarter; 32 x 32 pieces go through shared memory so that
    //                   eight lanes write 128 consecutive bytes of a row
    const int quarter = wid & 3, piece = lane & 7;
    float* epi = epi_s + (wid - 2) * kEpiFloats;
    const bool vec = (p.n & 3) == 0 && (((uintptr_t)p.y) & 15) == 0;
    uint32_t t = 0;
    bool lost = false;  // a wait ran out
    for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x, ++t) {
      const uint32_t buf = t & 1u;
      const int64_t row0 = (int64_t)tile * kM + quarter * 32;
      lost = lost || !__all_sync(0xffffffffu, wait_bar(bars.acc_full + buf, (t >> 1) & 1, failed));
      if (lost) {
        for (int64_t row = row0; row < row0 + 32 && row < p.m; ++row)
          for (int c = lane; c < tile_cols; c += 32) p.y[row * p.n + col0 + c] = __int_as_float(0x7fffffff);
        continue;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int c0 = 0; c0 < tile_cols; c0 += 32) {
        uint32_t r1[32], r2[32];
        const uint32_t at = tmem + ((uint32_t)(quarter * 32) << 16) + buf * 256u + (uint32_t)c0;
        tmem_ld32(at, r1);
        tmem_ld32(at + 128u, r2);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (c0 + 32 >= tile_cols) {  // the accumulators have been read
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) arrive(bars.acc_empty + buf);
        }
        const int col = col0 + c0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          float v[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int j = 4 * q + e;
            float a = __uint_as_float(r1[j]);
            if (p.bias != nullptr) a += bias_s[c0 + j];
            a += __uint_as_float(r2[j]);
            v[e] = p.relu && a <= 0.f ? 0.f : a;  // a NaN stays one, as in torch.relu
          }
          *reinterpret_cast<float4*>(epi + lane * 36 + 4 * q) = make_float4(v[0], v[1], v[2], v[3]);
        }
        __syncwarp();
        const int c = col + 4 * piece;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int rl = (lane >> 3) + 4 * q;
          const int64_t row = row0 + rl;
          if (row >= p.m || c >= p.n) continue;
          const float4 v = *reinterpret_cast<const float4*>(epi + rl * 36 + 4 * piece);
          float* o = p.y + row * p.n + c;
          if (vec) {
            *reinterpret_cast<float4*>(o) = v;
          } else {
            o[0] = v.x;
            if (c + 1 < p.n) o[1] = v.y;
            if (c + 2 < p.n) o[2] = v.z;
            if (c + 3 < p.n) o[3] = v.w;
          }
        }
        __syncwarp();
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (bars.failed) {
    // loads in flight write to this CTA's shared memory, MMAs in flight read it and write its TMEM: wait (bounded) for what was issued
    volatile int expired = 0;  // (set by a wait that runs out again; the next one then gives up soon)
    if (tid == 0) {
      if (p.resident) wait_bar(&bars.weights, 0, &expired);
      for (int q = 0; q < p.stages; ++q) {
        const uint32_t uses = round + (q < s ? 1u : 0u);
        if (uses > 0) wait_bar(bars.full + q, (uses - 1) & 1, &expired);
      }
    } else if (tid == 32) {
      commit(&bars.drain);
      wait_bar(&bars.drain, 0, &expired);
    }
    __syncthreads();
  }
  if (wid == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
  if (tid == 0 && bars.failed) report_wait(p.error, 3);
}

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                              const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeFn encode_fn() {
  static std::mutex m;
  static EncodeFn fn = nullptr;
  std::lock_guard<std::mutex> lock(m);
  if (fn == nullptr) {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult found{};
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &found) == cudaSuccess && found == cudaDriverEntryPointSuccess)
      fn = (EncodeFn)f;
  }
  return fn;
}

// row-major [rows, cols] floats, boxes of box_rows x 32
static bool make_map(EncodeFn fn, CUtensorMap* map, const float* base, int64_t rows, int64_t cols, int box_rows) {
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)cols * 4};
  const cuuint32_t box[2] = {kK, (cuuint32_t)box_rows}, step[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_TFLOAT32, 2, (void*)base, dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace sg
}  // namespace f2c

using namespace f2c;

extern "C" int f2c_sage_forward(const float* x1, const float* x2, const float* w1, const float* w2, const float* bias, float* y, int64_t m,
                                int64_t n, int64_t k, int relu, void* stream) {
  const char* op = "sage_forward";
  F2C_REQUIRE(m >= 0 && n >= 1 && k >= 1, F2C_ERR_INVALID, "%s: bad shape m=%lld n=%lld k=%lld", op, (long long)m, (long long)n, (long long)k);
  F2C_REQUIRE(k % 4 == 0, F2C_ERR_UNSUPPORTED, "%s: k must be a multiple of 4", op);
  F2C_REQUIRE(m < (1ll << 31) - sg::kM && n <= 65536 && k <= 65536, F2C_ERR_LIMIT, "%s: shape too large", op);
  if (m == 0) return F2C_OK;
  F2C_REQUIRE(x1 && x2 && w1 && w2 && y, F2C_ERR_INVALID, "%s: null pointer", op);
  F2C_REQUIRE(aligned(x1, 16) && aligned(x2, 16) && aligned(w1, 16) && aligned(w2, 16), F2C_ERR_INVALID, "%s: misaligned operand", op);
  sg::EncodeFn fn = sg::encode_fn();
  F2C_REQUIRE(fn != nullptr, F2C_ERR_CUDA, "%s: the driver does not offer cuTensorMapEncodeTiled", op);
  sg::Params p{};
  p.y = y; p.bias = bias; p.m = m; p.n = (int)n; p.k = (int)k; p.relu = relu; p.error = stream_error_word();
  p.tiles = (int)ceil_div(m, sg::kM);
  p.b_rows = (int)(n < sg::kN ? (n + 15) / 16 * 16 : sg::kN);
  const int steps = 2 * (int)ceil_div(k, sg::kK);
  const size_t b_bytes = (size_t)p.b_rows * sg::kK * 4, room = sg::kSmemLimit - 1024 - sizeof(sg::Bars) - 4 * sg::kEpiFloats * 4 - sg::kN * 4 - 256;
  // resident weights while at least four stages of rows fit beside them
  p.resident = steps * b_bytes + 4 * sg::kABytes <= room;
  const size_t stage = sg::kABytes + (p.resident ? 0 : b_bytes), fixed = p.resident ? steps * b_bytes : 0;
  p.stages = (int)((room - fixed) / stage);
  if (p.stages > sg::kMaxStages) p.stages = sg::kMaxStages;
  size_t smem = fixed + p.stages * stage + 1024;
  if (smem < 120 * 1024) smem = 120 * 1024;  // one CTA per SM: it owns all of TMEM
  CUtensorMap maps[4];
  const bool ok = sg::make_map(fn, maps, x1, m, k, sg::kM) && sg::make_map(fn, maps + 1, x2, m, k, sg::kM) &&
                  sg::make_map(fn, maps + 2, w1, n, k, p.b_rows) && sg::make_map(fn, maps + 3, w2, n, k, p.b_rows);
  F2C_REQUIRE(ok, F2C_ERR_CUDA, "%s: tensor map", op);
  cudaError_t e = cudaFuncSetAttribute(sg::sage_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return set_error(F2C_ERR_CUDA, "%s: %s", op, cudaGetErrorString(e));
  const int col_tiles = (int)ceil_div(n, sg::kN);
  int64_t grid = current_sm_count() / col_tiles;
  if (grid < 1) grid = 1;
  if (grid > p.tiles) grid = p.tiles;
  launch_dependent(sg::sage_forward_kernel, dim3((unsigned)grid, (unsigned)col_tiles), sg::kThreads, smem, (cudaStream_t)stream, maps[0], maps[1], maps[2],
                                                                                                               maps[3], p);
  return check_launch(op);
}
