// Launch parameters shared by the fused VQ / two-level aggregation kernels.
#pragma once
#include "common.cuh"

namespace f2c {

// Row-sharded tables (PEER kernels): node row r (VQ codes, slot) lives on shard r / rps_nodes, hot row h on shard
// h / rps_hot; every shard is mapped into this process (own memory or CUDA-IPC peer mappings).
struct VqPeer {
  const uint8_t* code[8];
  const int32_t* slot[8];   // all null = hot-first numbering
  const uint8_t* hot[8];
  uint32_t rps_nodes, rps_hot;
  unsigned long long magic_nodes, magic_hot;  // floor(2^64 / rps) + 1: exact 32-bit division by one multiply-high
};

struct VqParams {
  const void* codes;       // [n_src, n_cb]
  const float* codebooks;  // [n_cb, K, cs]
  const void* indptr;
  const void* indices;
  float* out;
  int64_t n_dst;
  int n_cb, cs, feat_dim;
  uint32_t K;
  int code_kind;           // 0 u8, 1 i8, 2 i16
  int cb_per_part;         // codebooks (subspaces) handled by one blockIdx.y
  int reduce;
  int vec_store;
  DropoutArgs drop;
  // two-level extension
  const uint8_t* sq_codes;  // [n_hot, sq_row_bytes]
  const float* sq_codebooks;
  const int32_t* slot;      // [n_src] row of the SQ table or -1; nullptr = hot-first numbering: source s is hot iff s < n_hot, row s
  int64_t n_hot;
  int64_t sq_row_bytes;
  int sq_cs, sq_n_cb, sq_signed;
  // geometry of the codebooks staged by the pipelined kernel (fused_vq_fast.cu)
  int fast_stride;    // bytes between consecutive codes of one subspace in shared memory
  int fast_spq;       // subspaces interleaved per 128-byte line (1 = natural layout)
  int fast_cb_bytes;  // staged bytes per column part
  VqPeer peer;        // only read by PEER kernels
};

// Codebooks of n_sub subspaces (n_sub x K centroids of cs floats, cs % 4 == 0, 16-byte aligned) into shared memory with threads
// 0 .. nthr-1: as they are (spq = 1), or - cs a power of two below 32 - with the centroids `code` of spq consecutive subspaces
// side by side in a 128-byte line.  Copies are asynchronous, so that all of a thread's are in flight at once (loads through
// registers with a division per piece took 2.4 us more for 16 x 256 x 8 floats); they are complete after
// codebooks_staged() and a barrier.
__device__ __forceinline__ void copy16_async(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void stage_codebooks(unsigned char* dst, const float* __restrict__ src, int n_sub, int K, int cs, int spq, int nthr) {
  const uint32_t to = (uint32_t)__cvta_generic_to_shared(dst);
  if (spq > 1) {
    const int lg4 = 31 - __clz(cs >> 2);
    const int piece = threadIdx.x & 7, q = piece & ((1 << lg4) - 1);  // nthr is a multiple of 8
    for (int grp = 0; grp * spq < n_sub; ++grp) {
      const int sl = grp * spq + (piece >> lg4);
      const uint32_t line0 = to + (uint32_t)grp * K * 128 + piece * 16;
      if (sl < n_sub) {
        const float* from = src + (int64_t)sl * K * cs + 4 * q;
        for (int code = threadIdx.x >> 3; code < K; code += nthr >> 3) copy16_async(line0 + code * 128, from + code * cs);
      }
    }
  } else {
    const int n16 = n_sub * K * (cs / 4);
    for (int i = threadIdx.x; i < n16; i += nthr) copy16_async(to + i * 16, src + 4 * i);
  }
}
__device__ __forceinline__ void codebooks_staged() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// A code row (ANY: the part's piece of it, which may start anywhere) as it arrives from memory.  A piece of up to ROWW words is
// read as the two aligned blocks of ROWW words it may touch and shifted into place by whole words, then by bytes (one load per
// word it may touch instead: two-level, 90,000 rows x 12, 100 columns in 8 121 us against 84).
template <int ROWW, bool ANY> struct CodePiece {
  uint32_t w[ROWW * (ANY ? 2 : 1)];
  uint32_t off = 0u;  // bytes before the piece
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < ROWW * (ANY ? 2 : 1); ++i) w[i] = 0u;
  }
  __device__ __forceinline__ void block(int at, const uint8_t* q, bool on) {
    if (ROWW == 1) w[at] = ldg_nc_u32_if(q, on);
    else if (ROWW == 2) { const uint2 v = ldg_nc_u64_if(q, on); w[at] = v.x; w[at + (ROWW > 1 ? 1 : 0)] = v.y; }
    else { const uint4 v = ldg_nc_u128_if(q, on); w[at] = v.x; w[at + (ROWW > 1 ? 1 : 0)] = v.y; w[at + (ROWW > 2 ? 2 : 0)] = v.z; w[at + (ROWW > 3 ? 3 : 0)] = v.w; }
  }
  __device__ __forceinline__ void fetch(const uint8_t* at, uint32_t bytes, bool on) {
    if (ANY) {  // only blocks that hold a byte of it are read
      off = (uint32_t)(reinterpret_cast<uintptr_t>(at) & (4u * ROWW - 1u));
      block(0, at - off, on);
      block(ANY ? ROWW : 0, at - off + 4 * ROWW, on && off + bytes > 4u * ROWW);
    } else {
      block(0, at, on);
    }
  }
  __device__ __forceinline__ void join(uint32_t (&c)[ROWW]) const {
    if constexpr (!ANY) {
#pragma unroll
      for (int i = 0; i < ROWW; ++i) c[i] = w[i];
    } else {
      uint32_t x[ROWW + 2];
#pragma unroll
      for (int i = 0; i < ROWW + 2; ++i) {  // whole words: 2 of ROWW = 4 here, then 1
        const int j = i < 2 * ROWW ? i : 2 * ROWW - 1, k = i + 2 < 2 * ROWW ? i + 2 : 2 * ROWW - 1;
        x[i] = ROWW == 4 && (off & 8u) ? w[k] : w[j];
      }
#pragma unroll
      for (int i = 0; i < ROWW + 1; ++i) x[i] = ROWW > 1 && (off & 4u) ? x[i + 1] : x[i];
#pragma unroll
      for (int i = 0; i < ROWW; ++i) c[i] = __funnelshift_r(x[i], x[i + 1], (off & 3u) * 8u);
    }
  }
};

// Streamed (fused_vq_stream.cu) or register-prefetch (fused_vq_fast.cu) kernel for the common shapes, by `variant`
// (an f2c_kernel value); sets *served = false (and launches nothing) when the shape is not one of theirs.
int launch_vq_fast(VqParams& p, int hot_bits, int index_dtype, int variant, cudaStream_t st, const char* op, bool* served,
                   bool peer = false);

// Two destination rows per warp, nearly any shape (fused_vq_rows.cu), for VQ tables of this GPU.
int launch_vq_rows(VqParams& p, int index_dtype, cudaStream_t st, const char* op, bool* served);

// Make sure the current device can read `ptr` (device memory of this or another GPU of the box): peer access is
// one-directional and is requested here when needed (idempotent).  Returns a status with the error text set.
int ensure_readable_from_current_device(const void* ptr, const char* op, const char* what, int index);

// Hot-row slot of source node `id`: looked up, or - with hot-first numbering (no slot array) - the id itself.
__device__ __forceinline__ int hot_slot_of(const VqParams& p, int64_t id) {
  if (p.slot != nullptr) return __ldg(p.slot + id);
  return id < p.n_hot ? (int)id : -1;
}

}  // namespace f2c
