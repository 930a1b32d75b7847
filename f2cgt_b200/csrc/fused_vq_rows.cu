// Fused VQ decode + aggregation, two destination rows per warp (reference operator vq_decompress_spmm_csr,
// src/fusion_spmm.cu:72-141; same arithmetic and CSC summation order as the general kernel of fused_vq_spmm.cu), for the shapes
// that the pipelined kernel of fused_vq_fast.cu does not take: code rows of any length and alignment, 16-bit codes, rows of the
// output that are not whole 16-byte pieces, column slices that do not divide 128 - and for parts of at most 64 columns, where a
// whole warp per row would leave half of its lanes idle.
//
// What bounds it.  A code row is a few bytes, so HBM moves little; what counts is shared memory (a centroid per edge and
// subspace: 512 bytes per edge at 128 columns, four wavefronts), the gather of the code rows, and the instructions around
// them.  So
//  * half a warp owns a destination row: a lane owns four columns of each 64-column chunk of the part, and the work per row
//    is done for two rows at once; additions are packed (add.f32x2), the mean is one reciprocal per row and two exact
//    corrections per column, loads are predicated instead of branched around;
//  * lane t of a half holds neighbour t's code bytes as aligned blocks, joined by shifts where rows start anywhere,
//    and turns them into a tile [subspace][neighbour]: a lane then reads the codes of its subspace of all 16 neighbours
//    at once.
// Codebooks of a column part of at most 128 columns are staged once per persistent CTA, subspaces narrower than 32 columns
// interleaved in 128-byte lines: the eight lanes of a quarter-warp read eight different bank groups whatever the codes are.
// Pipeline over the row pairs of a warp: the code rows of a pair, the ids of the next and the offsets of the one after are in
// flight between two iterations.
// Measured on B200, 90,000 rows x 12 neighbours, general kernel -> this one: 110 columns in slices of 8 95 -> 51 us, 200 in 32
// 173 -> 62, 100 in 16 89 -> 37, 128 in 16 with 1024 centroids 280 -> 122; 128 columns in 8 or 32 tie with the pipelined kernel (39,
// 32 us), which stays for them because it starts faster (300 rows: 7.9 against 8.6 us).
#include "sq_fused.cuh"
#include "vq_params.cuh"

namespace f2c {
namespace vqr {

constexpr int kThreads = 768;
constexpr int kWarps = kThreads / 32;
constexpr int kNb = 16;  // neighbours held per row; rows with more take further rounds, fetched on the spot
constexpr size_t kSmemLimit = 227 * 1024;
// a warp's tile of codes: per half WORDS * 4 code bytes x 16 neighbours, the halves in different banks
constexpr int tile_bytes(int words) { return 2 * (words * 4 * kNb + 16); }

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint4 lds_u128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ void add_if(unsigned long long& acc, unsigned long long v, bool on) {
  asm("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q add.rn.f32x2 %0, %0, %1;\n\t}" : "+l"(acc) : "l"(v), "r"((uint32_t)on));
}
// NCH: 64-column chunks per part (1, 2).  WORDS: words of a row's code bytes in the part.  ANY: any alignment.  EB: bytes per code.
template <typename IdxT, int NCH, int WORDS, bool ANY, int EB>
__global__ void __launch_bounds__(kThreads, 1) vq_rows_kernel(const VqParams p) {
  dependency_wait();
  release_dependents();
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int SUBS = WORDS * 4 / EB;  // subspaces a part may have
  constexpr int HALF = tile_bytes(WORDS) / 2;
  unsigned char* cb_s = smem;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, half = lane >> 4, hl = lane & 15;
  unsigned char* tile = smem + p.fast_cb_bytes + wid * 2 * HALF;  // per half: codes of subspace s of the 16 neighbours at s * 16 * EB
  float* out_s = reinterpret_cast<float*>(smem + p.fast_cb_bytes + kWarps * 2 * HALF) + wid * 2 * 64 * NCH;  // unless vec_store

  const int s_begin = (int)blockIdx.y * p.cb_per_part, s_end = min(s_begin + p.cb_per_part, p.n_cb), n_sub = s_end - s_begin;
  const int col_begin = s_begin * p.cs, col_end = min(s_end * p.cs, p.feat_dim);
  const int K = (int)p.K, cs = p.cs, spq = p.fast_spq, stride = p.fast_stride;
  stage_codebooks(cb_s, p.codebooks + (int64_t)s_begin * K * cs, n_sub, K, cs, spq, kThreads);
  // ---- lane constants
  uint32_t cb_addr[NCH], code_addr[NCH];
  bool active[NCH];
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    const int col = col_begin + 64 * c + 4 * hl;
    active[c] = col < col_end;
    const int cc = active[c] ? col : col_begin;
    const int s = cc / cs, sl = s - s_begin, off = cc - s * cs;
    cb_addr[c] = smem_u32(cb_s) + (spq > 1 ? (uint32_t)((sl / spq) * K * 128 + (sl % spq) * cs * 4 + off * 4) : (uint32_t)(sl * K * stride + off * 4));
    code_addr[c] = smem_u32(tile) + (uint32_t)(half * HALF + sl * kNb * EB);
  }
  codebooks_staged();
  __syncthreads();

  const IdxT* __restrict__ indptr = reinterpret_cast<const IdxT*>(p.indptr);
  const IdxT* __restrict__ indices = reinterpret_cast<const IdxT*>(p.indices);
  const uint32_t row_bytes = (uint32_t)p.n_cb * EB, part_bytes = (uint32_t)n_sub * EB;
  const uint8_t* __restrict__ codes = reinterpret_cast<const uint8_t*>(p.codes) + (uint32_t)s_begin * EB;
  const int n_dst = (int)p.n_dst;
  const bool clamp = (uint32_t)K < (EB == 1 ? 256u : 65536u);

  auto stage_codes = [&](const CodePiece<WORDS, ANY>& c, int cnt) {  // lane hl of a half holds neighbour hl
    if (hl < cnt) {
      uint32_t x[WORDS];
      c.join(x);
#pragma unroll
      for (int i = 0; i < WORDS; ++i) {
        if (clamp) {  // codes >= K read the last centroid, as in the general kernel
          uint32_t y = 0;
#pragma unroll
          for (int b = 0; b < 4 / EB; ++b) y |= min((x[i] >> (8 * EB * b)) & (EB == 1 ? 0xFFu : 0xFFFFu), (uint32_t)(K - 1)) << (8 * EB * b);
          x[i] = y;
        }
      }
      unsigned char* to = tile + half * HALF + hl * EB;
#pragma unroll
      for (int s = 0; s < SUBS; ++s) {
        const uint32_t v = x[s * EB / 4] >> (8 * (s * EB % 4));
        if (s < n_sub) {
          if (EB == 1) to[s * kNb] = (unsigned char)v;
          else *reinterpret_cast<uint16_t*>(to + s * kNb * 2) = (uint16_t)v;
        }
      }
    }
  };
  unsigned long long acc[NCH][2];
  auto aggregate = [&](int cnt) {  // the tile's neighbours; cnt is this half's
    const int most = max(cnt, __shfl_xor_sync(0xffffffffu, cnt, 16));
    uint32_t word[NCH][4 * EB];  // codes of this lane's subspace of all neighbours
#pragma unroll
    for (int c = 0; c < NCH; ++c)
#pragma unroll
      for (int e = 0; e < EB; ++e) {
        const uint4 v = lds_u128(code_addr[c] + 16u * e);
        word[c][4 * e] = v.x; word[c][4 * e + 1] = v.y; word[c][4 * e + 2] = v.z; word[c][4 * e + 3] = v.w;
      }
#pragma unroll
    for (int u0 = 0; u0 < kNb; u0 += 4) {
      if (u0 >= most) break;  // warp uniform
      unsigned long long v[4][NCH][2];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
          const int u = u0 + i;
          // a slot behind the half's count holds an older row's code, or - never written - anything: keep the read inside
          const uint32_t code = (word[c][u * EB / 4] >> (8 * (u * EB % 4))) & (EB == 1 ? 0xFFu : 0xFFFFu);
          lds_2x64(cb_addr[c] + (u < cnt ? code : 0u) * (uint32_t)stride, v[i][c][0], v[i][c][1]);
        }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < NCH; ++c) { add_if(acc[c][0], v[i][c][0], u0 + i < cnt); add_if(acc[c][1], v[i][c][1], u0 + i < cnt); }
    }
  };

  // ---- pipeline over the pairs q0, q0 + W, ...; stage k of the iteration at pair q works on pair q - k * W
  const int W = (int)gridDim.x * kWarps;
  const int q0 = (int)blockIdx.x * kWarps + wid, pairs = (n_dst + 1) >> 1;
  int64_t lo0 = 0, hi0 = 0;         // offsets                (loaded by stage 0, read by stage 1)
  int64_t beg1 = 0; int deg1 = 0;   // row of stage 1 -> 2
  IdxT id1 = 0;                     // this lane's neighbour   (loaded by stage 1, read by stage 2)
  int64_t beg2 = 0; int deg2 = 0;   // row of stage 2 -> 3
  CodePiece<WORDS, ANY> code2;          // its code row            (loaded by stage 2, read by stage 3)
  code2.fetch(codes, 0u, false);
  for (int q = q0;; q += W) {
    const int qa = q - 3 * W;  // pair aggregated in this iteration
    if (qa >= pairs) break;
    if (qa >= q0) {
      const int row = 2 * qa + half;
#pragma unroll
      for (int c = 0; c < NCH; ++c) acc[c][0] = acc[c][1] = 0ull;
      const int cnt = min(deg2, kNb);
      __syncwarp();
      stage_codes(code2, cnt);
      __syncwarp();
      aggregate(cnt);
      const int most = max(deg2, __shfl_xor_sync(0xffffffffu, deg2, 16));
      for (int k0 = kNb; k0 < most; k0 += kNb) {
        const int n = max(0, min(deg2 - k0, kNb));
        CodePiece<WORDS, ANY> more;
        const int64_t id = hl < n ? (int64_t)indices[beg2 + k0 + hl] : 0;
        more.fetch(codes + id * row_bytes, part_bytes, hl < n);
        __syncwarp();
        stage_codes(more, n);
        __syncwarp();
        aggregate(n);
      }
      const float degf = (float)deg2, rcp = p.reduce == F2C_MEAN && deg2 > 1 ? 1.0f / degf : 0.0f;
      if (p.vec_store) {
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
          if (row < n_dst && active[c]) {
            float4 v = make_float4(lo32(acc[c][0]), hi32(acc[c][0]), lo32(acc[c][1]), hi32(acc[c][1]));
            if (rcp != 0.0f) v = div4(v, degf, rcp);
            const int64_t at = (int64_t)row * p.feat_dim + col_begin + 64 * c + 4 * hl;
            if (p.drop.enabled) v = dropout_apply4(v, (uint64_t)at, p.drop);
            stg_cs_f4(p.out + at, v);
          }
        }
      } else {  // rows start anywhere: through shared memory, so that lanes write consecutive columns
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
          float4 v = make_float4(lo32(acc[c][0]), hi32(acc[c][0]), lo32(acc[c][1]), hi32(acc[c][1]));
          if (rcp != 0.0f) v = div4(v, degf, rcp);
          *reinterpret_cast<float4*>(out_s + half * 64 * NCH + 64 * c + 4 * hl) = v;
        }
        __syncwarp();
        if (row < n_dst)
          store_run(p.out, (int64_t)row * p.feat_dim + col_begin, col_end - col_begin, hl, 16, p.drop, [&](int c) { return out_s[half * 64 * NCH + c]; });
      }
    }
    // ---- stage 2: ids have arrived; fetch the code rows
    beg2 = beg1; deg2 = deg1;
    code2.fetch(codes + (int64_t)id1 * row_bytes, part_bytes, hl < deg1);
    // ---- stage 1: offsets have arrived; fetch the ids
    beg1 = lo0; deg1 = (int)(hi0 - lo0);
    id1 = (IdxT)0;
    if (hl < deg1) id1 = __ldg(indices + beg1 + hl);
    // ---- stage 0: offsets of this lane's row of pair q
    const int next = 2 * q + half;
    lo0 = hi0 = 0;
    if (q < pairs && next < n_dst) { lo0 = (int64_t)__ldg(indptr + next); hi0 = (int64_t)__ldg(indptr + next + 1); }
  }
}

template <typename IdxT, int NCH, int WORDS, bool ANY, int EB>
static int launch(const VqParams& p, dim3 grid, size_t smem, cudaStream_t st, const char* op) {
  auto kern = vq_rows_kernel<IdxT, NCH, WORDS, ANY, EB>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return set_error(F2C_ERR_CUDA, "%s: %s", op, cudaGetErrorString(e));
  launch_dependent(kern, grid, dim3(kThreads), smem, st, p);
  return check_launch(op);
}

template <typename IdxT, int NCH, int EB>
static int launch_words(const VqParams& p, int words, bool any, dim3 grid, size_t smem, cudaStream_t st, const char* op) {
  if (any) {
    if (words == 1) return launch<IdxT, NCH, 1, true, EB>(p, grid, smem, st, op);
    if (words == 2) return launch<IdxT, NCH, 2, true, EB>(p, grid, smem, st, op);
    return launch<IdxT, NCH, 4, true, EB>(p, grid, smem, st, op);
  }
  if (words == 1) return launch<IdxT, NCH, 1, false, EB>(p, grid, smem, st, op);
  if (words == 2) return launch<IdxT, NCH, 2, false, EB>(p, grid, smem, st, op);
  return launch<IdxT, NCH, 4, false, EB>(p, grid, smem, st, op);
}

}  // namespace vqr

// VQ aggregation on the kernel above; *served = false when the shape is not one of its own.
int launch_vq_rows(VqParams& p, int index_dtype, cudaStream_t st, const char* op, bool* served) {
  using namespace vqr;
  *served = false;
  const int eb = p.code_kind == 2 ? 2 : 1;
  if (p.code_kind == 1 || p.K > (eb == 1 ? 256u : 32768u) || p.n_dst >= (1ll << 30) || p.cs % 4 != 0 || !aligned(p.codebooks, 16)) return F2C_OK;
  const bool pow2 = (p.cs & (p.cs - 1)) == 0;
  auto words_of = [&](int n_sub) { const int w = (n_sub * eb + 3) / 4; return w > 2 ? 4 : w; };
  // interleaved lines while a part of at least 64 columns fits in them; else the natural layout, whose occasional bank conflicts
  // matter less than a part with few columns
  int spq = pow2 && p.cs < 32 ? 32 / p.cs : 1, per_part = 0;
  auto cb_bytes = [&](int n_sub) { return spq > 1 ? (size_t)ceil_div(n_sub, spq) * p.K * 128 : (size_t)n_sub * p.K * p.cs * 4; };
  for (;; spq = 1) {
    per_part = 128 / p.cs;
    if (per_part * eb > 16) per_part = 16 / eb;  // code bytes a lane holds
    if (per_part > p.n_cb) per_part = p.n_cb;
    while (per_part >= 1 && cb_bytes(per_part) + (size_t)kWarps * tile_bytes(words_of(per_part)) + (p.vec_store ? 0 : (size_t)kWarps * 2 * 64 * 2 * 4) > kSmemLimit)
      --per_part;
    if (spq == 1 || per_part * p.cs >= 64 || per_part == p.n_cb) break;
  }
  if (per_part < 1) return F2C_OK;
  const int parts = (int)ceil_div(p.n_cb, per_part);
  if (parts > 16) return F2C_OK;
  per_part = (int)ceil_div(p.n_cb, parts);  // even parts
  const int bytes = per_part * eb, words = words_of(per_part), nch = per_part * p.cs > 64 ? 2 : 1;
  p.cb_per_part = per_part;
  p.fast_spq = spq;
  p.fast_stride = spq > 1 ? 128 : p.cs * 4;
  p.fast_cb_bytes = (int)((cb_bytes(per_part) + 15) / 16 * 16);
  // aligned loads: every row and part is one whole load
  const size_t row = (size_t)p.n_cb * eb, load = (size_t)words * 4;
  const bool any = !(row % load == 0 && bytes == (int)load && p.n_cb % per_part == 0 && aligned(p.codes, load));
  const size_t smem = (size_t)p.fast_cb_bytes + (size_t)kWarps * tile_bytes(words) + (p.vec_store ? 0 : (size_t)kWarps * 2 * 64 * nch * 4);
  int64_t grid_x = current_sm_count() / parts;
  if (grid_x < 1) grid_x = 1;
  const int64_t need = ceil_div(p.n_dst, 2 * kWarps);
  if (grid_x > need) grid_x = need;
  const dim3 grid((unsigned)grid_x, (unsigned)parts);
  *served = true;
#define F2C_VQR(T)                                                                                                                     \
  if (eb == 2) return nch == 2 ? launch_words<T, 2, 2>(p, words, any, grid, smem, st, op) : launch_words<T, 1, 2>(p, words, any, grid, smem, st, op); \
  return nch == 2 ? launch_words<T, 2, 1>(p, words, any, grid, smem, st, op) : launch_words<T, 1, 1>(p, words, any, grid, smem, st, op)
  if (index_dtype == F2C_I32) { F2C_VQR(int32_t); }
  F2C_VQR(int64_t);
#undef F2C_VQR
}

}  // namespace f2c
