// Features -> stored codes in one pass: what the offline compressor does with sq_compress, a cast and packbits
// (reference: examples/process_compress.py:120-141), i.e. fp32-valued codes written and read again, a byte per element
// written and read again, then the packed bytes.  Here a value is read once and its code leaves packed.
//
// What bounds it.  The pass moves 4 + bits/8 bytes per element; the reference's expression (log2f, an IEEE division, floor)
// takes several times as long in instructions.  For 2, 4 and 8 bits it is therefore evaluated only where its result is not
// already certain: the position before floor() comes from the hardware's approximate log2 with one FMA, and unless it lies
// within its error bound of an integer (a few elements in a hundred thousand to ten thousand) floor() of it is the level.
// Clamped values, one in a hundred by construction, need no care of their own: the expression is monotonic, so once its
// levels AT the clamps are known, positions beyond them are clamped to a point inside those levels.  16-bit codes take the
// expression (the bound exceeds a hundredth of a level), 1-bit codes are a sign test.
//
// Rows whose length is a multiple of 4 columns are read as float4 by threads that keep their columns (and so their codebook
// row's constants) for life, other rows as groups over super-rows or, where codes do not end with a row, through shared memory
// in whole tiles, so that their loads are aligned too.
// Measured on B200 (fp32 in + codes out): 1,000,000 x 128 at 1 / 2 / 4 / 8 / 16 bits 76 / 106 / 113 / 141 / 301 us = 6.9 / 5.1 / 5.1 /
// 4.5 / 2.5 TB/s (4 bits as three passes before: 800 us); 500,001 x 117 58 / 125 / 129 us at 1 / 2 / 4 bits through the tiles.  Two rows in
// flight per thread and four CTAs per SM: more rows in flight cost registers, i.e. warps (4 rows, two CTAs: +9 %).
#include <algorithm>

#include "row_lanes.cuh"
#include "sq_encode.cuh"

namespace f2c {
namespace enc {

constexpr int kThreads = 256;
constexpr int kCtasPerSm = 4;  // vector kernel: 64 registers a thread
constexpr int kParams = 8;  // floats per codebook row in shared memory
constexpr int kMaxBooks = 512;

// floor() value of the expression for |x| = v
template <int BITS>
__device__ __forceinline__ float level(float v, const float* cb) {
  constexpr float drange = (float)(1 << (BITS - 1));
  const float fmin = __ldg(cb), fmax = __ldg(cb + 1), emin = __ldg(cb + 2), emax = __ldg(cb + 3);
  v = fminf(fmaxf(v, fmin), fmax);
  v = log2f(v);
  v = (v - emin) / (emax - emin) * drange;
  return floorf(v);
}

// Constants of one codebook row: position = log2(|x|) * scale + bias, clamped to [lo, hi]; positions within `guard` of an
// integer are undecided.  guard >= 0.5: the whole row takes the expression.
struct Row { float scale, bias, lo, hi, limit; };  // limit = 0.5 - guard

template <int BITS>
__device__ void build_params(float* par, const float* __restrict__ codebooks, int n_cb) {
  if (BITS != 1 && BITS != 16) {
    constexpr float drange = (float)(1 << (BITS - 1));
    for (int row = threadIdx.x; row < n_cb; row += blockDim.x) {
      const float* cb = codebooks + row * kCodebookDim;
      const float fmin = __ldg(cb), fmax = __ldg(cb + 1), emin = __ldg(cb + 2), emax = __ldg(cb + 3);
      const float scale = drange / (emax - emin);
      // lg2.approx is within 2^-22 or 2 ulps, log2f within an ulp, scale and bias add an ulp of |e| * scale each; the FMA and
      // the expression's subtraction, division and product a few ulps of the range
      const float guard = fabsf(scale) * (4.8e-7f + 7.2e-7f * fmaxf(fabsf(emin), fabsf(emax))) + drange * 4.8e-7f;
      const float bottom = level<BITS>(0.0f, cb), top = level<BITS>(3e38f, cb);  // at the clamps (the lower one can give -1)
      const bool sure = guard < 0.1f && fmin < fmax && fmin > 1e-30f && emin < emax && (bottom == 0.0f || bottom == -1.0f) && top == drange - 1.0f;
      float* t = par + row * kParams;
      t[0] = scale; t[1] = -emin * scale;
      t[2] = bottom == 0.0f ? 2.0f * guard : -0.5f;
      t[3] = drange - 2.0f * guard;
      t[4] = sure ? 0.5f - guard : -1.0f;
    }
  }
  __syncthreads();
}

__device__ __forceinline__ Row row_of(const float* p) { return Row{p[0], p[1], p[2], p[3], p[4]}; }

template <int BITS>
__device__ __noinline__ uint32_t encode_exact(float x, const float* cb) { return (uint32_t)(int)sq_encode<BITS>(x, cb); }

// Code of x, low bits of the result as stored (the caller masks 16-bit ones); `worst` collects how close the position
// came to an integer: once it reaches row.limit the codes of the group are to be computed again by the expression.
template <int BITS>
__device__ __forceinline__ uint32_t encode_fast(float x, const Row& row, const float* __restrict__ cb, float& worst) {
  if (BITS == 1) return x <= 0.0f ? 0u : 1u;
  if (BITS == 16) return (uint32_t)(int)sq_encode<16>(x, cb);
  constexpr uint32_t MASK = BITS >= 8 ? 0xffu : (1u << BITS) - 1u;
  constexpr uint32_t DR = BITS >= 8 ? 0u : (1u << (BITS - 1));
  float lg;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(lg) : "f"(fabsf(x)));  // a denormal becomes -inf: below the lower clamp either way
  float pos = fmaf(lg, row.scale, row.bias);
  pos = fminf(fmaxf(pos, row.lo), row.hi);        // NaN goes to the lower clamp, as in the expression
  const float big = __fadd_rd(pos, 12582912.0f);  // 1.5 * 2^23: the low mantissa bits are floor(pos)
  worst = fmaxf(worst, fabsf(pos - (big - 12582912.0f) - 0.5f));
  // level l: x > 0 stores l (+ DR when packed), else -1 - l (+ DR)
  return (__float_as_uint(big) ^ (x <= 0.0f ? MASK ^ DR : DR)) & MASK;
}

struct Args {
  const float* x;
  unsigned char* out;
  const float* codebooks;
  int64_t rows;
  int n_cb, dim, row_bytes, column_slice;
  int units;   // vector kernel: units of E columns per row (the last may be short)
};

// dim % 4 == 0, x 16-byte aligned, at most kThreads units per row.
template <int BITS>
__global__ void __launch_bounds__(kThreads, kCtasPerSm) encode_vec_kernel(const Args a) {
  dependency_wait();
  release_dependents();
  constexpr int E = BITS >= 8 ? 4 : 8;  // columns per thread and row
  constexpr int Q = E / 4;
  constexpr int F = BITS >= 8 ? 4 : 2;  // rows in flight per thread
  extern __shared__ float par[];
  build_params<BITS>(par, a.codebooks, a.n_cb);
  const int rows_per_cta = kThreads / a.units;
  const int local = (int)threadIdx.x / a.units, c0 = ((int)threadIdx.x - local * a.units) * E;
  if (local >= rows_per_cta) return;
  const bool second = Q == 2 && c0 + 4 < a.dim;  // the row's last unit may be half a unit
  // codebook rows of the two groups of four columns (each group inside one row, or `mixed`)
  const int cb_lo = c0 / a.column_slice, cb_hi = min(c0 + E, a.dim) - 1;
  const bool mixed = cb_hi / a.column_slice != cb_lo;
  const Row prow = (BITS == 1 || BITS == 16) ? Row{} : row_of(par + cb_lo * kParams);
  const float* cb = a.codebooks + cb_lo * kCodebookDim;
  const int64_t step = (int64_t)gridDim.x * rows_per_cta;
  auto emit = [&](const float4 (&v)[Q], int64_t row) {
    float e[E];
#pragma unroll
    for (int q = 0; q < Q; ++q) { e[4 * q] = v[q].x; e[4 * q + 1] = v[q].y; e[4 * q + 2] = v[q].z; e[4 * q + 3] = v[q].w; }
    uint32_t code[E];
    float worst = 0.0f;
    if (!mixed) {
#pragma unroll
      for (int i = 0; i < E; ++i) code[i] = encode_fast<BITS>(e[i], prow, cb, worst);
    }
    if (mixed || (BITS != 1 && BITS != 16 && worst >= prow.limit)) {
#pragma unroll
      for (int i = 0; i < E; ++i) {
        const int r = min(c0 + i, a.dim - 1) / a.column_slice;
        code[i] = encode_exact<BITS>(e[i], a.codebooks + r * kCodebookDim);
      }
    }
    unsigned char* o = a.out + row * a.row_bytes;
    if (BITS == 16) {
      const uint32_t w0 = (code[0] & 0xffffu) | (code[1] << 16), w1 = (code[2] & 0xffffu) | (code[3] << 16);
      *reinterpret_cast<uint2*>(o + 2 * c0) = make_uint2(w0, w1);
    } else if (BITS == 8) {
      *reinterpret_cast<uint32_t*>(o + c0) = (code[0] & 0xffu) | ((code[1] & 0xffu) << 8) |
                                             ((code[2] & 0xffu) << 16) | (code[3] << 24);
    } else {
      constexpr int B = BITS >= 8 ? 1 : BITS;
      uint32_t w = 0;
#pragma unroll
      for (int i = 0; i < E; ++i)
        if (i < 4 || second) w |= (code[i] & ((1u << B) - 1u)) << (B * i);
      o += c0 * B / 8;
      if (B == 4) {  // row_bytes is even
        if (second && (a.row_bytes & 3) == 0) {
          *reinterpret_cast<uint32_t*>(o) = w;
        } else {
          *reinterpret_cast<uint16_t*>(o) = (uint16_t)w;
          if (second) *reinterpret_cast<uint16_t*>(o + 2) = (uint16_t)(w >> 16);
        }
      } else if (B == 2) {
        o[0] = (unsigned char)w;
        if (second) o[1] = (unsigned char)(w >> 8);
      } else {
        o[0] = (unsigned char)w;
      }
    }
  };
  for (int64_t row = (int64_t)blockIdx.x * rows_per_cta + local; row < a.rows; row += F * step) {
    float4 v[F][Q];
#pragma unroll
    for (int f = 0; f < F; ++f) {
      const int64_t r = row + f * step;
      const float4* src = reinterpret_cast<const float4*>(a.x + r * a.dim + c0);
#pragma unroll
      for (int q = 0; q < Q; ++q)
        v[f][q] = (r < a.rows && (q == 0 || second)) ? __ldcs(src + q) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int f = 0; f < F; ++f)
      if (row + f * step < a.rows) emit(v[f], row + f * step);
  }
}

// Codes of 4, 8 or 16 bits in rows that are no multiple of four columns but follow each other without a gap (4 bits: an even
// number of columns): two or four rows make a super-row of whole 16-byte groups of features, whose four codes are one aligned
// store.  A thread keeps its group - four columns with their codebook rows - for its whole life and walks over super-rows, two
// in flight (rows through shared memory in tiles: 500,001 x 117 8-bit codes 154 us, now 114; 16-bit 219, now 154;
// 100,000 x 110 8-bit 45, now 16.  One branch for a group of four instead of one per column: 8 bits 130).
constexpr int kGroupThreads = 512;

template <int BITS>
__global__ void __launch_bounds__(kGroupThreads, 2) encode_groups_kernel(const Args a, int rows_per_super, int groups, int part, int supers_per_cta) {
  dependency_wait();
  release_dependents();
  extern __shared__ float par[];
  build_params<BITS>(par, a.codebooks, a.n_cb);
  const int sub = (int)threadIdx.x / part, group = (int)blockIdx.y * part + ((int)threadIdx.x - sub * part);
  if (sub >= supers_per_cta || group >= groups) return;
  int row_of_column[4], book[4];
  Row prow[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    row_of_column[e] = (4 * group + e) / a.dim;
    book[e] = (4 * group + e - row_of_column[e] * a.dim) / a.column_slice;
    prow[e] = BITS == 16 ? Row{} : row_of(par + book[e] * kParams);
  }
  auto codes_of = [&](float4 x, uint32_t (&c)[4]) {
    const float v[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float* cb = a.codebooks + book[e] * kCodebookDim;
      float worst = 0.0f;
      c[e] = encode_fast<BITS>(v[e], prow[e], cb, worst);
      if (BITS != 16 && worst >= prow[e].limit) c[e] = encode_exact<BITS>(v[e], cb);
      c[e] &= (1u << BITS) - 1u;
    }
  };
  const int64_t step = (int64_t)gridDim.x * supers_per_cta, full = a.rows / rows_per_super;
  const int64_t super = (int64_t)rows_per_super * a.dim;  // columns
  int64_t s = (int64_t)blockIdx.x * supers_per_cta + sub;
  constexpr int F = 2;  // super-rows in flight
  for (; s < full; s += F * step) {
    float4 x[F];
#pragma unroll
    for (int f = 0; f < F; ++f)
      x[f] = s + f * step < full ? __ldcs(reinterpret_cast<const float4*>(a.x + (s + f * step) * super) + group) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int f = 0; f < F; ++f) {
      if (s + f * step >= full) break;
      uint32_t c[4];
      codes_of(x[f], c);
      unsigned char* o = a.out + ((s + f * step) * super + 4 * group) * BITS / 8;
      if (BITS == 16) *reinterpret_cast<uint2*>(o) = make_uint2(c[0] | (c[1] << 16), c[2] | (c[3] << 16));
      else if (BITS == 8) *reinterpret_cast<uint32_t*>(o) = c[0] | (c[1] << 8) | (c[2] << 16) | (c[3] << 24);
      else *reinterpret_cast<uint16_t*>(o) = (uint16_t)(c[0] | (c[1] << 4) | (c[2] << 8) | (c[3] << 12));
    }
  }
  // the rows behind the full super-rows: one thread per group of the super-row that they begin
  const int rest = (int)(a.rows - full * rows_per_super);
  if (rest == 0 || blockIdx.x != 0 || sub != 0) return;
  int live = 0;
#pragma unroll
  for (int e = 0; e < 4; ++e) live += row_of_column[e] < rest ? 1 : 0;
  if (live == 0) return;
  const float* q = a.x + full * super + 4 * group;
  uint32_t c[4];
  codes_of(make_float4(q[0], live > 1 ? q[1] : 0.f, live > 2 ? q[2] : 0.f, live > 3 ? q[3] : 0.f), c);
  unsigned char* o = a.out + (full * super + 4 * group) * BITS / 8;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    if (e >= live) break;
    if (BITS == 16) reinterpret_cast<uint16_t*>(o)[e] = (uint16_t)c[e];
    else if (BITS == 8) o[e] = (unsigned char)c[e];
    else if (e % 2 == 1) o[e / 2] = (unsigned char)(c[e - (e > 0)] | (c[e] << 4));  // an even number is live
  }
}

// Any row length up to kTileFloats / 4: tiles of `tile_rows` rows (a multiple of 4, so that a tile starts on a 16-byte boundary
// of an aligned matrix) are copied to shared memory, encoded byte by byte into a second tile, and copied out.
constexpr int kTileFloats = 6144;

template <int BITS>
__global__ void __launch_bounds__(kThreads) encode_tile_kernel(const Args a, int tile_rows, int aligned_in) {
  dependency_wait();
  release_dependents();
  constexpr int B = BITS >= 8 ? 8 : BITS;
  constexpr int PER = 8 / B;           // elements per stored byte (16 bits: per stored pair of bytes)
  extern __shared__ __align__(16) float tile_smem[];
  float* tile = tile_smem;
  unsigned char* packed = reinterpret_cast<unsigned char*>(tile + tile_rows * a.dim);
  float* par = reinterpret_cast<float*>(packed + (((size_t)tile_rows * a.row_bytes + 15) & ~(size_t)15));
  build_params<BITS>(par, a.codebooks, a.n_cb);
  const Row first = (BITS == 1 || BITS == 16) ? Row{} : row_of(par);
  const int units = BITS == 16 ? a.dim : a.row_bytes;  // stored items per row
  const int64_t tiles = (a.rows + tile_rows - 1) / tile_rows;
  for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    const int64_t row0 = t * tile_rows;
    const int live = (int)min((int64_t)tile_rows, a.rows - row0);
    const int n = live * a.dim;
    const float* src = a.x + row0 * a.dim;
    if (aligned_in) {
      for (int i = threadIdx.x; i < n / 4; i += kThreads) reinterpret_cast<float4*>(tile)[i] = __ldcs(reinterpret_cast<const float4*>(src) + i);
      for (int i = n / 4 * 4 + (int)threadIdx.x; i < n; i += kThreads) tile[i] = __ldcs(src + i);
    } else {
      for (int i = threadIdx.x; i < n; i += kThreads) tile[i] = __ldcs(src + i);
    }
    __syncthreads();
    const int items = live * units;
    int r = (int)threadIdx.x / units, b = (int)threadIdx.x - r * units;
    const int dr = kThreads / units, db = kThreads - dr * units;
    for (int i = threadIdx.x; i < items; i += kThreads) {
      const int col = b * PER;
      uint32_t w = 0;
#pragma unroll
      for (int e = 0; e < PER; ++e) {
        if (col + e < a.dim) {
          const int row = a.n_cb == 1 ? 0 : (col + e) / a.column_slice;
          const float* cb = a.codebooks + row * kCodebookDim;
          const float v = tile[r * a.dim + col + e];
          const Row prow = (BITS == 1 || BITS == 16) ? Row{} : a.n_cb == 1 ? first : row_of(par + row * kParams);
          float worst = 0.0f;
          uint32_t code = encode_fast<BITS>(v, prow, cb, worst);
          if (BITS != 1 && BITS != 16 && worst >= prow.limit) code = encode_exact<BITS>(v, cb);
          w |= (code & (BITS == 16 ? 0xffffu : (1u << B) - 1u)) << (B * e);
        }
      }
      if (BITS == 16) reinterpret_cast<uint16_t*>(packed)[i] = (uint16_t)w; else packed[i] = (unsigned char)w;
      r += dr; b += db;
      if (b >= units) { b -= units; ++r; }
    }
    __syncthreads();
    const int bytes = live * a.row_bytes;
    unsigned char* dst = a.out + row0 * a.row_bytes;  // a multiple of 4 bytes from `out`
    for (int i = threadIdx.x; i < bytes / 4; i += kThreads) reinterpret_cast<uint32_t*>(dst)[i] = reinterpret_cast<const uint32_t*>(packed)[i];
    for (int i = bytes / 4 * 4 + (int)threadIdx.x; i < bytes; i += kThreads) dst[i] = packed[i];
    __syncthreads();
  }
}

template <int BITS>
static int launch_encode(Args a, cudaStream_t st, const char* op) {
  constexpr int E = BITS >= 8 ? 4 : 8;
  a.units = (a.dim + E - 1) / E;
  const size_t par_bytes = (BITS == 1 || BITS == 16) ? 16 : (size_t)a.n_cb * kParams * 4;
  if (a.dim % 4 == 0 && aligned(a.x, 16) && aligned(a.out, 8) && a.units <= kThreads) {
    auto kern = encode_vec_kernel<BITS>;
    int64_t grid = ceil_div(a.rows, kThreads / a.units);
    const int64_t cap = kCtasPerSm * (int64_t)current_sm_count();
    if (grid > cap) grid = cap;
    launch_dependent(kern, (unsigned)grid, kThreads, par_bytes, st, a);
    return check_launch(op);
  }
  if constexpr (BITS == 4 || BITS == 8 || BITS == 16) {
    if (a.dim * BITS % 8 == 0 && aligned(a.x, 16) && aligned(a.out, BITS / 2)) {
      const int per = a.dim % 4 == 0 ? 1 : a.dim % 2 == 0 ? 2 : 4;
      const int64_t groups = (int64_t)a.dim * per / 4, supers = ceil_div(a.rows, per);
      const int sms = current_sm_count();
      const Lanes ln = lanes_of_rows(groups, supers, sms, kGroupThreads);
      const int64_t grid = std::min(ceil_div(supers, ln.rows_per_cta), ceil_div((int64_t)sms * 2 * kGroupThreads / ln.threads, ln.parts));
      launch_dependent(encode_groups_kernel<BITS>, dim3((unsigned)grid, (unsigned)ln.parts), ln.threads, par_bytes, st, a, per, (int)groups,
                       ln.part, ln.rows_per_cta);
      return check_launch(op);
    }
  }
  F2C_REQUIRE(aligned(a.out, 4), F2C_ERR_INVALID, "%s: the codes must be 4-byte aligned", op);
  int tile_rows = kTileFloats / a.dim / 4 * 4;
  if (tile_rows > 256) tile_rows = 256;
  const size_t smem = (size_t)tile_rows * a.dim * 4 + (((size_t)tile_rows * a.row_bytes + 15) & ~(size_t)15) + par_bytes;
  auto kern = encode_tile_kernel<BITS>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return set_error(F2C_ERR_CUDA, "%s: %s", op, cudaGetErrorString(e));
  }
  int64_t grid = ceil_div(a.rows, tile_rows);
  const int64_t cap = 5 * (int64_t)current_sm_count();
  if (grid > cap) grid = cap;
  launch_dependent(kern, (unsigned)grid, kThreads, smem, st, a, tile_rows, aligned(a.x, 16) ? 1 : 0);
  return check_launch(op);
}

}  // namespace enc
}  // namespace f2c

using namespace f2c;

extern "C" int f2c_sq_encode(const float* x, void* codes, const float* codebooks, int64_t n_codebooks, int64_t rows, int64_t feat_dim,
                             int bits, int64_t column_slice, void* stream) {
  const char* op = "sq_encode";
  F2C_REQUIRE(rows >= 0 && feat_dim >= 0, F2C_ERR_INVALID, "%s: negative size", op);
  F2C_REQUIRE(is_sq_bits(bits), F2C_ERR_UNSUPPORTED, "%s: target_bits must be 1, 2, 4, 8 or 16 (got %d)", op, bits);
  F2C_REQUIRE(column_slice >= 1 && column_slice < (1ll << 31) && feat_dim < (1ll << 24), F2C_ERR_LIMIT, "%s: bad column_slice / feat_dim", op);
  F2C_REQUIRE(n_codebooks * column_slice >= feat_dim, F2C_ERR_INVALID, "%s: %lld codebook rows of %lld columns do not cover feat_dim %lld",
              op, (long long)n_codebooks, (long long)column_slice, (long long)feat_dim);
  F2C_REQUIRE(feat_dim <= 1024, F2C_ERR_LIMIT, "%s: at most 1024 columns", op);
  if (rows * feat_dim == 0) return F2C_OK;
  F2C_REQUIRE(x && codes && codebooks, F2C_ERR_INVALID, "%s: null pointer", op);
  enc::Args a{};
  a.x = x; a.out = (unsigned char*)codes; a.codebooks = codebooks; a.rows = rows;
  a.n_cb = (int)ceil_div(feat_dim, column_slice);  // rows behind the last column are not looked at
  F2C_REQUIRE(a.n_cb <= enc::kMaxBooks, F2C_ERR_LIMIT, "%s: at most %d codebook rows", op, enc::kMaxBooks);
  a.dim = (int)feat_dim; a.column_slice = (int)column_slice;
  a.row_bytes = (int)(bits == 16 ? 2 * feat_dim : ceil_div(feat_dim * bits, 8));
  cudaStream_t st = (cudaStream_t)stream;
  switch (bits) {
    case 1: return enc::launch_encode<1>(a, st, op);
    case 2: return enc::launch_encode<2>(a, st, op);
    case 4: return enc::launch_encode<4>(a, st, op);
    case 8: return enc::launch_encode<8>(a, st, op);
    default: return enc::launch_encode<16>(a, st, op);
  }
}
