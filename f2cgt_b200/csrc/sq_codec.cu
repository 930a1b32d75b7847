// Scalar quantisation: log2-domain sign-magnitude codes of 1/2/4/8/16 bits
// (reference operators sq_compress / sq_decompress, src/sq_quantization.cu).
//
// Both are streaming element-wise kernels bound by HBM: compress moves 8 B per element
// (fp32 in, fp32-valued code out), decompress bits/8 + 4 B per element.  The arithmetic is the reference's expression compiled with
// the same math flags, so codes and decoded values carry the reference kernel's bits.
#include <algorithm>

#include "row_lanes.cuh"
#include "sq_encode.cuh"

namespace f2c {

// ---------------------------------------------------------------- compress
template <int BITS>
__global__ void __launch_bounds__(256) sq_compress_vec_kernel(const float4* __restrict__ src, float4* __restrict__ dst,
                                                              const float* __restrict__ codebooks, int64_t n_vec,
                                                              int vec_per_row, int column_slice) {
  dependency_wait();
  release_dependents();
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_vec) return;
  int c0 = (int)(i % vec_per_row) * 4;
  float4 x = src[i], y;
  y.x = sq_encode<BITS>(x.x, codebooks + (c0 + 0) / column_slice * kCodebookDim);
  y.y = sq_encode<BITS>(x.y, codebooks + (c0 + 1) / column_slice * kCodebookDim);
  y.z = sq_encode<BITS>(x.z, codebooks + (c0 + 2) / column_slice * kCodebookDim);
  y.w = sq_encode<BITS>(x.w, codebooks + (c0 + 3) / column_slice * kCodebookDim);
  dst[i] = y;
}

template <int BITS>
__global__ void __launch_bounds__(256) sq_compress_scalar_kernel(const float* __restrict__ src, float* __restrict__ dst,
                                                                 const float* __restrict__ codebooks, int64_t numel,
                                                                 int feat_dim, int column_slice) {
  dependency_wait();
  release_dependents();
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= numel) return;
  int c = (int)(i % feat_dim);
  dst[i] = sq_encode<BITS>(src[i], codebooks + c / column_slice * kCodebookDim);
}

template <int BITS>
static int launch_compress(const float* src, float* dst, const float* cb, int64_t rows, int64_t D, int64_t cs,
                           cudaStream_t st) {
  int64_t numel = rows * D;
  if (numel == 0) return F2C_OK;
  if (D % 4 == 0 && aligned(src, 16) && aligned(dst, 16)) {
    int64_t n_vec = numel / 4;
    launch_dependent(sq_compress_vec_kernel<BITS>, (unsigned)ceil_div(n_vec, 256), 256, 0, st, 
        (const float4*)src, (float4*)dst, cb, n_vec, (int)(D / 4), (int)cs);
  } else {
    launch_dependent(sq_compress_scalar_kernel<BITS>, (unsigned)ceil_div(numel, 256), 256, 0, st, src, dst, cb, numel, (int)D, (int)cs);
  }
  return check_launch("sq_compress");
}

// ---------------------------------------------------------------- decompress
// A thread keeps EPT neighbouring columns for its whole life (a CTA holds as many whole rows of columns as fit, the threads left
// over end), so where its code lies in a row, its shift in the byte and its codebook row are found once, the next row is an add
// away and any row width costs the same; eight rows are in flight per thread.  EPT is 4 (one load, one 16-byte store) where rows,
// slices and addresses allow it, else 1.
// Bound by HBM: bits/8 + 4 B per element.  One exp2f per element hides behind that; a table of decoded values in shared memory
// was never faster (27,000 x 128 8-bit codes 6.0 us with one, 4.2 without).  Row widths that are no multiple of 4 columns took one
// thread and two 64-bit divisions per element before: 200,000 x 357 4-bit codes 288 us, now 77; x 101 8-bit 78, now 18
// (by groups, below); x 201 1-bit 142, now 32.
constexpr int kSqDecThreads = 512;

template <int BITS, typename CodeT, int EPT>
__global__ void __launch_bounds__(kSqDecThreads, 3) sq_decompress_kernel(
    const void* __restrict__ codes, float* __restrict__ out, const float* __restrict__ codebooks, int64_t rows, int64_t row_bytes,
    int feat_dim, int chunks, int part, int rows_per_cta, int column_slice, int n_cb) {
  dependency_wait();
  release_dependents();
  constexpr int B = BITS >= 8 ? 8 * (int)sizeof(CodeT) : BITS;  // stored bits of a code
  constexpr uint32_t MASK = (1u << B) - 1u;
  const int sub = threadIdx.x / part;
  const int chunk = blockIdx.y * part + (threadIdx.x - sub * part);
  if (sub >= rows_per_cta || chunk >= chunks) return;
  const int c0 = chunk * EPT;
  int cb_row = c0 / column_slice;
  if (cb_row >= n_cb) cb_row = n_cb - 1;
  const float* cb = codebooks + (int64_t)cb_row * kCodebookDim;
  const float emin = __ldg(cb + 2), scale = sq_scale<BITS>(emin, __ldg(cb + 3)), mean = __ldg(cb + 4);
  const int64_t bit0 = (int64_t)c0 * B;
  const int shift = (int)(bit0 & 7);
  const int64_t step = (int64_t)gridDim.x * rows_per_cta;
  int64_t row = (int64_t)blockIdx.x * rows_per_cta + sub;
  const uint8_t* cp = reinterpret_cast<const uint8_t*>(codes) + row * row_bytes + (bit0 >> 3);
  float* op = out + row * feat_dim + c0;
  const int64_t cstep = step * row_bytes, ostep = step * feat_dim;
  auto fetch = [&](const uint8_t* q) -> uint2 {
    constexpr int BYTES = EPT * B >= 8 ? EPT * B / 8 : 1;
    if (BYTES == 8) return *reinterpret_cast<const uint2*>(q);
    if (BYTES == 4) return make_uint2(*reinterpret_cast<const uint32_t*>(q), 0u);
    if (BYTES == 2) return make_uint2(*reinterpret_cast<const uint16_t*>(q), 0u);
    return make_uint2((uint32_t)*q >> (EPT * B < 8 ? shift : 0), 0u);
  };
  auto emit = [&](uint2 raw, float* o) {
    float v[EPT];
#pragma unroll
    for (int e = 0; e < EPT; ++e) {
      const uint32_t code = ((B * e >= 32 ? raw.y : raw.x) >> ((B * e) & 31)) & MASK;
      v[e] = sq_decode<BITS>(BITS >= 8 ? (float)(CodeT)code : (float)code, scale, emin, mean);
    }
    if constexpr (EPT == 4) stg_cs_f4(o, make_float4(v[0], v[1], v[2], v[3]));
    else __stcs(o, v[0]);
  };
  constexpr int kInFlight = 8;  // rows in flight per thread
  for (; row + (kInFlight - 1) * step < rows; row += kInFlight * step, cp += kInFlight * cstep, op += kInFlight * ostep) {
    uint2 raw[kInFlight];
#pragma unroll
    for (int u = 0; u < kInFlight; ++u) raw[u] = fetch(cp + u * cstep);
#pragma unroll
    for (int u = 0; u < kInFlight; ++u) emit(raw[u], op + u * ostep);
  }
  uint2 raw[kInFlight];
#pragma unroll
  for (int u = 0; u < kInFlight - 1; ++u)
    if (row + u * step < rows) raw[u] = fetch(cp + u * cstep);
#pragma unroll
  for (int u = 0; u < kInFlight - 1; ++u)
    if (row + u * step < rows) emit(raw[u], op + u * ostep);
}

// Rows that are no multiple of four columns (or whose slices or codes forbid one load for four): two or four of them make a
// super-row of whole 16-byte groups, and a thread keeps one group of it for its whole life - four columns with their own row,
// code position and codebook row, found once.  Stores are whole and aligned whatever the width; a warp of single columns starts
// its 128 bytes anywhere, which is two partly written sectors per store.
//   ONE   the rows' codes follow each other without a gap, so that a group's codes are one aligned load; else four loads
// 200,000 x 101 8-bit codes 24.4 us by columns, 18.4 by groups; x 110 8-bit 33.2, 21.1; x 255 16-bit 68, 58; x 399 8-bit 118, 94.
template <int BITS, typename CodeT, bool ONE>
__global__ void __launch_bounds__(kSqDecThreads, 2) sq_decompress_groups_kernel(
    const uint8_t* __restrict__ codes, float* __restrict__ out, const float* __restrict__ codebooks, int64_t rows, int64_t row_bytes,
    int feat_dim, int rows_per_super, int groups, int part, int supers_per_cta, int column_slice, int n_cb) {
  dependency_wait();
  release_dependents();
  constexpr int B = BITS >= 8 ? 8 * (int)sizeof(CodeT) : BITS;  // stored bits of a code
  constexpr uint32_t MASK = (1u << B) - 1u;
  constexpr int LOADS = ONE ? 1 : 4;
  const int sub = threadIdx.x / part;
  const int group = blockIdx.y * part + (threadIdx.x - sub * part);
  if (sub >= supers_per_cta || group >= groups) return;
  int row_of[4], shift[4];
  int64_t at[4];
  float emin[4], scale[4], mean[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int f = 4 * group + e;
    row_of[e] = f / feat_dim;
    const int c = f - row_of[e] * feat_dim;
    at[e] = row_of[e] * row_bytes + (((int64_t)c * B) >> 3);
    shift[e] = (c * B) & 7;
    int cb_row = c / column_slice;
    if (cb_row >= n_cb) cb_row = n_cb - 1;
    const float* cb = codebooks + (int64_t)cb_row * kCodebookDim;
    emin[e] = __ldg(cb + 2);
    scale[e] = sq_scale<BITS>(emin[e], __ldg(cb + 3));
    mean[e] = __ldg(cb + 4);
  }
  struct Raw { uint32_t w[ONE ? 2 : 4]; };
  auto fetch = [&](const uint8_t* super, int live, Raw& r) {  // the first `live` columns of the group exist
    if constexpr (ONE) {
      constexpr int BYTES = 4 * B / 8 > 0 ? 4 * B / 8 : 1;
      const uint8_t* q = super + at[0];
      if (live == 4) {
        if (BYTES == 8) { const uint2 v = *reinterpret_cast<const uint2*>(q); r.w[0] = v.x; r.w[1] = v.y; }
        else if (BYTES == 4) r.w[0] = *reinterpret_cast<const uint32_t*>(q);
        else if (BYTES == 2) r.w[0] = *reinterpret_cast<const uint16_t*>(q);
        else r.w[0] = *q;
      } else {
        r.w[0] = r.w[1] = 0u;
#pragma unroll
        for (int b = 0; b < BYTES; ++b)
          if (8 * b < live * B) r.w[b / 4] |= (uint32_t)q[b] << (8 * (b % 4));
      }
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (e < live) r.w[e] = B == 16 ? (uint32_t)*reinterpret_cast<const uint16_t*>(super + at[e]) : (uint32_t)super[at[e]] >> shift[e];
    }
  };
  auto emit = [&](const Raw& r, float* o, int live) {
    float v[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const uint32_t code = (ONE ? (B * e >= 32 ? r.w[1] : r.w[0]) >> ((B * e) & 31) : r.w[ONE ? 0 : e]) & MASK;
      v[e] = sq_decode<BITS>(BITS >= 8 ? (float)(CodeT)code : (float)code, scale[e], emin[e], mean[e]);
    }
    if (live == 4) {
      stg_cs_f4(o, make_float4(v[0], v[1], v[2], v[3]));
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (e < live) o[e] = v[e];
    }
  };
  const int64_t step = (int64_t)gridDim.x * supers_per_cta, full = rows / rows_per_super;
  int64_t s = (int64_t)blockIdx.x * supers_per_cta + sub;
  const int64_t cstep = step * rows_per_super * row_bytes, ostep = step * rows_per_super * feat_dim;
  const uint8_t* cp = codes + s * rows_per_super * row_bytes;
  float* op = out + s * rows_per_super * feat_dim + 4 * group;
  constexpr int kInFlight = LOADS == 1 ? 8 : 4;  // super-rows in flight per thread
  for (; s + (kInFlight - 1) * step < full; s += kInFlight * step, cp += kInFlight * cstep, op += kInFlight * ostep) {
    Raw r[kInFlight];
#pragma unroll
    for (int u = 0; u < kInFlight; ++u) fetch(cp + u * cstep, 4, r[u]);
#pragma unroll
    for (int u = 0; u < kInFlight; ++u) emit(r[u], op + u * ostep, 4);
  }
  // what is left of the full super-rows, and the rows behind them
  Raw r[kInFlight];
  const int rest = (int)(rows - full * rows_per_super);
  int tail = 0;  // columns of the group that lie in those rows
#pragma unroll
  for (int e = 0; e < 4; ++e) tail += row_of[e] < rest ? 1 : 0;
#pragma unroll
  for (int u = 0; u < kInFlight; ++u) {
    const int live = s + u * step < full ? 4 : s + u * step == full ? tail : 0;
    if (live > 0) fetch(cp + u * cstep, live, r[u]);
  }
#pragma unroll
  for (int u = 0; u < kInFlight; ++u) {
    const int live = s + u * step < full ? 4 : s + u * step == full ? tail : 0;
    if (live > 0) emit(r[u], op + u * ostep, live);
  }
}

template <int BITS, typename CodeT>
static int launch_decompress_groups(const void* codes, float* out, const float* cb, int64_t rows, int64_t row_bytes, int64_t D, int64_t cs,
                                    cudaStream_t st, bool* served) {
  constexpr int B = BITS >= 8 ? 8 * (int)sizeof(CodeT) : BITS;
  const int per = D % 4 == 0 ? 1 : D % 2 == 0 ? 2 : 4;
  const int64_t groups = D * per / 4, supers = ceil_div(rows, per);
  const int sms = current_sm_count();
  const Lanes ln = lanes_of_rows(groups, supers, sms, kSqDecThreads);
  const int64_t grid = std::min(ceil_div(supers, ln.rows_per_cta), ceil_div((int64_t)sms * 2 * kSqDecThreads / ln.threads, ln.parts));
  const bool one = 4 * B % 8 == 0 && row_bytes * 8 == D * B && aligned(codes, 4 * B / 8 > 0 ? 4 * B / 8 : 1);
  // Fewer groups than columns means fewer threads, so it takes some work before whole stores pay: 27,000 x 101 8-bit codes 5.2 us
  // against 4.7 by columns, x 255 16-bit 7.8 against 8.4.  Four loads per group pay later and only for the narrowest codes
  // (200,000 x 357 4-bit codes 94 us against 77; x 333 2-bit 79 against 87; 27,000 x 201 1-bit 7.1 against 6.8).
  *served = aligned(out, 16) && rows * D >= (one ? 3 << 20 : 8 << 20) && (one || BITS <= 2);
  if (!*served) return F2C_OK;
  auto kern = one ? sq_decompress_groups_kernel<BITS, CodeT, true> : sq_decompress_groups_kernel<BITS, CodeT, BITS <= 2 ? false : true>;
  launch_dependent(kern, dim3((unsigned)grid, (unsigned)ln.parts), ln.threads, 0, st, (const uint8_t*)codes, out, cb, rows, row_bytes, (int)D, per,
                   (int)groups, ln.part, ln.rows_per_cta, (int)cs, (int)ceil_div(D, cs));
  return check_launch("sq_decompress");
}

template <int BITS, typename CodeT, int EPT>
static int launch_decompress_ept(const void* codes, float* out, const float* cb, int64_t rows, int64_t row_bytes, int64_t D, int64_t cs,
                                 cudaStream_t st) {
  const int64_t chunks = D / EPT;
  const int sms = current_sm_count();
  const Lanes ln = lanes_of_rows(chunks, rows, sms, kSqDecThreads);
  const int64_t grid = std::min(ceil_div(rows, ln.rows_per_cta), ceil_div((int64_t)sms * 3 * kSqDecThreads / ln.threads, ln.parts));
  launch_dependent(sq_decompress_kernel<BITS, CodeT, EPT>, dim3((unsigned)grid, (unsigned)ln.parts), ln.threads, 0, st, codes, out, cb, rows,
                   row_bytes, (int)D, (int)chunks, ln.part, ln.rows_per_cta, (int)cs, (int)ceil_div(D, cs));
  return check_launch("sq_decompress");
}

template <int BITS, typename CodeT>
static int launch_decompress(const void* codes, float* out, const float* cb, int64_t rows, int64_t src_dim, int64_t D,
                             int64_t cs, cudaStream_t st) {
  if (rows * D == 0) return F2C_OK;
  // bytes of four columns' codes and the alignment their single load needs
  constexpr int LOAD_BYTES = BITS >= 8 ? 4 * (int)sizeof(CodeT) : (BITS == 4 ? 2 : 1);
  const int64_t row_bytes = src_dim * (int64_t)sizeof(CodeT);
  const bool vec = D % 4 == 0 && aligned(out, 16) && aligned(codes, LOAD_BYTES) && row_bytes % LOAD_BYTES == 0 && (cs >= D || cs % 4 == 0);
  if (vec) return launch_decompress_ept<BITS, CodeT, 4>(codes, out, cb, rows, row_bytes, D, cs, st);
  bool served = false;
  const int rc = launch_decompress_groups<BITS, CodeT>(codes, out, cb, rows, row_bytes, D, cs, st, &served);
  if (served || rc) return rc;
  return launch_decompress_ept<BITS, CodeT, 1>(codes, out, cb, rows, row_bytes, D, cs, st);
}

}  // namespace f2c

using namespace f2c;

extern "C" int f2c_sq_compress(const float* src, float* dst, const float* codebooks, int64_t n_codebooks,
                               int64_t rows, int64_t feat_dim, int bits, int64_t column_slice, void* stream) {
  F2C_REQUIRE(rows >= 0 && feat_dim >= 0, F2C_ERR_INVALID, "sq_compress: negative size");
  F2C_REQUIRE(is_sq_bits(bits), F2C_ERR_UNSUPPORTED, "sq_compress: target_bits must be 1, 2, 4, 8 or 16 (got %d)", bits);
  F2C_REQUIRE(column_slice >= 1, F2C_ERR_INVALID, "sq_compress: column_slice must be >= 1");
  F2C_REQUIRE(feat_dim < (1ll << 31) && column_slice < (1ll << 31), F2C_ERR_LIMIT, "sq_compress: feat_dim too large");
  F2C_REQUIRE(n_codebooks * column_slice >= feat_dim, F2C_ERR_INVALID,
              "sq_compress: %lld codebook rows of %lld columns do not cover feat_dim %lld", (long long)n_codebooks,
              (long long)column_slice, (long long)feat_dim);
  F2C_REQUIRE(rows * feat_dim == 0 || (src && dst && codebooks), F2C_ERR_INVALID, "sq_compress: null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  switch (bits) {
    case 1: return launch_compress<1>(src, dst, codebooks, rows, feat_dim, column_slice, st);
    case 2: return launch_compress<2>(src, dst, codebooks, rows, feat_dim, column_slice, st);
    case 4: return launch_compress<4>(src, dst, codebooks, rows, feat_dim, column_slice, st);
    case 8: return launch_compress<8>(src, dst, codebooks, rows, feat_dim, column_slice, st);
    default: return launch_compress<16>(src, dst, codebooks, rows, feat_dim, column_slice, st);
  }
}

namespace f2c {
// Shared argument check of every SQ-decoding entry point.
int validate_sq(const char* op, int code_dtype, int64_t n_codebooks, int64_t src_dim, int64_t feat_dim, int bits,
                int64_t column_slice) {
  F2C_REQUIRE(is_sq_bits(bits), F2C_ERR_UNSUPPORTED, "%s: target_bits must be 1, 2, 4, 8 or 16 (got %d)", op, bits);
  F2C_REQUIRE(is_code_dtype(code_dtype), F2C_ERR_UNSUPPORTED, "%s: codes must be uint8, int8 or int16", op);
  F2C_REQUIRE(bits >= 8 || code_dtype != F2C_I16, F2C_ERR_UNSUPPORTED,
              "%s: packed %d-bit codes must be a uint8/int8 tensor", op, bits);
  F2C_REQUIRE(column_slice >= 1 && feat_dim >= 0 && src_dim >= 0, F2C_ERR_INVALID, "%s: bad column_slice/feat_dim", op);
  F2C_REQUIRE(feat_dim < (1ll << 24) && column_slice < (1ll << 31), F2C_ERR_LIMIT, "%s: feat_dim too large", op);
  int64_t capacity = bits >= 8 ? src_dim : src_dim * (8 / bits);
  F2C_REQUIRE(feat_dim <= capacity, F2C_ERR_INVALID, "%s: feat_dim %lld exceeds the %lld elements a code row holds", op,
              (long long)feat_dim, (long long)capacity);
  F2C_REQUIRE(n_codebooks * column_slice >= feat_dim, F2C_ERR_INVALID,
              "%s: %lld codebook rows of %lld columns do not cover feat_dim %lld", op, (long long)n_codebooks,
              (long long)column_slice, (long long)feat_dim);
  return F2C_OK;
}
}  // namespace f2c

extern "C" int f2c_sq_decompress(const void* codes, int code_dtype, const float* codebooks, int64_t n_codebooks,
                                 float* out, int64_t rows, int64_t src_dim, int64_t feat_dim, int bits,
                                 int64_t column_slice, void* stream) {
  F2C_REQUIRE(rows >= 0, F2C_ERR_INVALID, "sq_decompress: negative size");
  int rc = validate_sq("sq_decompress", code_dtype, n_codebooks, src_dim, feat_dim, bits, column_slice);
  if (rc) return rc;
  F2C_REQUIRE(rows * feat_dim == 0 || (codes && out && codebooks), F2C_ERR_INVALID, "sq_decompress: null pointer");
  cudaStream_t st = (cudaStream_t)stream;
#define F2C_DEC(B, T) return launch_decompress<B, T>(codes, out, codebooks, rows, src_dim, feat_dim, column_slice, st)
  if (bits < 8) {
    switch (bits) {
      case 1: F2C_DEC(1, uint8_t);
      case 2: F2C_DEC(2, uint8_t);
      default: F2C_DEC(4, uint8_t);
    }
  }
  if (bits == 8) {
    if (code_dtype == F2C_I8) F2C_DEC(8, int8_t);
    if (code_dtype == F2C_U8) F2C_DEC(8, uint8_t);
    F2C_DEC(8, int16_t);
  }
  if (code_dtype == F2C_I16) F2C_DEC(16, int16_t);
  if (code_dtype == F2C_I8) F2C_DEC(16, int8_t);
  F2C_DEC(16, uint8_t);
#undef F2C_DEC
}
