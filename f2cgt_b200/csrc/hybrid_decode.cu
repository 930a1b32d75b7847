// Two-level decode in one launch: out = cat(sq_decompress(sq rows), vq_decompress(vq rows)).
// This is the operator `fusion_decompress` that the reference's tests/test_fusion_decompress.py:40-43
// calls and pins to that concatenation; the reference's src/ no longer contains it.  It produces the
// h_self matrix of a two-level minibatch (examples/compress.py:74-106: SQ seed rows first, then the
// level-2 rows of the remaining destination nodes).
//
// Streaming kernel bound by the fp32 output; one thread per float4 of the output, the row index
// selects the codec.  Shapes that cannot take the vector path are served by the two standalone
// decoders back to back, which is the definition of the operator.
#include "common.cuh"

namespace f2c {

int validate_vq(const char* op, int code_dtype, int64_t n_cb, int64_t length, int64_t cs, int64_t feat_dim);
int validate_sq(const char* op, int code_dtype, int64_t n_codebooks, int64_t src_dim, int64_t feat_dim, int bits,
                int64_t column_slice);

struct HybridDecodeParams {
  const uint8_t* sq_codes; const float* sq_cb; int64_t sq_rows, sq_row_bytes; int sq_cs, sq_n_cb, sq_signed;
  const void* vq_codes; const float* vq_cb; int64_t vq_rows; int vq_kind, vq_n_cb, vq_cs; uint32_t K;
  float* out; int feat_dim;
};

template <int BITS>
__global__ void __launch_bounds__(256) hybrid_decode_kernel(const HybridDecodeParams p) {
  dependency_wait();
  release_dependents();
  const int vec_per_row = p.feat_dim / 4;
  const int64_t n_vec = (p.sq_rows + p.vq_rows) * vec_per_row;
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_vec) return;
  const int64_t row = i / vec_per_row;
  const int col = (int)(i % vec_per_row) * 4;
  float4 v;
  if (row < p.sq_rows) {
    int cb_row = col / p.sq_cs;
    if (cb_row >= p.sq_n_cb) cb_row = p.sq_n_cb - 1;
    const float emin = __ldg(p.sq_cb + cb_row * kCodebookDim + 2), emax = __ldg(p.sq_cb + cb_row * kCodebookDim + 3);
    const float mean = __ldg(p.sq_cb + cb_row * kCodebookDim + 4);
    const float scale = sq_scale<BITS>(emin, emax);
    const uint8_t* r = p.sq_codes + row * p.sq_row_bytes;
    float c[4];
    if (BITS == 16) {
      uint2 raw = *reinterpret_cast<const uint2*>(r + 2 * col);
      c[0] = (float)(int16_t)(raw.x & 0xFFFFu); c[1] = (float)(int16_t)(raw.x >> 16);
      c[2] = (float)(int16_t)(raw.y & 0xFFFFu); c[3] = (float)(int16_t)(raw.y >> 16);
    } else if (BITS == 8) {
      uint32_t raw = *reinterpret_cast<const uint32_t*>(r + col);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        uint32_t b = (raw >> (8 * e)) & 0xFFu;
        c[e] = p.sq_signed ? (float)(int8_t)b : (float)b;
      }
    } else {
      constexpr int B = BITS >= 8 ? 4 : BITS;
      uint32_t raw;
      if (B == 4) raw = *reinterpret_cast<const uint16_t*>(r + col / 2);
      else if (B == 2) raw = r[col / 4];
      else raw = (uint32_t)r[col / 8] >> (col & 7);
#pragma unroll
      for (int e = 0; e < 4; ++e) c[e] = (float)((raw >> (B * e)) & ((1u << B) - 1u));
    }
    v = make_float4(sq_decode<BITS>(c[0], scale, emin, mean), sq_decode<BITS>(c[1], scale, emin, mean),
                    sq_decode<BITS>(c[2], scale, emin, mean), sq_decode<BITS>(c[3], scale, emin, mean));
  } else {
    const int64_t vr = row - p.sq_rows;
    const int s = col / p.vq_cs, off = col - s * p.vq_cs;
    int code;
    const int64_t pos = vr * p.vq_n_cb + s;
    if (p.vq_kind == 0) code = reinterpret_cast<const uint8_t*>(p.vq_codes)[pos];
    else if (p.vq_kind == 1) code = reinterpret_cast<const int8_t*>(p.vq_codes)[pos];
    else code = reinterpret_cast<const int16_t*>(p.vq_codes)[pos];
    uint32_t u = (uint32_t)code < p.K ? (uint32_t)code : p.K - 1;
    v = __ldg(reinterpret_cast<const float4*>(p.vq_cb + ((int64_t)s * p.K + u) * p.vq_cs + off));
  }
  stg_cs_f4(p.out + row * p.feat_dim + col, v);
}

}  // namespace f2c

using namespace f2c;

extern "C" int f2c_hybrid_decompress(const void* sq_codes, int sq_dtype, const float* sq_codebooks, int64_t sq_n_codebooks,
                                     int bits, int64_t sq_column_slice, int64_t sq_rows, int64_t sq_src_dim,
                                     const void* vq_codes, int vq_dtype, const float* vq_codebooks, int64_t vq_rows,
                                     int64_t vq_n_codebooks, int64_t length, int64_t vq_column_slice, float* out,
                                     int64_t feat_dim, void* stream) {
  const char* op = "fusion_decompress";
  F2C_REQUIRE(sq_rows >= 0 && vq_rows >= 0, F2C_ERR_INVALID, "%s: negative size", op);
  int rc = validate_sq(op, sq_dtype, sq_n_codebooks, sq_src_dim, feat_dim, bits, sq_column_slice);
  if (rc) return rc;
  rc = validate_vq(op, vq_dtype, vq_n_codebooks, length, vq_column_slice, feat_dim);
  if (rc) return rc;
  if ((sq_rows + vq_rows) * feat_dim == 0) return F2C_OK;
  F2C_REQUIRE(out && (sq_rows == 0 || (sq_codes && sq_codebooks)) && (vq_rows == 0 || (vq_codes && vq_codebooks)),
              F2C_ERR_INVALID, "%s: null pointer", op);
  const int sq_bytes = dtype_size(sq_dtype);
  const int64_t sq_row_bytes = sq_src_dim * sq_bytes;
  const int row_align = bits == 16 ? 8 : bits == 8 ? 4 : bits == 4 ? 2 : 1;
  bool vec = feat_dim % 4 == 0 && vq_column_slice % 4 == 0 && (sq_n_codebooks == 1 || sq_column_slice % 4 == 0) &&
             (bits == 16) == (sq_bytes == 2) && sq_row_bytes % row_align == 0 && aligned(sq_codes, row_align) &&
             aligned(vq_codebooks, 16) && aligned(out, 16);
  if (!vec) {  // the definition: two decoders, one after the other, on the same stream
    rc = f2c_sq_decompress(sq_codes, sq_dtype, sq_codebooks, sq_n_codebooks, out, sq_rows, sq_src_dim, feat_dim, bits,
                           sq_column_slice, stream);
    if (rc) return rc;
    return f2c_vq_decompress(vq_codes, vq_dtype, vq_codebooks, F2C_F32, out + sq_rows * feat_dim, vq_rows,
                             vq_n_codebooks, length, vq_column_slice, feat_dim, stream);
  }
  HybridDecodeParams p{};
  p.sq_codes = (const uint8_t*)sq_codes; p.sq_cb = sq_codebooks; p.sq_rows = sq_rows; p.sq_row_bytes = sq_row_bytes;
  p.sq_cs = (int)sq_column_slice; p.sq_n_cb = (int)sq_n_codebooks; p.sq_signed = sq_dtype == F2C_I8;
  p.vq_codes = vq_codes; p.vq_cb = vq_codebooks; p.vq_rows = vq_rows; p.vq_kind = vq_dtype == F2C_U8 ? 0 : vq_dtype == F2C_I8 ? 1 : 2;
  p.vq_n_cb = (int)vq_n_codebooks; p.vq_cs = (int)vq_column_slice; p.K = (uint32_t)length; p.out = out; p.feat_dim = (int)feat_dim;
  int64_t n_vec = (sq_rows + vq_rows) * (feat_dim / 4);
  unsigned grid = (unsigned)ceil_div(n_vec, 256);
  cudaStream_t st = (cudaStream_t)stream;
  switch (bits) {
    case 1: launch_dependent(hybrid_decode_kernel<1>, grid, 256, 0, st, p); break;
    case 2: launch_dependent(hybrid_decode_kernel<2>, grid, 256, 0, st, p); break;
    case 4: launch_dependent(hybrid_decode_kernel<4>, grid, 256, 0, st, p); break;
    case 8: launch_dependent(hybrid_decode_kernel<8>, grid, 256, 0, st, p); break;
    default: launch_dependent(hybrid_decode_kernel<16>, grid, 256, 0, st, p); break;
  }
  return check_launch(op);
}
