// Vector (product) quantisation decode: out[i, j] = codebooks[s][codes[i, s]][j - s*cs], s = j / cs
// (reference operator vq_decompress, src/vq_quantization.cu:5-60).
//
// A pure gather bound by the fp32 output stream (4 B per element against 1/cs code bytes); the
// codebooks (a few hundred KB) are read from shared memory or L2.  A code outside [0, length) cannot be told from a valid one
// by the reference (it reads out of bounds); here it is clamped to the last centroid so that a bad table cannot fault the device.
#include <algorithm>
#include <type_traits>

#include "row_lanes.cuh"
#include "vq_params.cuh"

namespace f2c {

__device__ __forceinline__ float4 load_cb4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float4 load_cb4(const __half* p) {
  uint2 raw = __ldg(reinterpret_cast<const uint2*>(p));
  __half2 a = *reinterpret_cast<__half2*>(&raw.x), b = *reinterpret_cast<__half2*>(&raw.y);
  float2 fa = __half22float2(a), fb = __half22float2(b);
  return make_float4(fa.x, fa.y, fb.x, fb.y);
}
__device__ __forceinline__ float load_cb1(const float* p) { return __ldg(p); }
__device__ __forceinline__ float load_cb1(const __half* p) { return __half2float(__ldg(p)); }

// A thread keeps EPT neighbouring columns for its whole life (a CTA holds as many whole rows of columns as fit), so its subspace
// and its offset in the centroid are found once, the next row is an add away and any row width costs the same; the codes of
// several rows are in flight per thread, and all their centroid pieces are asked for before the first is stored.
//   EPT     4 where a centroid is read and a row written in 16-byte pieces, else 1
//   STAGED  the codebooks of the CTA's columns lie in shared memory instead of L1 and L2.  Where those of a whole row do not fit,
//           the columns are cut into parts (grid.y) whose codebooks do.  Subspaces narrower than 32 columns (a power of two) are
//           interleaved inside 128-byte lines: lanes on neighbouring columns read different banks whatever the codes.
// Row widths that are no multiple of 4 columns took one thread and two 64-bit divisions per element before: 200,000 x 110 of
// 8-column subspaces 91.3 us, now 23.7; x 357 of 64 columns 279, now 71.  Widths of 4 n columns: 200,000 x 128 of 8 columns
// 23.5 us, now 18.7; x 200 of 32 41.3, now 27.8.
constexpr int kVqStagedThreads = 1024;
constexpr size_t kVqStagedSmem = 200 * 1024;
constexpr int kVqThreads = 512;

template <typename CodeT, typename CbT, int EPT, bool STAGED>
__global__ void __launch_bounds__(STAGED ? kVqStagedThreads : kVqThreads, STAGED ? 1 : 3) vq_decompress_kernel(
    const CodeT* __restrict__ codes, const CbT* __restrict__ cbs, float* __restrict__ out, int64_t rows, int units, int part, int rows_per_cta,
    int n_cb, int K, int cs, int feat_dim, int sub_per_part, int spq, int stride) {
  dependency_wait();
  release_dependents();
  extern __shared__ __align__(128) unsigned char vq_smem[];
  const int s0 = STAGED ? (int)blockIdx.y * sub_per_part : 0;  // first subspace of the part
  if constexpr (STAGED) {
    stage_codebooks(vq_smem, cbs + (int64_t)s0 * K * cs, min(sub_per_part, n_cb - s0), K, cs, spq, (int)blockDim.x);
    codebooks_staged();
    __syncthreads();
  }
  const int sub = threadIdx.x / part;
  const int unit = blockIdx.y * part + (threadIdx.x - sub * part);
  if (sub >= rows_per_cta || unit >= units) return;
  const int j = unit * EPT;
  const int s = j / cs, off = j - s * cs;
  const int sl = s - s0;
  const uint32_t lane_base = STAGED ? (uint32_t)__cvta_generic_to_shared(vq_smem) +
                                          (spq > 1 ? (uint32_t)((sl / spq) * K * 128 + (sl % spq) * cs * 4 + off * 4) : (uint32_t)(sl * K * stride + off * 4))
                                    : 0u;
  const CbT* const cb = cbs + (int64_t)s * K * cs + off;
  const int64_t step = (int64_t)gridDim.x * rows_per_cta;
  int64_t row = (int64_t)blockIdx.x * rows_per_cta + sub;
  const CodeT* cp = codes + row * n_cb + s;
  float* op = out + row * feat_dim + j;
  const int64_t cstep = step * n_cb, ostep = step * feat_dim;
  const uint32_t kmax = (uint32_t)K - 1u;
  auto fetch = [&](const CodeT* q) { return min((uint32_t)(int)__ldg(q), kmax); };
  constexpr int kInFlight = EPT == 4 && !STAGED ? 4 : 8;  // rows in flight per thread: what the registers of three CTAs hold
  auto value4 = [&](uint32_t c) {
    float4 v;
    if constexpr (STAGED) asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(lane_base + c * (uint32_t)stride));
    else v = load_cb4(cb + (int64_t)c * cs);
    return v;
  };
  auto value1 = [&](uint32_t c) {
    float v;
    if constexpr (STAGED) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(lane_base + c * (uint32_t)stride));
    else v = load_cb1(cb + (int64_t)c * cs);
    return v;
  };
  auto batch = [&](auto on) {
    uint32_t c[kInFlight];
#pragma unroll
    for (int u = 0; u < kInFlight; ++u) c[u] = on(u) ? fetch(cp + u * cstep) : 0u;
    if constexpr (EPT == 4) {
      float4 v[kInFlight];
#pragma unroll
      for (int u = 0; u < kInFlight; ++u) if (on(u)) v[u] = value4(c[u]);
#pragma unroll
      for (int u = 0; u < kInFlight; ++u) if (on(u)) stg_cs_f4(op + u * ostep, v[u]);
    } else {
      float v[kInFlight];
#pragma unroll
      for (int u = 0; u < kInFlight; ++u) if (on(u)) v[u] = value1(c[u]);
#pragma unroll
      for (int u = 0; u < kInFlight; ++u) if (on(u)) __stcs(op + u * ostep, v[u]);
    }
  };
  for (; row + (kInFlight - 1) * step < rows; row += kInFlight * step, cp += kInFlight * cstep, op += kInFlight * ostep) batch([](int) { return true; });
  if (row < rows) batch([&](int u) { return row + u * step < rows; });
}

template <typename CodeT, typename CbT, int EPT>
static int launch_vq_ept(const CodeT* codes, const CbT* cbs, float* out, int64_t rows, int64_t n_cb, int64_t K, int64_t cs, int64_t D, cudaStream_t st) {
  const int sms = current_sm_count();
  const int64_t units = D / EPT;
  if constexpr (std::is_same<CbT, float>::value) {
    // Reads of single floats from narrow centroids spread a warp over many lines of L1, so 8 and 16 columns are staged once there
    // is work for the copy of up to 200 KB per multiprocessor: 200,000 x 110 of 8 columns 23.7 us against 33.6 from L1, x 375 of
    // 16 69 against 78, but 27,000 x 110 8.9 against 7.5.  From 32 columns on L1 is as good or better (x 357 of 64: 88 against 71).
    // 16-byte reads from centroids of 16 columns or more gain from about 100 M outputs on, where the copy is nothing: calls in a row,
    // 24 / 48 / 96 / 128 / 192 / 256 M outputs, 128 columns of 32 18.0 / 33.5 / 66.1 / 88.5 / 132.4 / 176.6 us staged, 17.1 / 32.6 / 67.4 / 90.4 / 136.0 /
    // 180.2 not; 128 of 64 18.1 / 33.3 / 64.5 / 85.9 / 126.9 / 168.6 and 17.4 / 33.1 / 66.4 / 89.5 / 134.4 / 178.6; 192 of 32 18.3 / 33.5 / 66.5 / 89.2 /
    // 134.6 / 179.3 and 18.2 / 33.4 / 73.9 / 102.5 / 179.5 / 242.0; 112 of 16 70.4 / 70.4 at 96 M, 142.0 / 142.7 at 192 M,
    // 187.9 / 190.5 at 256 M.  Eight columns do not: 128 of 8 76.0 staged, 69.3 not at 96 M, 190.0 against 179.6 at 256 M.
    const int64_t used = ceil_div(D, cs);  // subspaces that hold columns
    const int spq = (cs & (cs - 1)) == 0 && cs < 32 ? (int)(32 / cs) : 1;
    const int64_t line = spq > 1 ? 128 * K : 4 * K * cs;  // bytes of spq subspaces
    const int64_t fit = (int64_t)kVqStagedSmem / line * spq;
    const bool worth = EPT == 1 ? cs < 32 && rows * D >= (8 << 20) : cs >= 16 && used <= fit && rows * D >= (96 << 20);
    if (fit > 0 && worth && cs % 4 == 0 && aligned(cbs, 16)) {
      int64_t parts = ceil_div(used, fit);
      while (parts < used && ceil_div(ceil_div(used, parts), spq) * spq * cs / EPT > kVqStagedThreads) ++parts;
      const int64_t spp = ceil_div(ceil_div(used, parts), spq) * spq;
      parts = ceil_div(used, spp);
      const int64_t part = spp < used ? spp * cs / EPT : units;
      if (part <= kVqStagedThreads && parts <= sms) {
        const Lanes ln = lanes_of_rows(part, rows, sms, kVqStagedThreads);
        const size_t smem = (size_t)(ceil_div(spp < n_cb ? spp : n_cb, spq) * line);
        auto kern = vq_decompress_kernel<CodeT, CbT, EPT, true>;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kVqStagedSmem) != cudaSuccess) return check_launch("vq_decompress");
        const int64_t grid = std::min(ceil_div(rows, ln.rows_per_cta), (int64_t)sms / parts);
        launch_dependent(kern, dim3((unsigned)grid, (unsigned)parts), ln.threads, smem, st, codes, cbs, out, rows, (int)units, (int)part,
                         ln.rows_per_cta, (int)n_cb, (int)K, (int)cs, (int)D, (int)spp, spq, spq > 1 ? 128 : (int)cs * 4);
        return check_launch("vq_decompress");
      }
    }
  }
  const Lanes ln = lanes_of_rows(units, rows, sms, kVqThreads);
  const int64_t grid = std::min(ceil_div(rows, ln.rows_per_cta), ceil_div((int64_t)sms * 3 * kVqThreads / ln.threads, ln.parts));
  launch_dependent(vq_decompress_kernel<CodeT, CbT, EPT, false>, dim3((unsigned)grid, (unsigned)ln.parts), ln.threads, 0, st, codes, cbs, out, rows,
                   (int)units, ln.part, ln.rows_per_cta, (int)n_cb, (int)K, (int)cs, (int)D, 0, 1, 0);
  return check_launch("vq_decompress");
}

template <typename CodeT, typename CbT>
static int launch_vq_decompress(const void* codes, const void* cbs, float* out, int64_t rows, int64_t n_cb, int64_t length,
                                int64_t cs, int64_t D, cudaStream_t st) {
  if (rows * D == 0) return F2C_OK;
  if (cs % 4 == 0 && D % 4 == 0 && aligned(out, 16) && aligned(cbs, 4 * sizeof(CbT)))
    return launch_vq_ept<CodeT, CbT, 4>((const CodeT*)codes, (const CbT*)cbs, out, rows, n_cb, length, cs, D, st);
  return launch_vq_ept<CodeT, CbT, 1>((const CodeT*)codes, (const CbT*)cbs, out, rows, n_cb, length, cs, D, st);
}

int validate_vq(const char* op, int code_dtype, int64_t n_cb, int64_t length, int64_t cs, int64_t feat_dim) {
  F2C_REQUIRE(is_code_dtype(code_dtype), F2C_ERR_UNSUPPORTED, "%s: codes must be uint8, int8 or int16", op);
  F2C_REQUIRE(n_cb >= 1 && length >= 1 && cs >= 1 && feat_dim >= 0, F2C_ERR_INVALID, "%s: bad codebook shape", op);
  F2C_REQUIRE(feat_dim <= n_cb * cs, F2C_ERR_INVALID, "%s: feat_dim %lld exceeds n_codebooks*column_slice = %lld", op,
              (long long)feat_dim, (long long)(n_cb * cs));
  F2C_REQUIRE(feat_dim < (1ll << 24) && length < (1ll << 31) && cs < (1ll << 24) && n_cb < (1ll << 24), F2C_ERR_LIMIT,
              "%s: shape too large", op);
  return F2C_OK;
}

}  // namespace f2c

using namespace f2c;

extern "C" int f2c_vq_decompress(const void* codes, int code_dtype, const void* codebooks, int codebook_dtype, float* out,
                                 int64_t rows, int64_t n_codebooks, int64_t length, int64_t column_slice,
                                 int64_t feat_dim, void* stream) {
  F2C_REQUIRE(rows >= 0, F2C_ERR_INVALID, "vq_decompress: negative size");
  int rc = validate_vq("vq_decompress", code_dtype, n_codebooks, length, column_slice, feat_dim);
  if (rc) return rc;
  F2C_REQUIRE(codebook_dtype == F2C_F32 || codebook_dtype == F2C_F16, F2C_ERR_UNSUPPORTED,
              "vq_decompress: codebooks must be float32 or float16");
  F2C_REQUIRE(rows * feat_dim == 0 || (codes && out && codebooks), F2C_ERR_INVALID, "vq_decompress: null pointer");
  cudaStream_t st = (cudaStream_t)stream;
#define F2C_VQ(T, C) return launch_vq_decompress<T, C>(codes, codebooks, out, rows, n_codebooks, length, column_slice, feat_dim, st)
  if (codebook_dtype == F2C_F32) {
    if (code_dtype == F2C_U8) F2C_VQ(uint8_t, float);
    if (code_dtype == F2C_I8) F2C_VQ(int8_t, float);
    F2C_VQ(int16_t, float);
  }
  if (code_dtype == F2C_U8) F2C_VQ(uint8_t, __half);
  if (code_dtype == F2C_I8) F2C_VQ(int8_t, __half);
  F2C_VQ(int16_t, __half);
#undef F2C_VQ
}
