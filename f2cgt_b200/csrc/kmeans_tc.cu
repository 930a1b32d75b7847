// Entry points of the tensor-core k-means assignment (the kernel: kmeans_tc.cuh).
#include <mutex>

#include "kmeans_tc.cuh"

namespace f2c {

namespace tc {

template <int C, int NB, bool NO_WAITS = false>
__global__ void __launch_bounds__(kThreads, 1) kmeans_tc_kernel(const __grid_constant__ Params p) {
  dependency_wait();
  release_dependents();
  run<C, NB, NO_WAITS>(p);
}

// (All of this is the file's own, as `static` says: a type of that name, and a dispatch alike, is in the other file too.)
struct Kernel {
  void (*kern)(const Params);
  size_t smem;
};
template <int C>
static Kernel kernel_for(int64_t k) {
  return k <= 128 ? Kernel{kmeans_tc_kernel<C, 4>, Ring<C, 4>::bytes} : Kernel{kmeans_tc_kernel<C, 8>, Ring<C, 8>::bytes};
}
static Kernel kernel_for(int64_t k, int64_t d, bool no_waits) {
  if (no_waits) return Kernel{kmeans_tc_kernel<8, 8, true>, Ring<8, 8>::bytes};  // for any number of dimensions
  switch ((d + 7) / 8) {
    case 1: return kernel_for<1>(k);
    case 2: return kernel_for<2>(k);
    case 3: return kernel_for<3>(k);
    case 4: return kernel_for<4>(k);
    case 5: return kernel_for<5>(k);
    case 6: return kernel_for<6>(k);
    case 7: return kernel_for<7>(k);
    default: return kernel_for<8>(k);
  }
}

}  // namespace tc

// Eligibility and scratch size of the tensor-core path.
bool kmeans_tc_supported(int64_t n, int64_t k, int64_t d) { return n >= 1 && n < (1ll << 31) && k >= 1 && k <= tc::kMaxN && d >= 1 && d <= 64; }
constexpr int64_t kTcWorkspace = 256;  // [points that the exact scorer assigned, error]
int64_t kmeans_tc_workspace() { return kTcWorkspace; }

int kmeans_assign_tc(const float* x, const float* y, int64_t* labels, int64_t n, int64_t k, int64_t d, int metric, void* workspace,
                     cudaStream_t st, int flags) {
  tc::Params p{};
  tc::describe(p, x, y, n, k, d, metric);
  p.labels = labels;
  int32_t* head = reinterpret_cast<int32_t*>(workspace);
  p.undecided = head; p.error = head + 1;
  cudaError_t e = cudaMemsetAsync(head, 0, 8, st);
  if (e != cudaSuccess) return set_error(F2C_ERR_CUDA, "kmeans_assign: %s", cudaGetErrorString(e));
  auto [kern, smem] = tc::kernel_for(k, d, (flags & F2C_NO_WAITS) != 0);
  if (smem < tc::kOneCta) smem = tc::kOneCta;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return set_error(F2C_ERR_CUDA, "kmeans_assign: %s", cudaGetErrorString(e));
  int64_t grid = ceil_div(n, tc::kTileM);
  if (grid > current_sm_count()) grid = current_sm_count();  // one CTA per SM (it owns all 512 TMEM columns)
  launch_dependent(kern, (unsigned)grid, tc::kThreads, smem, st, p);
  return check_launch("kmeans_assign (tensor cores)");
}

// ------------------------------------------------------------------------------------------------------
// K-means assignment for callers that cannot allocate device memory.
//
// f2c_kmeans_assign reports to a buffer of the caller's, which means one small device allocation per call (or a buffer the caller
// has to carry around).  Some callers cannot do that: a data-loader or serving thread that lives inside a process whose framework
// allocator already owns almost all of HBM (a raw cudaMalloc there can fail, or make the framework drop its cache), and callers on
// a latency-critical path, where cudaMalloc / cudaFree would stall every stream of the device.  For them the report lives in a
// fixed array in the library's device image.  (It held a list of undecided points, too, which is where the limit of points per
// call comes from.)
//
// The array's name below is only a host-side handle; the device address is obtained once per device with
// cudaGetSymbolAddress while that device is current.  That happens on the first call made on a device (a
// synchronising runtime query, once).  All calls on a device share the one array, which is cleared at the start of every call:
// two calls that overlap on the GPU (different streams, or threads) would mix their reports - serialise them.
namespace tc {
constexpr int64_t kStaticMaxPoints = 1 << 20;
static __device__ __align__(256) unsigned char g_static_scratch[kTcWorkspace];

// Device address of the scratch array on the current device, looked up once per device (with that device current).
static int static_scratch(const char* op, void** scratch) {
  static std::mutex mu;
  static void* scratch_of_device[64] = {nullptr};
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 64) return set_error(F2C_ERR_CUDA, "%s: cudaGetDevice: %s", op, cudaGetErrorString(e));
  std::lock_guard<std::mutex> lock(mu);
  if (scratch_of_device[dev] == nullptr) {
    void* ptr = nullptr;
    e = cudaGetSymbolAddress(&ptr, g_static_scratch);
    if (e != cudaSuccess || ptr == nullptr) return set_error(F2C_ERR_CUDA, "%s: cudaGetSymbolAddress: %s", op, cudaGetErrorString(e));
    scratch_of_device[dev] = ptr;
  }
  *scratch = scratch_of_device[dev];
  return F2C_OK;
}
}  // namespace tc
}  // namespace f2c

extern "C" int f2c_kmeans_assign_static(const float* x, const float* centers, int64_t* labels, int64_t n, int64_t k,
                                        int64_t d, int metric, void* stream) {
  using namespace f2c;
  const char* op = "kmeans_assign_static";
  F2C_REQUIRE(n >= 0 && k >= 1 && d >= 1, F2C_ERR_INVALID, "%s: bad shape n=%lld k=%lld d=%lld", op, (long long)n, (long long)k,
              (long long)d);
  F2C_REQUIRE(metric == F2C_L2 || metric == F2C_COSINE, F2C_ERR_INVALID, "%s: unknown metric", op);
  F2C_REQUIRE(n <= tc::kStaticMaxPoints, F2C_ERR_LIMIT,
              "%s: %lld points exceed the %lld of one call; split it or use kmeans_assign with a workspace", op,
              (long long)n, (long long)tc::kStaticMaxPoints);
  F2C_REQUIRE(k <= tc::kMaxN && d <= 64, F2C_ERR_LIMIT, "%s: at most %d centres of at most 64 dimensions", op, tc::kMaxN);
  if (n == 0) return F2C_OK;
  F2C_REQUIRE(x && centers && labels, F2C_ERR_INVALID, "%s: null pointer", op);

  void* scratch = nullptr;
  int rc = tc::static_scratch(op, &scratch);
  if (rc) return rc;
  // same kernels as kmeans_assign; the header (count, error code) is cleared inside
  return kmeans_assign_tc(x, centers, labels, n, k, d, metric, scratch, (cudaStream_t)stream, 0);
}

// What the last f2c_kmeans_assign_static call on the current device left in the header of the built-in array: the
// number of points the tensor-core pass handed to the exact scorer, and the code the kernel writes when one of its
// bounded barrier waits ran out (0 = none; the exact scorer then assigned every point).  Waits for `stream`,
// copies the eight header bytes to the host, allocates nothing.  Returns F2C_ERR_CUDA when the code is non-zero.
extern "C" int f2c_kmeans_assign_static_status(int32_t* undecided_host, int32_t* error_host, void* stream) {
  using namespace f2c;
  const char* op = "kmeans_assign_static_status";
  void* scratch = nullptr;
  int rc = tc::static_scratch(op, &scratch);
  if (rc) return rc;
  cudaError_t e = cudaStreamSynchronize((cudaStream_t)stream);
  if (e != cudaSuccess) return set_error(F2C_ERR_CUDA, "%s: %s", op, cudaGetErrorString(e));
  int32_t head[2] = {0, 0};
  e = cudaMemcpy(head, scratch, sizeof(head), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return set_error(F2C_ERR_CUDA, "%s: %s", op, cudaGetErrorString(e));
  if (undecided_host) *undecided_host = head[0];
  if (error_host) *error_host = head[1];
  if (head[1] != 0) return set_error(F2C_ERR_CUDA, "%s: the tensor-core kernel gave up on a bounded wait (code %d)", op, head[1]);
  return F2C_OK;
}
