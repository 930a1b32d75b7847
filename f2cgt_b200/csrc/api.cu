// Error plumbing and version of the C ABI (include/f2cgt_b200.h).
#include <stddef.h>

#include <mutex>

#include "common.cuh"
#include "stream_pipe.cuh"

namespace f2c {

static thread_local char g_error[512] = "";

int set_error(int status, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_error, sizeof(g_error), fmt, ap);
  va_end(ap);
  return status;
}

int check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return set_error(F2C_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  return F2C_OK;
}

int sm_count(int device) {
  static std::mutex mu;
  static int cached[64] = {};
  if (device < 0 || device >= 64) return kSmCount;
  std::lock_guard<std::mutex> lock(mu);
  if (cached[device] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || n < 1) {
      (void)cudaGetLastError();
      n = kSmCount;
    }
    cached[device] = n;
  }
  return cached[device];
}

int current_sm_count() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) dev = 0;
  return sm_count(dev);
}

// The record that kernels with bounded waits raise when a wait runs out; one per device (it lives in the device image).
static __device__ WaitReport g_wait_expired;

namespace {
struct Reported {
  int* word = nullptr;             // &g_wait_expired.code on the device
  volatile int* seen = nullptr;    // its copy in host memory
};

// The current device's record, looked up and given its host word at the first call.  The host word is four bytes of pinned memory
// that stay until the process ends.  Both are set up in relaxed capture mode: the first call may come while a graph is captured.
const Reported* reported() {
  static std::mutex mu;
  static Reported of_device[64];
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  std::lock_guard<std::mutex> lock(mu);
  Reported& r = of_device[dev];
  if (r.word == nullptr) {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    const bool relaxed = cudaThreadExchangeStreamCaptureMode(&mode) == cudaSuccess;
    void *at = nullptr, *host = nullptr, *mapped = nullptr;
    if (cudaGetSymbolAddress(&at, g_wait_expired) == cudaSuccess) {
      if (cudaHostAlloc(&host, sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable) == cudaSuccess) {
        *(volatile int*)host = 0;
        cudaStream_t st = nullptr;  // a stream of its own: the legacy one would wait for (and may not be used beside) others
        cudaError_t e = cudaHostGetDevicePointer(&mapped, host, 0);
        if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
        if (e == cudaSuccess) e = cudaMemcpyAsync((char*)at + offsetof(WaitReport, seen), &mapped, sizeof(mapped), cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (st != nullptr) (void)cudaStreamDestroy(st);
        if (e == cudaSuccess) r.seen = (volatile int*)host;
        else (void)cudaFreeHost(host);
      }
      r.word = (int*)at;
    }
    (void)cudaGetLastError();
    if (relaxed) (void)cudaThreadExchangeStreamCaptureMode(&mode);
  }
  return r.word != nullptr ? &r : nullptr;
}

__global__ void report_kernel(int* word, int code) { report_wait(word, code); }
}  // namespace

int* stream_error_word() {
  const Reported* r = reported();
  return r != nullptr ? r->word : nullptr;
}

}  // namespace f2c

extern "C" int f2c_device_status(int32_t* code_host, void* stream) {
  using namespace f2c;
  F2C_REQUIRE(code_host != nullptr, F2C_ERR_INVALID, "device_status: null pointer");
  const Reported* r = reported();
  F2C_REQUIRE(r != nullptr, F2C_ERR_CUDA, "device_status: the status word of this device is not reachable");
  cudaError_t e = cudaStreamSynchronize((cudaStream_t)stream);
  if (e == cudaSuccess) e = cudaMemcpy(code_host, r->word, sizeof(int), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && *code_host != 0) {
    e = cudaMemset(r->word, 0, sizeof(int));
    if (r->seen != nullptr) *r->seen = 0;
  }
  if (e != cudaSuccess) return set_error(F2C_ERR_CUDA, "device_status: %s", cudaGetErrorString(e));
  return F2C_OK;
}

extern "C" int f2c_device_status_seen(int32_t* code_host) {
  using namespace f2c;
  F2C_REQUIRE(code_host != nullptr, F2C_ERR_INVALID, "device_status_seen: null pointer");
  const Reported* r = reported();
  F2C_REQUIRE(r != nullptr && r->seen != nullptr, F2C_ERR_CUDA, "device_status_seen: the status word of this device is not reachable");
  *code_host = *r->seen;
  return F2C_OK;
}

extern "C" int f2c_device_status_report(int32_t code, void* stream) {
  using namespace f2c;
  const Reported* r = reported();
  F2C_REQUIRE(r != nullptr, F2C_ERR_CUDA, "device_status_report: the status word of this device is not reachable");
  report_kernel<<<1, 1, 0, (cudaStream_t)stream>>>(r->word, code);
  return check_launch("device_status_report");
}

extern "C" const char* f2c_last_error(void) { return f2c::g_error; }
extern "C" int f2c_version(void) { return 100; }
