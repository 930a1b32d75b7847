// Lloyd iterations on the tensor cores: many of them in ONE cooperative kernel, one CTA per SM (kmeans_tc.cuh holds its two halves: the
// assignment, and the sums and new centres behind it).  Two grid barriers per iteration stand where three kernels followed one another
// before, each near its own latency (a set-up, a list of undecided points that is usually a few hundred long, a last CTA that replaced the
// centres alone); the CTAs keep their TMEM and barriers, score their own undecided points, and replace a share of the centres each.
//
// Measured, one iteration (before: three kernels): 149,000 x 32, 256 centres 54 -> 32 us, x 8 30 -> 24, x 64 78 -> 56; 30,000 x 32 28 -> 21;
// 2,449,029 x 32 577 -> 287.  Of the 32 us the assignment takes 10, the centres' way into shared memory 2.5, the two barriers with what CTAs
// wait for one another 8 (those with undecided points come 4 later than the rest).
#include "kmeans_tc.cuh"

namespace f2c {
namespace tc {

template <int C, int NB, bool NO_WAITS = false>
__global__ void __launch_bounds__(kThreads, 1) kmeans_fit_kernel(const __grid_constant__ FitParams p) {
  if (*(volatile const int32_t*)&p.state->done != 0) return;  // converged, or not finite
  run<C, NB, NO_WAITS>(p);
}

// (All of this is the file's own, as `static` says: a type of that name, and a dispatch alike, is in the other file too.)
struct Kernel {
  void (*kern)(const FitParams);
  size_t smem;
};
template <int C>
static Kernel kernel_for(int64_t k) {
  return k <= 128 ? Kernel{kmeans_fit_kernel<C, 4>, Ring<C, 4>::bytes} : Kernel{kmeans_fit_kernel<C, 8>, Ring<C, 8>::bytes};
}
static Kernel kernel_for(int64_t k, int64_t d, bool no_waits) {
  if (no_waits) return Kernel{kmeans_fit_kernel<8, 8, true>, Ring<8, 8>::bytes};  // for any number of dimensions
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

// labels: 2 n numbers; those from n on are 0xffff and sums and counts zero before the first call, and theirs from call to call.
// shifts: one number per CTA, kFitMaxCtas at most.
int kmeans_fit_tc(const float* x, float* centers, int64_t n, int64_t k, int64_t d, int metric, double tol, int iterations, FitState* state, long long* sums,
                  uint32_t* counts, const uint32_t* maxima, uint16_t* labels, double* shifts, int32_t* error, cudaStream_t st, int flags) {
  const char* op = "kmeans_fit_iterate";
  tc::FitParams p{};
  tc::describe(p, x, centers, n, k, d, metric);
  p.error = error;
  p.state = state; p.centers = centers; p.labels16 = labels; p.summed16 = labels + n; p.sums = sums; p.counts = counts; p.maxima = maxima;
  p.shifts = shifts; p.tol = tol;
  auto [kern, smem] = tc::kernel_for(k, d, (flags & F2C_NO_WAITS) != 0);
  if (smem < tc::kOneCta) smem = tc::kOneCta;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return set_error(F2C_ERR_CUDA, "%s: %s", op, cudaGetErrorString(e));
  int64_t grid = ceil_div(n, tc::kTileM);
  if (grid > current_sm_count()) grid = current_sm_count();
  if (grid > kFitMaxCtas) grid = kFitMaxCtas;
  void* args[] = {(void*)&p};
  // A launch takes every SM, registers and all, so that kernels of other streams wait for its end: it has as many iterations as take about a
  // millisecond, one at least (2,449,029 x 32: 3 of 287 us; 149,000 x 32, 32 us each: all that are queued at a time).
  const int64_t most = (1ll << 28) / (n * (d < 16 ? 16 : d));
  while (iterations > 0) {
    p.iterations = most < 1 ? 1 : most < iterations ? (int)most : iterations;
    e = cudaLaunchCooperativeKernel((const void*)kern, dim3((unsigned)grid), dim3(tc::kThreads), args, smem, st);
    if (e != cudaSuccess) return set_error(F2C_ERR_CUDA, "%s: cooperative launch: %s", op, cudaGetErrorString(e));
    iterations -= p.iterations;
  }
  return check_launch(op);
}

}  // namespace f2c
