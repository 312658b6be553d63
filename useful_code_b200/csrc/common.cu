// common.cu — status/error plumbing shared by every C-ABI entry point.
#include "lmm_common.cuh"

#include <cuda.h>

#include <atomic>
#include <cstdarg>
#include <cstdio>

#include "../../include/lmm_pipeline.h"

namespace lmm {

namespace {
thread_local char g_last_error[1024] = "no error";
}

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_last_error, sizeof(g_last_error), fmt, ap);
  va_end(ap);
}

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_last_error, sizeof(g_last_error), fmt, ap);
  va_end(ap);
  return code;
}

int check_cuda(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return LMM_OK;
  return fail(LMM_ECUDA, "%s: %s", what, cudaGetErrorString(e));
}

namespace {
std::atomic<long> g_launches{0};
}

int check_launch(const char* what) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return check_cuda(cudaGetLastError(), what);
}

int sm_count() {
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (cached[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) !=
            cudaSuccess ||
        n <= 0)
      n = 148;
    cached[dev] = n;
  }
  return cached[dev];
}

namespace {
template <class Fn>
Fn driver_fn(const char* name) {
  void* f = nullptr;
  cudaDriverEntryPointQueryResult found = cudaDriverEntryPointSymbolNotFound;
  if (cudaGetDriverEntryPointByVersion(name, &f, 12040, cudaEnableDefault, &found) !=
          cudaSuccess ||
      found != cudaDriverEntryPointSuccess)
    return nullptr;
  return reinterpret_cast<Fn>(f);
}
}  // namespace

int stream_sm_count(cudaStream_t s) {
  static const auto green_of =
      driver_fn<CUresult (*)(CUstream, CUgreenCtx*)>("cuStreamGetGreenCtx");
  static const auto resource_of =
      driver_fn<CUresult (*)(CUgreenCtx, CUdevResource*, CUdevResourceType)>(
          "cuGreenCtxGetDevResource");
  const int all = sm_count();
  CUgreenCtx green = nullptr;
  CUdevResource res;
  if (!green_of || !resource_of || green_of((CUstream)s, &green) != CUDA_SUCCESS || !green ||
      resource_of(green, &res, CU_DEV_RESOURCE_TYPE_SM) != CUDA_SUCCESS)
    return all;
  const int own = (int)res.sm.smCount;
  return own > 0 && own < all ? own : all;
}

// A kernel's limit is one value for all threads of the process.  One made to
// a launch's measure could be lowered by another thread's call between this
// call and the launch, so it only ever goes to the device's most: every
// thread that sets it sets the same value.
int allow_smem(const void* kern, size_t bytes, const char* what) {
  cudaFuncAttributes fa;
  int st = check_cuda(cudaFuncGetAttributes(&fa, kern), what);
  if (st) return st;
  constexpr size_t kUnasked = 48 * 1024;  // static and dynamic, without asking
  const size_t limit = (size_t)fa.maxDynamicSharedSizeBytes;
  if (bytes + fa.sharedSizeBytes <= kUnasked || (limit > kUnasked && bytes <= limit))
    return LMM_OK;
  int dev = 0, most = 0;
  st = check_cuda(cudaGetDevice(&dev), what);
  if (st) return st;
  st = check_cuda(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev),
                  what);
  if (st) return st;
  most -= (int)fa.sharedSizeBytes;
  if (bytes > (size_t)most)
    return fail(LMM_ECUDA, "%s: %zu bytes of shared memory, the device has %d", what, bytes,
                most);
  return check_cuda(
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most), what);
}

}  // namespace lmm

extern "C" const char* lmm_last_error_string(void) { return lmm::g_last_error; }

extern "C" int lmm_version(void) { return 1; }

extern "C" long lmm_launch_count(void) {
  return lmm::g_launches.load(std::memory_order_relaxed);
}
