// The launchers of the evaluation and tensor-core kernels on a process with two
// devices, against a stand-in for the CUDA runtime that keeps a kernel's dynamic
// shared-memory limit per device, as the real one does: a launch above 48 KB on a
// device whose limit was never raised fails.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <utility>
#include <vector>

#include "tc_gemm.h"
#include "tci_tasks.h"

cudaError_t tci_tt_eval_launch(const tci_core_ref* cores, int* cls, int L, int rmax, const uint8_t* pts, int64_t np,
                               double* out, int num_sms, cudaStream_t st);

static int device = 0, large = 0, fail_next_set = 0;
static cudaError_t last = cudaSuccess;
static std::map<std::pair<int, const void*>, int> limits;
static struct {
  dim3 grid, block;
  size_t smem;
  void* stream;
} cfg;

static CUresult encode(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                       const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                       CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
  return CUDA_SUCCESS;
}

extern "C" {
void** __cudaRegisterFatBinary(void*) {
  static void* h[1];
  return h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, void* st) {
  cfg = {g, b, s, st};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* st) {
  *g = cfg.grid;
  *b = cfg.block;
  *s = cfg.smem;
  *(void**)st = cfg.stream;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
  *k = (cudaKernel_t)f;
  return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void**, size_t smem, cudaStream_t) {
  if (smem > 48 * 1024) {
    ++large;
    const auto it = limits.find({device, (const void*)k});
    if (it == limits.end() || (size_t)it->second < smem) last = cudaErrorInvalidValue;
  }
  return last;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  if (fail_next_set) {
    fail_next_set = 0;
    return cudaErrorUnknown;
  }
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) limits[{device, f}] = v;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = device;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return std::exchange(last, cudaSuccess); }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** p, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* q) {
  *p = (void*)encode;
  *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
}

#define CHECK(x)                                  \
  if (!(x)) {                                     \
    std::printf("line %d: %s\n", __LINE__, #x);   \
    return 1;                                     \
  }

int main() {
  const int64_t dims[] = {1, 2, 128, 128, 2, 128, 128, 2, 1};
  const double* cores[3] = {nullptr, nullptr, nullptr};
  std::vector<char> ws(tci_tc_eval_workspace(3, dims) + 4096);
  // a failed set is reported and not kept
  fail_next_set = 1;
  CHECK(tci_tt_eval_launch(nullptr, nullptr, 3, 80, nullptr, 100000, nullptr, 152, nullptr) == cudaErrorUnknown);
  for (int round = 0; round < 2; ++round)
    for (device = 0; device < 3; ++device) {
      CHECK(tci_tt_eval_launch(nullptr, nullptr, 3, 80, nullptr, 100000, nullptr, 152, nullptr) == cudaSuccess);
      CHECK(tci_tc_evaluate_split(3, dims, cores, nullptr, 1000, nullptr, 0, nullptr, ws.data(), nullptr, 152,
                                  nullptr) == cudaSuccess);
      for (int64_t n : {64, 128, 256})
        CHECK(tci_tc_gemm_split(256, n, 64, nullptr, tci_map_stride(1), tci_map_stride(256), 0, nullptr,
                                tci_map_stride(1), tci_map_stride(n), 0, nullptr, tci_map_stride(1),
                                tci_map_stride(256), ws.data(), nullptr, nullptr) == cudaSuccess);
    }
  CHECK(large == 2 * 3 * 5);  // every launch was one that needs the limit
  std::puts("ok");
  return 0;
}
