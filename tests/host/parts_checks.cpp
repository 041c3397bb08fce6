// Both gradients of a product of 16-bit parts (k_gemm_parts.cu) without a GPU, over stubs of the CUDA runtime that count launches: if a tensor map
// cannot be made or there is no room, nothing has been launched when the caller is told to take another kernel, which would add to the
// weight's gradient once more.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include <cuda.h>
#include "../../rusttensor_b200/csrc/rt_internal.cuh"

rt_status rt_matmul_backward_parts_internal(rt_ctx* ctx, const float* a, const float* b, const float* g, int64_t m, int64_t k, int64_t n, float* da,
                                            float* db, int accumulate_db);

static int failures, launches, blocks, maps, maps_left = -1, mallocs_left = -1;
#define EXPECT(x) ((x) ? (void)0 : (void)(std::printf("line %d: %s\n", __LINE__, #x), ++failures))

static CUresult encode(CUtensorMap* m, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                       CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
  if (maps_left == 0) return CUDA_ERROR_INVALID_VALUE;
  if (maps_left > 0) --maps_left;
  ++maps;
  std::memset(m, 0, sizeof(*m));
  return CUDA_SUCCESS;
}
extern "C" {
rt_status rt_malloc(rt_ctx*, size_t bytes, void** out) {
  if (mallocs_left == 0) return RT_ERR_OOM;
  if (mallocs_left > 0) --mallocs_left;
  ++blocks;
  *out = std::malloc(bytes < 64 ? bytes : 64);  // never looked into
  return RT_OK;
}
rt_status rt_free(rt_ctx*, void* p) {
  --blocks;
  std::free(p);
  return RT_OK;
}
void** __cudaRegisterFatBinary(void*) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
char __cudaInitModule(void**) { return 1; }
unsigned __cudaPopCallConfiguration(void*, void*, size_t*, void*) { return 0; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaPeekAtLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "stub"; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return ++launches, cudaSuccess; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) { return ++launches, cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** f, unsigned long long, cudaDriverEntryPointQueryResult* q) {
  *f = reinterpret_cast<void*>(&encode);
  *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
}

int main() {
  rt_ctx ctx;
  alignas(16) float x[16];
  auto gradients = [&] {
    launches = maps = 0;
    return rt_matmul_backward_parts_internal(&ctx, x, x, x, 1300, 1101, 1203, x, x, 1);
  };
  EXPECT(gradients() == RT_OK && launches == 5 && maps == 4 && blocks == 0);  // sample, two splits, two products
  for (int k = 0; k < 4; ++k) {
    maps_left = k;
    EXPECT(gradients() == RT_ERR_UNIMPLEMENTED && launches == 0 && blocks == 0);
  }
  maps_left = -1;
  for (int k = 0; k < 5; ++k) {
    mallocs_left = k;
    EXPECT(gradients() == RT_ERR_UNIMPLEMENTED && launches == 0 && blocks == 0);
  }
  return failures ? 1 : 0;
}
