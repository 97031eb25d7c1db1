// The part of the CUDA runtime that the library's host code calls, for a machine without a GPU: kernel launches are
// checked against the attributes that were set for the kernel ON THE CURRENT DEVICE and are otherwise dropped.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <map>
#include <utility>

namespace {
int device = 0;
int launches = 0;
cudaError_t last = cudaSuccess;
std::map<std::pair<int, const void*>, int> smem_limit;
struct {
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
} config;

cudaError_t launch(const void* func, dim3 grid, dim3 block, size_t smem) {
  auto it = smem_limit.find({device, func});
  const size_t limit = it == smem_limit.end() ? 48 * 1024 : it->second;
  const bool fits = smem <= limit && grid.x && grid.y && grid.z && block.x * block.y * block.z <= 1024;
  if (!fits) return last = cudaErrorInvalidValue;
  ++launches;
  return cudaSuccess;
}
CUresult encode(...) { return CUDA_SUCCESS; }
}  // namespace

extern "C" {
void fake_set_device(int d) { device = d; }
int fake_launches() { return launches; }

void** __cudaRegisterFatBinary(void*) { static void* handle; return &handle; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
  config = {grid, block, smem, stream};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
  *grid = config.grid;
  *block = config.block;
  *smem = config.smem;
  *static_cast<cudaStream_t*>(stream) = config.stream;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* func, dim3 grid, dim3 block, void**, size_t smem, cudaStream_t) {
  return launch(func, grid, block, smem);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* func, void**) {
  return launch(func, c->gridDim, c->blockDim, c->dynamicSmemBytes);
}
cudaError_t cudaFuncSetAttribute(const void* func, cudaFuncAttribute attr, int value) {
  if (attr == cudaFuncAttributeMaxDynamicSharedMemorySize) smem_limit[{device, func}] = value;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaGetLastError() { cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
  *s = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPoint(const char*, void** fn, unsigned long long, cudaDriverEntryPointQueryResult* r) {
  *fn = reinterpret_cast<void*>(&encode);
  if (r) *r = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemset(void*, int, size_t) { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t) { *p = nullptr; return cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void*) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { *p = nullptr; return cudaSuccess; }
cudaError_t cudaDeviceEnablePeerAccess(int, unsigned) { return cudaSuccess; }
cudaError_t cudaIpcGetMemHandle(cudaIpcMemHandle_t*, void*) { return cudaErrorInvalidValue; }
cudaError_t cudaIpcOpenMemHandle(void**, cudaIpcMemHandle_t, unsigned) { return cudaErrorInvalidValue; }
cudaError_t cudaIpcCloseMemHandle(void*) { return cudaErrorInvalidValue; }
}
