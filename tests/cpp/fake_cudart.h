// A fake of the CUDA runtime calls that the launchers make, for host checks
// without a GPU.  Two contexts and more, told apart by `ctx`: a kernel's
// dynamic shared-memory limit is 48 KB in each until it is raised there, and a
// launch above the limit is refused, as the runtime does.
#pragma once
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <map>

// nvcc's host stubs call these; only what the launch needs is kept
#include <cuda_runtime.h>

namespace fake {
inline unsigned long long ctx = 1;  // identity of the current context
inline std::map<std::pair<unsigned long long, const void*>, size_t> limit;
inline int launches = 0, refused = 0, attribute_calls = 0, queries = 0;
inline bool fail_query = false;
inline int get_id(void*, unsigned long long* id) { return *id = ctx, 0; }
inline size_t limit_of(const void* f) {
  auto it = limit.find({ctx, f});
  return it == limit.end() ? 48 * 1024 : it->second;
}
}  // namespace fake

extern "C" {
void** __cudaRegisterFatBinary(void*) {
  static void* h = nullptr;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) { return *k = (cudaKernel_t)f, cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, struct CUstream_st*) { return 1; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMaxSharedMemoryPerMultiprocessor  ? 228 * 1024
       : a == cudaDevAttrMaxRegistersPerMultiprocessor   ? 65536
       : a == cudaDevAttrMaxThreadsPerMultiProcessor     ? 2048
                                                         : 0;
  return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
  fake::queries++;
  if (fake::fail_query) return cudaErrorUnknown;
  std::memset(a, 0, sizeof *a);
  a->numRegs = 64;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  fake::attribute_calls++;
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) fake::limit[{fake::ctx, f}] = (size_t)v;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int, size_t smem, unsigned) {
  fake::queries++;
  if (fake::fail_query) return cudaErrorUnknown;
  return *n = smem <= fake::limit_of(f) ? 3 : 0, cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  fake::launches++;
  if (c->dynamicSmemBytes <= fake::limit_of(f)) return cudaSuccess;
  return fake::refused++, cudaErrorInvalidValue;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char* name, void** p, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* r) {
  const bool id = !std::strcmp(name, "cuCtxGetId");
  *p = id ? reinterpret_cast<void*>(&fake::get_id) : nullptr;
  *r = id ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
  return cudaSuccess;
}
}
