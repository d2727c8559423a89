// A stand-in for the CUDA runtime for host tests of allocation paths: device memory is
// host memory, kernels do nothing, and the allocation of a chosen number fails.
// Built without the real runtime; never linked into the library.
#include "fake_cudart.h"

#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <utility>

namespace fake {
static std::map<void*, size_t> g_live;
static int g_fail_in = 0;  // the g_fail_in-th allocation from now fails; 0: none
void fail_in(int n) { g_fail_in = n; }
bool live(const void* p) { return g_live.count(const_cast<void*>(p)) != 0; }
size_t live_blocks() { return g_live.size(); }
size_t live_bytes() {
  size_t n = 0;
  for (auto& b : g_live) n += b.second;
  return n;
}
int bad_frees = 0;
int device = 0, refused = 0;
static std::set<std::pair<int, const void*>> g_opted_in;
size_t opted_in() { return g_opted_in.size(); }
}  // namespace fake

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
  *p = nullptr;
  if (fake::g_fail_in > 0 && --fake::g_fail_in == 0) return cudaErrorMemoryAllocation;
  *p = std::calloc(1, n ? n : 1);
  fake::g_live[*p] = n;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  if (!p) return cudaSuccess;
  if (!fake::g_live.erase(p)) ++fake::bad_frees;
  else std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
  std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = nullptr;
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  *p = std::calloc(1, n);
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = fake::device;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int) {
  fake::g_opted_in.insert({fake::device, f});
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  if (c->dynamicSmemBytes > 48 * 1024 && !fake::g_opted_in.count({fake::device, f})) ++fake::refused;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }

// what nvcc's host code calls
void** __cudaRegisterFatBinary(void*) {
  static void* h = nullptr;
  return &h;
}
char __cudaInitModule(void**) { return 0; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return 1; }  // non-zero: the launch is left out
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
cudaError_t __cudaGetKernel(void*, const void*) { return cudaSuccess; }
cudaError_t __cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, void*) { return cudaSuccess; }
}
