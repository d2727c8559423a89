// Programmatic dependent launch: a kernel launched with programmatic stream
// serialisation may start while its predecessor in the stream drains.  Such a
// kernel reads nothing its predecessor writes before grid_dep_wait(), and
// releases its own successor only after that wait, so no kernel's early part
// runs before the kernel two launches back has completed.  One exception: the
// motion-compensated row-local iteration (rowlocal.cuh) releases at its start
// and waits only before its update; its successor (the fused tTV kernel of
// the next iteration) waits before reading anything, and its own early part
// reads only what the launch three back wrote.
#pragma once

#include <atomic>

#include <cuda_runtime.h>

namespace gbn {

__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void grid_dep_release() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

// launch with programmatic stream serialisation (`first`: without it).  The first
// kernel of a chain follows one that does not release its successors, such as the
// kernels that write a group's control block, the scalar state or the tiles of a
// solve.  That one has ended when a successor starts early, but what it wrote is
// only certain to be seen after the successor's grid_dep_wait(), and these
// kernels read such data before it: the first one is launched plainly.
template <typename... KArgs, typename... Args>
inline void launch_chain(bool first, void (*kernel)(KArgs...), dim3 grid, int threads, int smem, cudaStream_t s,
                         Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = size_t(smem);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = first ? 0 : 1;
  cudaLaunchKernelEx(&cfg, kernel, args...);
}
template <typename... KArgs, typename... Args>
inline void launch_pdl(void (*kernel)(KArgs...), dim3 grid, int threads, int smem, cudaStream_t s, Args... args) {
  launch_chain(false, kernel, grid, threads, smem, s, args...);
}

// The devices a kernel's attribute has been set on: it holds on the device that is
// current when it is set, and a process may have contexts on several.
struct OptedIn {
  std::atomic<unsigned long long> devices{0};  // bit per device; those past 63 set it on every launch
};
template <typename K>
inline void opt_in(K kernel, cudaFuncAttribute attr, int value, OptedIn& done) {
  int dev = 0;
  cudaGetDevice(&dev);
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0;
  if (!(done.devices.load(std::memory_order_acquire) & bit)) {
    cudaFuncSetAttribute(kernel, attr, value);
    done.devices.fetch_or(bit, std::memory_order_release);
  }
}
// the current device's SMs
inline int device_sms() {
  static std::atomic<int> known[64];
  int dev = 0, n = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && (n = known[dev].load(std::memory_order_relaxed)) > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) n = 1;
  if (dev < 64) known[dev].store(n, std::memory_order_relaxed);
  return n;
}
// more than 48 KB of dynamic shared memory
template <typename K>
inline void allow_smem(K kernel, int bytes, OptedIn& done) {
  opt_in(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes, done);
}

}  // namespace gbn
