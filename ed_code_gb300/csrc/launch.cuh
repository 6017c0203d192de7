// Grid sizes of the kernels that are launched on every H*v.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace edg {
namespace {

struct Resident {
  int sms, per_sm;  // SMs of the current device, CTAs of the kernel that fit on one
};

// What the runtime says about (kernel, threads, shared memory) on the current
// device, remembered per thread: a launch asked three queries, about a
// microsecond, each time.  smem_most is the most that any launch of this kernel
// asks for (the limit of the kernel's dynamic shared memory, set once).
inline Resident resident(const void* kernel, int threads, size_t smem, size_t smem_most) {
  struct Entry {
    const void* kernel;
    size_t smem;
    int dev;
    Resident r;
  };
  constexpr int kEntries = 64;
  static thread_local Entry known[kEntries] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  const size_t h = (reinterpret_cast<size_t>(kernel) >> 4) * 31 + smem * 7 + (size_t)dev;
  Entry& e = known[h % kEntries];
  if (e.kernel == kernel && e.smem == smem && e.dev == dev && e.r.per_sm > 0) return e.r;
  Resident r{0, 0};
  cudaDeviceGetAttribute(&r.sms, cudaDevAttrMultiProcessorCount, dev);
  if (smem_most > 48 * 1024)
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_most);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r.per_sm, kernel, threads, smem);
  if (r.per_sm < 1) r.per_sm = 1;
  e = Entry{kernel, smem, dev, r};
  return r;
}

}  // namespace
}  // namespace edg
