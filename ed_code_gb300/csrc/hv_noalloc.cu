// edg_hv_noalloc: the stored-row H*v of targets.cu for callers that must not
// allocate device memory.
//
// The stored-row H*v runs in two kernels: the first writes u = v / norm into a
// scratch vector of n_p entries, the second streams the rows and gathers
// from u.  edg_hv keeps that scratch in a buffer that edg_sector_build_targets
// allocates with cudaMalloc.  Some callers cannot have the library allocate or
// free device memory while they run: applications whose own allocator already
// owns the device's free memory (a framework's caching allocator, an arena
// sized at start-up), so that an extra cudaMalloc fails or fragments it, and
// latency-bound loops, where cudaMalloc/cudaFree would synchronise the device.
// This file gives them a variant whose scratch is a fixed array in the
// library's own device image, so the call itself allocates nothing.
//
// Limits and sharing:
//  * the array holds kScratchBytes = 16 MiB on every GPU that loads this
//    library's device code, until the process exits; hence at most 1,048,576
//    entries for complex128 and 2,097,152 for complex64 -- larger sectors are
//    rejected with EDG_ERR_INVALID;
//  * every call on a device uses the same array.  Nothing in it has to start
//    at zero (the first kernel writes entries 0..n_p-1 before the second one
//    reads them), but calls that overlap on the GPU -- on two streams, from
//    two threads, for two sectors -- overwrite each other's u and race.
//    Order them on one stream or with events.
#include <cuda_runtime.h>

#include <cstddef>
#include <mutex>
#include <string>

#include "../../include/edgpu.h"
#include "edg_sector.cuh"

struct edg_sector {
  edg::Sector s;
};

namespace edg {
int fail(int code, const std::string& msg);
int cuda_fail(cudaError_t e, const char* what);
}  // namespace edg

namespace {

constexpr size_t kScratchBytes = size_t(16) << 20;
constexpr int kMaxDevices = 64;

}  // namespace

// The scratch vector u.  In host code this name is only a host-side handle:
// kernels are given the device address that cudaGetSymbolAddress returns.
static __device__ __align__(256) double2 g_hv_scratch[kScratchBytes / sizeof(double2)];

namespace {

std::mutex g_setup_mutex;
void* g_scratch_addr[kMaxDevices] = {};

// Device address of g_hv_scratch on `dev`, looked up once per device (with
// that device current) and cached.
cudaError_t scratch_address(int dev, void** out) {
  std::lock_guard<std::mutex> lock(g_setup_mutex);
  if (!g_scratch_addr[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_hv_scratch);
    if (e != cudaSuccess) return e;
    g_scratch_addr[dev] = p;
  }
  *out = g_scratch_addr[dev];
  return cudaSuccess;
}

}  // namespace

extern "C" int edg_hv_noalloc(edg_sector* s, const void* v, void* w, int dtype, void* stream) {
  using namespace edg;
  if (!s || !v || !w) return fail(EDG_ERR_INVALID, "NULL argument");
  if (dtype != EDG_C128 && dtype != EDG_C64) return fail(EDG_ERR_INVALID, "dtype must be EDG_C128 or EDG_C64");
  if (v == w) return fail(EDG_ERR_INVALID, "v and w must not alias");
  const Sector& S = s->s;
  const size_t elem = dtype == EDG_C128 ? 16 : 8;
  const int64_t max_n = (int64_t)(kScratchBytes / elem);
  if (S.P.n_p > max_n)
    return fail(EDG_ERR_INVALID, "edg_hv_noalloc: sector has " + std::to_string(S.P.n_p) +
                                     " states; its fixed 16 MiB scratch holds at most " + std::to_string(max_n) +
                                     (dtype == EDG_C128 ? " complex128" : " complex64") + " entries (use edg_hv)");
  if (!S.col) return fail(EDG_ERR_INVALID, "edg_hv_noalloc needs stored rows (edg_sector_build_targets)");
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e, "edg_hv_noalloc: cudaGetDevice");
  if (dev != S.device) return fail(EDG_ERR_INVALID, "edg_hv_noalloc: make the sector's device current first");
  if (dev < 0 || dev >= kMaxDevices) return fail(EDG_ERR_INVALID, "edg_hv_noalloc: device index out of range");
  void* u = nullptr;
  e = scratch_address(dev, &u);
  if (e != cudaSuccess) return cuda_fail(e, "edg_hv_noalloc: cudaGetSymbolAddress of the scratch array");
  const cudaStream_t st = (cudaStream_t)stream;
  if (S.folded) u = const_cast<void*>(v);  // the rows gather v itself
  else e = launch_u(S, v, u, dtype == EDG_C128, st);
  if (e == cudaSuccess) e = launch_hv_rows(S, v, u, w, dtype == EDG_C128, 0, S.P.n_p, st);
  if (e != cudaSuccess) return cuda_fail(e, "edg_hv_noalloc launch");
  return EDG_OK;
}
