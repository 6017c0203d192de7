// H applied to NV vectors at once (NV = 2 or 4) on the stored rows.
//
// The 36-site H*v moves about 1.5x its algorithmic bytes: the targets that a
// flip sends to another orbit member land at random positions of u, and each
// such gather moves a whole line from HBM for one 8-byte entry.  With NV
// vectors interleaved by row (element i of vector q at [i * NV + q]) one
// gather brings the entry of every vector -- 16 bytes (NV = 2) or 32 bytes
// (NV = 4) in FP32, still inside the line the single-vector gather already
// moves -- and the row's entries are read once for all NV vectors.
//
// It is the single-vector kernel (hv_rows.cuh) with NV sums per row: vector q
// of the block gets, bit for bit, what it gets alone.  Consumers: block
// solvers, and the FP64 Rayleigh quotients of several Ritz vectors (one pass
// instead of one H*v each).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <string>

#include "../../include/edgpu.h"
#include "hv_rows.cuh"

struct edg_sector {
  edg::Sector s;
};

namespace edg {

int fail(int code, const std::string& msg);
int cuda_fail(cudaError_t e, const char* what);

namespace {

// u[i*NV + q] = v[i*NV + q] / norm_i
template <typename Real, int NV>
__global__ void k_u_scale_blk(const typename CT2<Real>::T* __restrict__ v, const uint8_t* __restrict__ lid,
                              const double* __restrict__ nrm_inv_tab, int64_t n,
                              typename CT2<Real>::T* __restrict__ u) {
  __shared__ Real tab[65];
  for (int k = threadIdx.x; k < 65; k += blockDim.x) tab[k] = (Real)nrm_inv_tab[k];
  __syncthreads();
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n * NV; e += (int64_t)gridDim.x * blockDim.x) {
    typename CT2<Real>::T x = v[e];
    const Real s = tab[lid[e / NV]];
    x.x *= s;
    x.y *= s;
    u[e] = x;
  }
}

// Four entries of a row in flight for every vector (two in FP64 with four
// vectors): 16 to 32 registers of gathered entries beside the 8 NV partial sums.
// Two FP32 vectors take eight: at 28, 30 and 36 sites 175 -> 147 us, 678 -> 562 us
// and 85.0 -> 76.5 ms.
template <typename Real, int NV, int kPol, int kFmt>
cudaError_t launch_blk(const Sector& S, const void* v, void* w, void* u, cudaStream_t st) {
  using CT = typename CT2<Real>::T;
  const int64_t n = S.P.n_p;
  constexpr int kG = sizeof(Real) == 8 && NV == 4 ? 2 : sizeof(Real) == 4 && NV == 2 ? 8 : 4;
  constexpr int kU = kG == 8 ? 8 : 4;
  // rows that gather v itself: by 16-byte loads, so from a copy of an FP32 v that
  // starts between two of them
  if (S.folded) {
    if (u) {
      const cudaError_t e = cudaMemcpyAsync(u, v, sizeof(CT) * n * NV, cudaMemcpyDeviceToDevice, st);
      if (e != cudaSuccess) return e;
    }
    return launch_rows_k<Real, NV, true, kPol, kFmt, kU, kG, true>(S, v, u ? u : v, w, 0, n, st);
  }
  k_u_scale_blk<Real, NV><<<(int)std::min<int64_t>((n * NV + 255) / 256, 152 * 32), 256, 0, st>>>(
      reinterpret_cast<const CT*>(v), S.lid, params_field(S, offsetof(SectorParams, nrm_inv)), n,
      reinterpret_cast<CT*>(u));
  return launch_rows_k<Real, NV, true, kPol, kFmt, kU, kG, true>(S, v, u, w, 0, n, st);
}

template <typename Real, int NV>
cudaError_t launch_blk2(const Sector& S, const void* v, void* w, void* u, cudaStream_t st) {
  if (S.pack_cb)
    return S.csr_pol == 2 ? launch_blk<Real, NV, 2, kPacked>(S, v, w, u, st)
                          : launch_blk<Real, NV, 1, kPacked>(S, v, w, u, st);
  return S.csr_pol == 2 ? launch_blk<Real, NV, 2, kSplit>(S, v, w, u, st)
                        : launch_blk<Real, NV, 1, kSplit>(S, v, w, u, st);
}

}  // namespace

// W = H V for nv = 2 or 4 interleaved vectors on the stored rows; u is the
// caller's n_p * nv scratch (nullptr: folded rows and an aligned v need none).  The value table must fit in shared memory.
cudaError_t launch_hv_block(const Sector& S, const void* v, void* w, int nv, bool fp64, void* u, cudaStream_t st) {
  if (fp64) return nv == 2 ? launch_blk2<double, 2>(S, v, w, u, st) : launch_blk2<double, 4>(S, v, w, u, st);
  return nv == 2 ? launch_blk2<float, 2>(S, v, w, u, st) : launch_blk2<float, 4>(S, v, w, u, st);
}

}  // namespace edg

extern "C" int edg_hv_block(edg_sector* s, const void* v, void* w, int n_vectors, int dtype, void* stream) {
  using namespace edg;
  if (!s || !v || !w) return fail(EDG_ERR_INVALID, "NULL argument");
  if (dtype != EDG_C128 && dtype != EDG_C64) return fail(EDG_ERR_INVALID, "dtype must be EDG_C128 or EDG_C64");
  if (n_vectors != 2 && n_vectors != 4) return fail(EDG_ERR_INVALID, "edg_hv_block: n_vectors must be 2 or 4");
  if (v == w) return fail(EDG_ERR_INVALID, "v and w must not alias");
  Sector& S = s->s;
  if (!S.col) return fail(EDG_ERR_INVALID, "edg_hv_block needs stored rows (edg_sector_build_targets)");
  const bool fp64 = dtype == EDG_C128;
  if ((size_t)S.n_rvals * (fp64 ? 16 : 8) > 96 * 1024)
    return fail(EDG_ERR_UNSUPPORTED, "edg_hv_block: value table larger than 96 KB");
  const size_t bytes = (size_t)S.P.n_p * n_vectors * (fp64 ? 16 : 8);
  const bool scratch = !S.folded || reinterpret_cast<uintptr_t>(v) % 16 != 0;
  if (scratch && S.ublk.bytes < bytes) {
    if (S.ublk.ptr) cudaFree(S.ublk.ptr);
    S.ublk = DeviceBuffer{};
    if (cudaMalloc(&S.ublk.ptr, bytes) != cudaSuccess) {
      cudaGetLastError();
      return fail(EDG_ERR_NOMEM, "edg_hv_block: scratch of n_p x n_vectors entries");
    }
    S.ublk.bytes = bytes;
    S.device_bytes += bytes;
  }
  const cudaError_t e = launch_hv_block(S, v, w, n_vectors, fp64, scratch ? S.ublk.ptr : nullptr, (cudaStream_t)stream);
  if (e != cudaSuccess) return cuda_fail(e, "edg_hv_block launch");
  return EDG_OK;
}
