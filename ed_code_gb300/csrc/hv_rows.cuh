// The stored-row H*v kernel on 1, 2 or 4 vectors (targets.cu, hv_block.cu).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>

#include "csr_row.cuh"
#include "edg_sector.cuh"
#include "launch.cuh"

namespace edg {

namespace {

constexpr int kRowThreads = 256, kRowWarps = kRowThreads / 32;

// w_i = norm_i * sum_t vtab[vid_t] * u[col_t] + Ezz_i * v_i (u = v / norm, or v
// itself where the values include the targets' 1/norm) for the rows
// [row0, row1) of n, row0 a multiple of 32: a warp per slice of 32 rows, or
// wps warps with a share of its slots each (warps_per_slice).  NV vectors are
// interleaved by row (entry i of vector q at i * NV + q); each gets the bits
// that NV = 1 gives it alone.
//
// The CTAs stride over the slices, 8 / wps neighbouring ones at a time, so the
// columns that neighbouring rows share meet in one SM's L1 (0.33 u sectors per
// nonzero instead of 0.68 reach L2 on a 28-site sector), and the grid sets how
// many rows are in flight: fewer keep the window of u their targets touch in
// L2, which the largest sectors need.
//
// Measured against 8 to 32 lanes per row: FP64 at 28 sites 1,085 -> 533 us (528
// with more entries in flight; 4 FMAs a nonzero are 460 us of FP64 issue), real
// values 926 -> 226 us; FP32 at 30 sites 593 -> 392 us (L1 66 % busy, 0.52
// sectors a nonzero from L2), at 36 sites 60.5 -> 55.3 ms (DRAM: the
// re-translated targets miss L2); four FP32 vectors at 32 sites 5.68 -> 4.03 ms.
// Folded rows (targets.cu) took another 10 us off the first, 17 us off 30 sites
// and 0.17 ms off the block: the pass over v and its launch.
// 256 threads: 512 and 1,024 left fewer warps an SM (30 sites 445 us), and a
// register cap that would fit more CTAs measured 408 us.
template <typename Real, int NV, bool kSmemTab, int kPol, int kFmt, int kU, int kG, bool kPipe>
__global__ void __launch_bounds__(kRowThreads) k_hv_rows(RowsView<Real> R, int n_vals, const double* __restrict__ ezz,
                                                         const uint8_t* __restrict__ lid,
                                                         const double* __restrict__ nrm_tab, int64_t row0,
                                                         int64_t row1, int wps,
                                                         const typename CT2<Real>::T* __restrict__ v,
                                                         typename CT2<Real>::T* __restrict__ w) {
  using CT = typename CT2<Real>::T;
  extern __shared__ __align__(16) uint8_t sm[];
  __shared__ Real nrm[65];
  __shared__ Real red[kRowWarps][2 * NV][32];
  CT* tab = reinterpret_cast<CT*>(sm);
  for (int k = threadIdx.x; k < 65; k += blockDim.x) nrm[k] = (Real)nrm_tab[k];
  if (kSmemTab) {
    for (int k = threadIdx.x; k < n_vals; k += blockDim.x) tab[k] = R.vtab[k];
    R.vtab = tab;
  }
  __syncthreads();
  const uint64_t pf = kPol == 2 ? l2_evict_first() : 0, pl = l2_evict_last();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int per_cta = kRowWarps / wps, part = wid % wps;
  for (int64_t s0 = row0 / 32 + (int64_t)blockIdx.x * per_cta; s0 * 32 < row1; s0 += (int64_t)gridDim.x * per_cta) {
    const int64_t i = (s0 + wid / wps) * 32 + lane;
    const Slice s = slice_at(R.row_ptr, i, row1);
    CT vi[NV];
    Real ni = 0, d = 0;
    if (part == 0 && i < row1) {  // in flight during the sums
#pragma unroll
      for (int k = 0; k < NV; ++k) vi[k] = v[i * NV + k];
      ni = nrm[lid[i]];
      d = (Real)ezz[i];
    }
    int lo = 0, hi = s.mx;
    if (wps > 1) {
      const int share = (s.mx + wps - 1) / wps;
      lo = min(s.mx, part * share);
      hi = min(s.mx, lo + share);
    }
    Real sum[2 * NV];
    slice_sums<Real, NV, kFmt, kPol, kU, kG, kPipe>(R, s, lo, hi, pf, pl, sum);
    if (wps > 1) {
#pragma unroll
      for (int k = 0; k < 2 * NV; ++k) red[wid][k][lane] = sum[k];
      __syncthreads();
      if (part == 0)
        for (int p = 1; p < wps; ++p)
#pragma unroll
          for (int k = 0; k < 2 * NV; ++k) sum[k] += red[wid + p][k][lane];
      __syncthreads();
    }
    if (part == 0 && i < row1) {
#pragma unroll
      for (int k = 0; k < NV; ++k) w[i * NV + k] = row_out(sum[2 * k], sum[2 * k + 1], ni, d, vi[k]);
    }
  }
}

inline const double* params_field(const Sector& S, size_t offset) {
  return reinterpret_cast<const double*>(reinterpret_cast<const char*>(S.dP) + offset);
}

template <typename Real>
RowsView<Real> rows_of(const Sector& S, const void* u) {
  using CT = typename CT2<Real>::T;
  const CT* tab = reinterpret_cast<const CT*>(sizeof(Real) == 8 ? (const void*)S.rtab64 : (const void*)S.rtab32);
  return RowsView<Real>{S.row_ptr, S.col, S.vid, tab, reinterpret_cast<const CT*>(u), S.pack_cb};
}

// Grid of the row kernel: the CTAs that fit on every SM at once, at most cap
// per SM when cap > 0, no more than the slices need; without a cap, several
// turns of them, as slices differ in their length and their gathers' misses and
// one turn ends in a tail of few CTAs.  FP64 takes 8 turns with one or two
// vectors (28 sites 520 -> 497 us, 30 sites 1,937 -> 1,854 us, 36 sites 122.7 ->
// 112.7 ms); FP32, and FP64 with four (28 sites 1,196 -> 1,253 us with 8), as many, up to 8, as leave a warp 64 slices, for every turn
// starts its loads anew (36 sites 54.8 -> 52.3 ms; 8 turns at 30 sites, with
// 5 slices a warp, 374 -> 385 us).
template <typename Real, int NV, typename K>
int rows_grid(K kernel, size_t smem, int64_t slices, int per_cta, int cap) {
  Resident r = resident((const void*)kernel, kRowThreads, smem, 96 * 1024);
  if (cap > 0 && r.per_sm > cap) r.per_sm = cap;
  const int64_t want = (slices + per_cta - 1) / per_cta;
  const int64_t once = (int64_t)r.sms * r.per_sm;
  const int64_t most = sizeof(Real) == 8 && NV <= 2 ? 8 : std::min<int64_t>(8, slices / (64 * once * per_cta));
  return (int)std::max<int64_t>(1, std::min<int64_t>(want, once * (cap > 0 ? 1 : std::max<int64_t>(1, most))));
}

// rows [r0, r1) of w = H v from u = v / norm
template <typename Real, int NV, bool kSmemTab, int kPol, int kFmt, int kU, int kG, bool kPipe>
cudaError_t launch_rows_k(const Sector& S, const void* v, const void* u, void* w, int64_t r0, int64_t r1,
                          cudaStream_t st) {
  using CT = typename CT2<Real>::T;
  if (r1 <= r0) return cudaGetLastError();
  const int wps = warps_per_slice(S.P.n_p);
  const size_t smem = kSmemTab ? sizeof(CT) * S.n_rvals : 0;
  auto kern = k_hv_rows<Real, NV, kSmemTab, kPol, kFmt, kU, kG, kPipe>;
  const int grid = rows_grid<Real, NV>(kern, smem, (r1 - r0 + 31) / 32, kRowWarps / wps, S.csr_cps);
  kern<<<grid, kRowThreads, smem, st>>>(rows_of<Real>(S, u), S.n_rvals, S.ezz, S.lid,
                                        params_field(S, offsetof(SectorParams, nrm)), r0, r1, wps,
                                        reinterpret_cast<const CT*>(v), reinterpret_cast<CT*>(w));
  return cudaGetLastError();
}

}  // namespace

}  // namespace edg
