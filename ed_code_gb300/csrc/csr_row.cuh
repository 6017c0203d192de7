// Pieces of the stored-row H*v shared by the single-sector kernels
// (targets.cu), the batch (batch.cu) and the dense path (dense.cu): the
// complex type of a precision, the L2 cache policies of the loads, the layout
// of the stored rows and the sums over them.
//
// Layout.  The rows are cut into slices of 32 consecutive rows, a warp's worth.
// row_ptr holds the usual offsets (row i has row_ptr[i+1] - row_ptr[i]
// entries, slice s starts at row_ptr[32 s]); inside a slice the entries stand
// slot by slot: first the first entry of every row that has one, in row order,
// then the second entries, and so on, with no padding.  A warp sums a slice
// with a lane per row: slot k is one coalesced load (its rows are the ballot
// of "more than k entries"), the sums need no exchange between lanes, and a
// row's entries are in the order of the flip groups, high sites first, so that
// one slot's gathers in neighbouring rows mostly go to neighbouring columns.
//
// With 8 to 32 lanes per row instead (entries row by row, a shuffle reduction
// per row) every gather instruction went to 32 unrelated places and, in FP64,
// the reductions took a quarter to a half of the FP64 issue that bounds it.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace edg {
namespace {

template <typename Real>
struct CT2;
template <>
struct CT2<float> { using T = float2; };
template <>
struct CT2<double> { using T = double2; };

// Cache policy of the row loads (tuned per sector).  The row data (col, vid)
// are read once per H*v; the gathered u entries are reused by other rows while
// they stay in L2.  Policy 1 reads the row data with the streaming hint
// (ld.global.cs); policy 2 gives them the L2 evict_first priority instead.
// Both give the u gathers L2 evict_last.
__device__ __forceinline__ uint64_t l2_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t l2_evict_last() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
template <int kPol>
__device__ __forceinline__ uint32_t ld_row(const uint32_t* a, uint64_t pol) {
  if (kPol == 1) return __ldcs(a);
  uint32_t r;
  asm volatile("ld.global.nc.L2::cache_hint.u32 %0, [%1], %2;" : "=r"(r) : "l"(a), "l"(pol));
  return r;
}
template <int kPol>
__device__ __forceinline__ int ld_row(const uint16_t* a, uint64_t pol) {
  if (kPol == 1) return __ldcs(a);
  uint16_t r;
  asm volatile("ld.global.nc.L2::cache_hint.u16 %0, [%1], %2;" : "=h"(r) : "l"(a), "l"(pol));
  return r;
}
// NV consecutive complex entries at a (16-byte loads for NV > 1, whose u is
// this library's own scratch)
template <int NV>
__device__ __forceinline__ void ld_keep(const float2* a, uint64_t pol, float (&x)[2 * NV]) {
  if (NV == 1) {
    asm volatile("ld.global.nc.L2::cache_hint.v2.f32 {%0, %1}, [%2], %3;" : "=f"(x[0]), "=f"(x[1]) : "l"(a), "l"(pol));
  } else {
#pragma unroll
    for (int k = 0; k < NV; k += 2)
      asm volatile("ld.global.nc.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
                   : "=f"(x[2 * k]), "=f"(x[2 * k + 1]), "=f"(x[(2 * k + 2) % (2 * NV)]), "=f"(x[(2 * k + 3) % (2 * NV)])
                   : "l"(a + k), "l"(pol));
  }
}
template <int NV>
__device__ __forceinline__ void ld_keep(const double2* a, uint64_t pol, double (&x)[2 * NV]) {
#pragma unroll
  for (int k = 0; k < NV; ++k)
    asm volatile("ld.global.nc.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;"
                 : "=d"(x[2 * k]), "=d"(x[2 * k + 1])
                 : "l"(a + k), "l"(pol));
}

// acc += c * x for complex c, x, as explicit FMAs in a fixed order, so every
// kernel that sums rows (single vector, block, batch) rounds the same way
// whatever the compiler would have contracted.
__device__ __forceinline__ float fmaR(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fmaR(double a, double b, double c) { return fma(a, b, c); }
// a row's result: norm_i * sum + Ezz_i * v_i
template <typename Real, typename CT>
__device__ __forceinline__ CT row_out(Real ar, Real ai, Real ni, Real d, const CT& vi) {
  CT out;
  out.x = fmaR(ar, ni, d * vi.x);
  out.y = fmaR(ai, ni, d * vi.y);
  return out;
}

// Entry formats of the stored rows.  kSplit: a u32 column array and a u16
// value-id array (6 bytes an entry).  kPacked: one u32 an entry, the column
// in the low cb bits and the value id above them (4 bytes), used when the
// deduplicated value table and the sector size leave room (cb < 32 and
// n_p < 2^cb).  kByVid: either, chosen per segment by vid == nullptr (the
// batch, whose segments may differ).
constexpr int kSplit = 0, kPacked = 1, kByVid = 2;

// A sector's stored rows as the sums read them.
template <typename Real>
struct RowsView {
  const uint64_t* row_ptr;
  const uint32_t* col;
  const uint16_t* vid;
  const typename CT2<Real>::T* vtab;  // global or shared memory
  const typename CT2<Real>::T* u;     // v / norm, NV vectors interleaved
  int cb;
};

// Where a warp's slice of rows stands: this lane's row length, the slots that
// all 32 rows have (mn) and that any has (mx), and the slice's first entry.
struct Slice {
  uint64_t base;
  int len, mn, mx;
};
__device__ __forceinline__ Slice slice_at(const uint64_t* __restrict__ row_ptr, int64_t i, int64_t n) {
  const unsigned long long* rp = reinterpret_cast<const unsigned long long*>(row_ptr);
  unsigned long long b = 0, e = 0;
  if (i < n) {
    b = __ldg(rp + i);
    e = __ldg(rp + i + 1);
  }
  Slice s;
  s.len = (int)(e - b);
  s.mn = (int)__reduce_min_sync(0xffffffffu, (unsigned)s.len);
  s.mx = (int)__reduce_max_sync(0xffffffffu, (unsigned)s.len);
  s.base = __shfl_sync(0xffffffffu, b, 0);  // lane 0's row exists whenever the slice does
  return s;
}

// Partial sums of a row.  FP64: slot k goes into sum (k - lo) mod 4.  FP32: every
// four slots are summed on their own, and these sums go into two partial sums
// in turn; that keeps the rounding error of eight chains (a row's error grows
// with the length of its chains) in a third of their registers, for an addition
// per four slots, which in FP64 would cost an eighth of its issue.
template <typename Real>
__host__ __device__ constexpr int partial_sums() {
  return sizeof(Real) == 4 ? 2 : 4;
}

// The bits of x that say it is not zero, hidden from the optimiser, which would
// make a comparison on the FP64 pipe of it.
__device__ __forceinline__ uint32_t nonzero_bits(double x) {
  uint32_t lo, hi;
  asm volatile("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "d"(x));
  return lo | (hi << 1);
}
__device__ __forceinline__ uint32_t nonzero_bits(float) { return 1u; }

// kB slots' products into the partial sums: gathered kG at a time, this lane
// has the slots in act.  In FP64 a batch whose values are all real in the warp
// takes half the multiply-adds (the products with a zero imaginary part add
// nothing to a finite sum): FP64 issue, 16 clocks a warp instruction and SM
// whether or not it is predicated off, is what bounds it, so the test is on a
// whole batch, which is then a branch and not predicated.
template <typename Real, int NV, int kFmt, int kB, int kG>
__device__ __forceinline__ void take_slots(const RowsView<Real>& R, const uint32_t (&e)[kB], const uint16_t (&h)[kB],
                                           uint32_t act, uint32_t cmask, bool packed, uint64_t pl,
                                           Real (&acc)[partial_sums<Real>()][2 * NV]) {
  using CT = typename CT2<Real>::T;
  constexpr int kAcc = partial_sums<Real>();
  static_assert(kB % 4 == 0 && kB % kG == 0, "whole fours and groups of gathers");
  Real four[2 * NV];
#pragma unroll
  for (int q0 = 0; q0 < kB; q0 += kG) {
    Real x[kG][2 * NV];
    CT c[kG];
#pragma unroll
    for (int q = 0; q < kG; ++q) {
#pragma unroll
      for (int k = 0; k < 2 * NV; ++k) x[q][k] = 0;
      if ((act >> (q0 + q)) & 1u) ld_keep<NV>(R.u + (int64_t)(e[q0 + q] & cmask) * NV, pl, x[q]);
    }
    uint32_t im = 0;
#pragma unroll
    for (int q = 0; q < kG; ++q) {
      c[q].x = 0;
      c[q].y = 0;
      if ((act >> (q0 + q)) & 1u) c[q] = R.vtab[packed ? e[q0 + q] >> R.cb : (uint32_t)h[q0 + q]];
      im |= nonzero_bits(c[q].y);
    }
    if (sizeof(Real) == 4 || __any_sync(0xffffffffu, im != 0)) {
#pragma unroll
      for (int q = 0; q < kG; ++q) {
        Real(&a)[2 * NV] = sizeof(Real) == 4 ? four : acc[(q0 + q) % kAcc];
        if (sizeof(Real) == 4 && (q0 + q) % 4 == 0) {
#pragma unroll
          for (int k = 0; k < 2 * NV; ++k) a[k] = 0;
        }
#pragma unroll
        for (int k = 0; k < NV; ++k) {
          a[2 * k] = fmaR(c[q].x, x[q][2 * k], fmaR(-c[q].y, x[q][2 * k + 1], a[2 * k]));
          a[2 * k + 1] = fmaR(c[q].x, x[q][2 * k + 1], fmaR(c[q].y, x[q][2 * k], a[2 * k + 1]));
        }
        if (sizeof(Real) == 4 && (q0 + q) % 4 == 3) {
#pragma unroll
          for (int k = 0; k < 2 * NV; ++k) acc[(q0 + q) / 4 % kAcc][k] += a[k];
        }
      }
    } else {
#pragma unroll
      for (int q = 0; q < kG; ++q)
#pragma unroll
        for (int k = 0; k < 2 * NV; ++k)
          acc[(q0 + q) % kAcc][k] = fmaR(c[q].x, x[q][k], acc[(q0 + q) % kAcc][k]);
    }
  }
  if (sizeof(Real) == 4 && kB % 8 != 0) {  // the next four go into the other sum
#pragma unroll
    for (int k = 0; k < 2 * NV; ++k) {
      const Real t = acc[0][k];
      acc[0][k] = acc[1][k];
      acc[1][k] = t;
    }
  }
}

// Sums of a slice's slots [lo, hi) in this lane's row: sum[2k], sum[2k+1] of
// vector k.  Slots that every row has come kU at a time, gathered kG at a time;
// kPipe loads the next kU entries before the current ones are gathered.  The
// rest come four at a time.  The result does not depend on kU, kG or kPipe.
template <typename Real, int NV, int kFmt, int kPol, int kU, int kG, bool kPipe>
__device__ __forceinline__ void slice_sums(const RowsView<Real>& R, const Slice& s, int lo, int hi, uint64_t pf,
                                           uint64_t pl, Real (&sum)[2 * NV]) {
  constexpr int kAcc = partial_sums<Real>(), kT = 4, kGT = kG < kT ? kG : kT;
  const bool packed = kFmt == kPacked || (kFmt == kByVid && R.vid == nullptr);
  const uint32_t cmask = packed ? (1u << R.cb) - 1u : 0xFFFFFFFFu;
  const int lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  Real acc[kAcc][2 * NV];
#pragma unroll
  for (int a = 0; a < kAcc; ++a)
#pragma unroll
    for (int k = 0; k < 2 * NV; ++k) acc[a][k] = 0;

  // slots that every row has: entry 32 k + lane
  int k = lo;
  const int full = min(s.mn, hi);
  uint64_t at = s.base + (uint64_t)32 * min(lo, s.mn);
  if (k + kU <= full) {
    uint32_t e[kU];
    uint16_t h[kU];
    auto load = [&](uint32_t(&e2)[kU], uint16_t(&h2)[kU], uint64_t p) {
#pragma unroll
      for (int q = 0; q < kU; ++q) {
        e2[q] = ld_row<kPol>(R.col + p + 32 * q + lane, pf);
        h2[q] = packed ? (uint16_t)0 : (uint16_t)ld_row<kPol>(R.vid + p + 32 * q + lane, pf);
      }
    };
    load(e, h, at);
    while (true) {
      k += kU;
      at += 32 * kU;
      const bool more = k + kU <= full;
      if (kPipe && more) {
        uint32_t en[kU];
        uint16_t hn[kU];
        load(en, hn, at);
        take_slots<Real, NV, kFmt, kU, kG>(R, e, h, 0xFFFFFFFFu, cmask, packed, pl, acc);
#pragma unroll
        for (int q = 0; q < kU; ++q) {
          e[q] = en[q];
          h[q] = hn[q];
        }
      } else {
        take_slots<Real, NV, kFmt, kU, kG>(R, e, h, 0xFFFFFFFFu, cmask, packed, pl, acc);
        if (!more) break;
        load(e, h, at);
      }
    }
  }
  // the others: the rows that have a slot, by ballot
  for (int b = s.mn; b < k; ++b) at += __popc(__ballot_sync(0xffffffffu, s.len > b));  // (lo past mn)
  for (; k < hi; k += kT) {
    uint32_t e[kT];
    uint16_t h[kT];
    uint32_t act = 0;
#pragma unroll
    for (int q = 0; q < kT; ++q) {
      const bool has = k + q < hi && s.len > k + q;
      const uint32_t m = __ballot_sync(0xffffffffu, has);
      e[q] = 0;
      h[q] = 0;
      if (has) {
        const uint64_t p = at + __popc(m & lt);
        e[q] = ld_row<kPol>(R.col + p, pf);
        if (!packed) h[q] = (uint16_t)ld_row<kPol>(R.vid + p, pf);
        act |= 1u << q;
      }
      at += __popc(m);
    }
    take_slots<Real, NV, kFmt, kT, kGT>(R, e, h, act, cmask, packed, pl, acc);
  }
  // (a + b is b + a, so it does not matter which of FP32's two comes last)
#pragma unroll
  for (int j = 0; j < 2 * NV; ++j) {
#pragma unroll
    for (int a = 0; a < kAcc / 2; ++a) acc[a][j] += acc[a + kAcc / 2][j];
    sum[j] = kAcc == 2 ? acc[0][j] : acc[0][j] + acc[1][j];
  }
}

// Warps that share a slice of a sector of n rows, whose sums are added in warp
// order.  A function of the size alone, so every kernel on one sector adds in
// the same order.
//  * A sector of a few thousand rows has too few slices to fill the chip with a
//    warp each, and a row's entries would be one long chain of loads.  The
//    lines lie where the next split stops paying (FP64, us per H v with 1, 2,
//    4, 8 warps): 3,520 slices 47.1, 51.3, 56.0, 77.3; 290 slices 20.5, 16.4,
//    13.7, 14.4; 26 slices 13.7, 11.2, 10.7, 10.6.
//  * A u far larger than the L2 (64 M rows are 512 MB in FP32) is read through
//    the window that the rows in flight touch: half the rows in flight took
//    53.2 ms instead of 58.6 ms at 36 sites (2.5e8 rows).  At 32 sites (1.9e7
//    rows, u 150 MB) the split cost 2.05 ms against 1.87 ms.
__host__ __device__ inline int warps_per_slice(int64_t n) {
  const int64_t slices = (n + 31) / 32;
  if (n >= (int64_t)1 << 26) return 2;
  return slices >= 152 * 8 ? 1 : slices >= 152 * 4 ? 2 : slices >= 152 ? 4 : 8;
}

}  // namespace
}  // namespace edg
