// Inner products of one vector with many (Gram-Schmidt coefficients, alpha,
// norms) in one kernel, the sums closed on the device, shared by the plain and
// the mixed-precision Lanczos.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "blas1.cuh"
#include "ff.cuh"

namespace edg {
namespace {

constexpr int kMdThreads = 256, kMdWarps = kMdThreads / 32;
constexpr int kMdE = 4;    // elements a thread holds at a time
constexpr int kMdChunk = kMdThreads * kMdE;
constexpr int kMdMaxCtas = 152 * 3;

// How a policy accumulates conj(a) b over four elements at a time (of an
// even or an odd chunk) and sums the accumulators of a warp.
struct Md32 {  // FP32 vectors, exact products in float-float
  static constexpr int kK = 8;     // vectors a group
  static constexpr int kCtas = 3;  // resident an SM
  using V = float2;
  struct A {
    FFAcc re, im;
  };
  template <bool kOdd>
  static __device__ __forceinline__ void take(A& s, const V (&a)[kMdE], const V (&b)[kMdE]) {
#pragma unroll
    for (int q = 0; q < kMdE; ++q) {
      s.re.add_prod(a[q].x, b[q].x);
      s.re.add_prod(a[q].y, b[q].y);
      s.im.add_prod(a[q].x, b[q].y);
      s.im.sub_prod(a[q].y, b[q].x);
    }
  }
  // float-float values: one sum's error is about 2^-48 of the magnitudes, as the
  // accumulation's
  struct S {
    float hi, lo;
  };
  static __device__ __forceinline__ S of(const FFAcc& x) { return S{x.hi, x.lo}; }
  static __device__ __forceinline__ S shfl(S x, int o) {
    return S{__shfl_xor_sync(0xffffffffu, x.hi, o), __shfl_xor_sync(0xffffffffu, x.lo, o)};
  }
  static __device__ __forceinline__ S add(S x, S y) {
    float s, e;
    two_sum(x.hi, y.hi, s, e);
    return S{s, __fadd_rn(__fadd_rn(x.lo, y.lo), e)};
  }
  static __device__ __forceinline__ double value(S x) { return (double)x.hi + (double)x.lo; }
};
// FP64 vectors: the products of four elements in a chain of FMAs, an even and an
// odd chunk's chains added up, and these added with compensation (two-sum).  FP64
// issue (16 clocks a warp instruction and SM) is what bounds it: 5.75
// instructions a complex product, against 16 with every sum compensated; the
// rounding errors are those of six plain additions' levels, no more than the
// trees over a thread per element had.
struct Md64 {
  static constexpr int kK = 4, kCtas = 2;
  using V = double2;
  struct One {
    double s = 0.0, c = 0.0, t = 0.0;
    template <bool kOdd>
    __device__ __forceinline__ void add(double x) {
      if (!kOdd) {
        t = x;
        return;
      }
      x += t;
      t = 0.0;
      const double n = s + x, b = n - s;
      c += (s - (n - b)) + (x - b);
      s = n;
    }
    __device__ __forceinline__ double value() const { return s + c; }
  };
  struct A {
    One re, im;
  };
  template <bool kOdd>
  static __device__ __forceinline__ void take(A& s, const V (&a)[kMdE], const V (&b)[kMdE]) {
    double r = 0.0, i = 0.0;
#pragma unroll
    for (int q = 0; q < kMdE; ++q) {
      r = fma(a[q].x, b[q].x, r);
      r = fma(a[q].y, b[q].y, r);
      i = fma(a[q].x, b[q].y, i);
      i = fma(-a[q].y, b[q].x, i);
    }
    s.re.template add<kOdd>(r);
    s.im.template add<kOdd>(i);
  }
  using S = double;
  static __device__ __forceinline__ S of(const One& x) { return x.value(); }
  static __device__ __forceinline__ S shfl(S x, int o) { return __shfl_xor_sync(0xffffffffu, x, o); }
  static __device__ __forceinline__ S add(S x, S y) { return x + y; }
  static __device__ __forceinline__ double value(S x) { return x; }
};

// The CTA that takes the last of `total` tickets goes on (and resets the
// counter); no CTA waits for another.
__device__ __forceinline__ bool md_last(int* cnt, int64_t total) {
  __shared__ int last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(cnt, 1) == (int)(total - 1);
    if (last) *cnt = 0;
  }
  __syncthreads();
  const bool r = last != 0;
  if (r) __threadfence();
  __syncthreads();
  return r;
}

// What becomes of the sums: value k (2 per vector, from vector k0 on).
enum { kMdComplex = 0, kMdReal = 1, kMdNorm = 2, kMdInvNorm = 3 };
__device__ __forceinline__ void md_store(double* out, int k0, int k, int mode, double a) {
  if (mode == kMdComplex) out[2 * k0 + k] = a;
  else if (k == 0) out[0] = mode == kMdReal ? a : mode == kMdNorm ? sqrt(a) : 1.0 / sqrt(a);
}

// out_k = <V_k|x>, k in [kf, K) (kf on the device, or 0), V_k = V + k ld.
//
// The work is groups of up to eight (FP64: four) vectors, each in chunks of 1,024 elements,
// cut into one even range per CTA of a grid that fills the chip: a range is a
// few segments of consecutive chunks of one group.  A thread holds four
// elements of x in registers while it takes those of each vector, so x is read
// from L2 once per group; a segment ends with one sum over the CTA, in
// which a warp closes its sums by an exchange that halves them at every step (16
// additions instead of 80 for 16 sums).  With kf set on the device most vectors are not
// wanted in most steps: a grid over (tiles, vectors) would be mostly CTAs that
// return at once.  The CTA that finishes a group's last segment sums its
// segments in order; with decide, the one that finishes the last group also
// says whether a second Gram-Schmidt pass is needed (Daniel, Gragg, Kaufman and
// Stewart's test: the first removed more than 1e-4 of |x|^2).
// part: md_part doubles; cnt: md_cnt ints, zero between launches.
//
// Bound by FP32 issue (40 instructions a float-float product) or FP64 issue.
// 300 FP32 vectors of 1.43e6 states: 3.1 ms with a CTA per vector and 1,400
// elements (its FP64 tree over the threads was most of it), 2.5 ms by tiles with
// a ticket each, 0.69 ms (5.0 TB/s) by ranges; 100 FP64 vectors of 112,632
// states 1.05 ms -> 0.15 ms.
template <class P>
__global__ void __launch_bounds__(kMdThreads, P::kCtas) k_mdot(const typename P::V* __restrict__ V, int64_t ld,
                                                               const typename P::V* __restrict__ x, int64_t n, int K,
                                                               double* __restrict__ part, double* __restrict__ out,
                                                               int mode, int* __restrict__ cnt, const double* run,
                                                               const int* kf, double* decide, const double* xn2) {
  using Vt = typename P::V;
  constexpr int kK = P::kK;
  if (run && *run == 0.0) return;
  const int first = kf ? *kf : 0;
  const int groups = (K - first + kK - 1) / kK;
  const int64_t chunks = (n + kMdChunk - 1) / kMdChunk, units = groups * chunks;
  const int64_t ctas = min((int64_t)gridDim.x, units);
  if (blockIdx.x >= ctas) return;
  // CTA c has the units [c units / ctas, (c + 1) units / ctas)
  auto cta_of = [&](int64_t u) { return ((u + 1) * ctas - 1) / units; };
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __shared__ double sums[kMdWarps][2 * kK];
  const int64_t u1 = (blockIdx.x + 1) * units / ctas;
  for (int64_t u = blockIdx.x * units / ctas; u < u1;) {
    const int g = (int)(u / chunks);
    const int64_t c0 = u - g * chunks, c1 = min(chunks, c0 + (u1 - u));
    u += c1 - c0;
    const int k0 = first + g * kK, nk = min(kK, K - k0);
    typename P::A acc[kK];
    const Vt* v = V + (int64_t)k0 * ld + threadIdx.x;
    int64_t i0 = c0 * kMdChunk;
    const int64_t end = min(n, c1 * kMdChunk);
    auto chunk = [&](auto is_odd) {  // all elements and vectors there: the next vector's loads ahead
      constexpr bool kOdd = decltype(is_odd)::value;
      Vt b[kMdE], a[2][kMdE];
#pragma unroll
      for (int q = 0; q < kMdE; ++q) {
        b[q] = x[i0 + q * kMdThreads + threadIdx.x];
        a[0][q] = __ldcs(v + i0 + q * kMdThreads);
      }
#pragma unroll
      for (int k = 0; k < kK; ++k) {
        if (k + 1 < kK) {
#pragma unroll
          for (int q = 0; q < kMdE; ++q) a[(k + 1) & 1][q] = __ldcs(v + (int64_t)(k + 1) * ld + i0 + q * kMdThreads);
        }
        P::template take<kOdd>(acc[k], a[k & 1], b);
      }
      i0 += kMdChunk;
    };
    if (nk == kK)
      while (i0 + 2 * kMdChunk <= end) {
        chunk(std::false_type{});
        chunk(std::true_type{});
      }
    for (; i0 < end; i0 += kMdChunk) {
      Vt b[kMdE];
      bool in[kMdE];
#pragma unroll
      for (int q = 0; q < kMdE; ++q) {
        const int64_t i = i0 + q * kMdThreads + threadIdx.x;
        in[q] = i < end;
        b[q].x = b[q].y = 0;
        if (in[q]) b[q] = x[i];
      }
#pragma unroll
      for (int k = 0; k < kK; ++k) {
        if (k >= nk) break;
        Vt a[kMdE];
#pragma unroll
        for (int q = 0; q < kMdE; ++q) {
          a[q].x = a[q].y = 0;
          if (in[q]) a[q] = __ldcs(v + (int64_t)k * ld + i0 + q * kMdThreads);
        }
        P::template take<true>(acc[k], a, b);
      }
    }
    // 2 kK sums over 32 lanes: every exchange halves them, then the lanes that
    // hold the same value (kLanes of them, value lane / kLanes) add up
    constexpr int kLanes = 16 / kK;
    typename P::S s[2 * kK];
#pragma unroll
    for (int k = 0; k < kK; ++k) {
      s[2 * k] = P::of(acc[k].re);
      s[2 * k + 1] = P::of(acc[k].im);
    }
#pragma unroll
    for (int o = 16, w = kK; o >= kLanes; o >>= 1, w >>= 1) {
      const bool up = lane & o;
#pragma unroll
      for (int j = 0; j < kK; ++j)
        if (j < w) {
          const typename P::S keep = up ? s[w + j] : s[j], give = up ? s[j] : s[w + j];
          s[j] = P::add(keep, P::shfl(give, o));
        }
    }
#pragma unroll
    for (int o = kLanes / 2; o > 0; o >>= 1) s[0] = P::add(s[0], P::shfl(s[0], o));
    if (lane % kLanes == 0) sums[wid][lane / kLanes] = P::value(s[0]);
    __syncthreads();
    const int64_t cf = cta_of(g * chunks), segs = cta_of((g + 1) * chunks - 1) - cf + 1;
    if (threadIdx.x < 2 * nk) {
      double a = 0;
#pragma unroll
      for (int w = 0; w < kMdWarps; ++w) a += sums[w][threadIdx.x];
      part[((int64_t)k0 * 2 + threadIdx.x) * kMdMaxCtas + (blockIdx.x - cf)] = a;
    }
    if (md_last(cnt + 1 + g, segs)) {
      for (int k = wid; k < 2 * nk; k += kMdWarps) {  // a warp per value
        const double* p = part + ((int64_t)k0 * 2 + k) * kMdMaxCtas;
        double a = 0;
        for (int64_t q = lane; q < segs; q += 32) a += __ldcg(p + q);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
        if (lane == 0) md_store(out, k0, k, mode, a);
      }
      if (decide && md_last(cnt, groups)) {
        __shared__ double sq[kMdThreads];
        double a = 0;
        for (int k = first + threadIdx.x; k < K; k += blockDim.x) {
          const double re = __ldcg(out + 2 * k), im = __ldcg(out + 2 * k + 1);
          a += re * re + im * im;
        }
        sq[threadIdx.x] = a;
        __syncthreads();
        for (int h = kMdThreads / 2; h > 0; h >>= 1) {
          if ((int)threadIdx.x < h) sq[threadIdx.x] += sq[threadIdx.x + h];
          __syncthreads();
        }
        if (threadIdx.x == 0) *decide = sq[0] > 1e-4 * *xn2 ? 1.0 : 0.0;
      }
    }
    __syncthreads();  // sums is reused by the next segment
  }
}

// Doubles of partials and ints of counters that k_mdot needs for K vectors.
inline size_t md_part(int K) { return (size_t)2 * K * kMdMaxCtas; }
inline size_t md_cnt(int K) { return 1 + (K + 3) / 4; }

template <class P>
void mdot(cudaStream_t st, const typename P::V* V, int64_t ld, int K, const typename P::V* x, int64_t n, double* part,
          int* cnt, double* out, int mode, const double* run = nullptr, const int* kf = nullptr,
          double* decide = nullptr, const double* xn2 = nullptr) {
  const int64_t units = (n + kMdChunk - 1) / kMdChunk * ((K + P::kK - 1) / P::kK);
  k_mdot<P><<<(unsigned)std::min<int64_t>(units, 152 * P::kCtas), kMdThreads, 0, st>>>(V, ld, x, n, K, part, out, mode,
                                                                                     cnt, run, kf, decide, xn2);
}

}  // namespace
}  // namespace edg
