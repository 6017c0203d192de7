// Real symmetric tridiagonal eigenproblem for the Lanczos T matrix.
//
// The reference rebuilds T (diagonal Re(alpha_j), off-diagonal beta_{j+1})
// and diagonalises it completely with LAPACK zheev at every iteration
// (lanczos.cpp:271-286), but only ever uses the lowest eigenvalue and, at the
// end of a cycle, its eigenvector (lanczos.cpp:286-318).  Here:
//   * eigenvalues: multisection on the count of sign changes of the leading
//     minors (Givens; Barth, Martin and Wilkinson's Sturm counts, Numer. Math. 9
//     (1967) 386, without their quotients), a warp each;
//   * eigenvector: inverse iteration with a tridiagonal LU factorisation with
//     partial pivoting (Wilkinson, "The Algebraic Eigenvalue Problem", 1965,
//     ch. 9), two sweeps from a fixed start vector.
// Host and device share the code; everything is FP64.
#pragma once
#include <math.h>
#include <stdint.h>

#if defined(__CUDACC__)
#define TD_HD __host__ __device__ inline
#else
#define TD_HD inline
#endif

namespace edg {

#if defined(__CUDACC__)
// Counts of eigenvalues below x from the signs of the leading minors
// p_i = det(T_i - x), p_i = (d_i - x) p_{i-1} - e_{i-1}^2 p_{i-2}, in FP32 or FP64:
// a sign change from p_{i-1} to p_i is an eigenvalue below x (a zero minor counts
// once whichever sign it is given).  e2[i] couples rows i and i + 1.  No division
// -- the Sturm quotients d_i - x - e^2 / q are a chain of FP64 divisions, about
// 1,200 clocks a row -- and no comparison on the FP64 pipe: signs and exponents
// are read as integers, and every four rows the pair is rescaled by a power of
// two.  A row's chain is one multiply-add.
__device__ __forceinline__ uint32_t sign_exp(float x) { return __float_as_uint(x); }
__device__ __forceinline__ uint32_t sign_exp(double x) { return (uint32_t)__double2hiint(x); }
__device__ __forceinline__ float minor_fma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double minor_fma(double a, double b, double c) { return fma(a, b, c); }
template <typename R>
__device__ __forceinline__ int minor_count(const R* __restrict__ d, const R* __restrict__ e2, int n, R x) {
  constexpr bool k64 = sizeof(R) == 8;
  constexpr uint32_t kExp = k64 ? 0x7FF00000u : 0x7F800000u;
  constexpr uint32_t kBig = k64 ? (1023u + 300u) << 20 : (127u + 30u) << 23;
  constexpr uint32_t kSmall = k64 ? (1023u - 300u) << 20 : (127u - 30u) << 23;
  const R down = k64 ? (R)0x1p-600 : (R)0x1p-60f, up = k64 ? (R)0x1p600 : (R)0x1p60f;
  R pm = 1, p = d[0] - x;
  int c = (int)(sign_exp(p) >> 31);
  int i = 1;
  auto row = [&]() {
    const R pn = minor_fma(d[i] - x, p, -(e2[i - 1] * pm));
    c += (int)((sign_exp(pn) ^ sign_exp(p)) >> 31);
    pm = p;
    p = pn;
    ++i;
  };
  while (i + 4 <= n) {
    row();
    row();
    row();
    row();
    const uint32_t ex = max(sign_exp(p) & kExp, sign_exp(pm) & kExp);
    if (ex > kBig) {
      p *= down;
      pm *= down;
    } else if (ex < kSmall) {
      p *= up;
      pm *= up;
    }
  }
  while (i < n) row();
  return c;
}
// e^2 as the counts take it: a decoupled row couples by less than any rounding
// instead (of |T| ~ 1), so that no minor stays zero
__device__ __forceinline__ double minor_e2(double e) { return fmax(e * e, 1e-290); }
__device__ __forceinline__ float minor_e232(double e) { return fmaxf((float)e * (float)e, 1e-30f); }

// T in shared memory for warp_eigenvalue: diagonal, e[i] coupling rows i - 1 and
// i, its squares, and both in FP32 (m entries each).
struct TdT {
  double *d, *e, *e2;
  float *d32, *e232;
  static __host__ __device__ size_t bytes(int m) { return (size_t)m * (3 * sizeof(double) + 2 * sizeof(float)); }
  __device__ TdT(void* at, int m) {
    d = static_cast<double*>(at);
    e = d + m;
    e2 = e + m;
    d32 = reinterpret_cast<float*>(e2 + m);
    e232 = d32 + m;
  }
  __device__ __forceinline__ void set(int i, double di, double ei) {
    d[i] = di;
    e[i] = i > 0 ? ei : 0.0;
    e2[i] = i > 0 ? minor_e2(ei) : 0.0;
    d32[i] = (float)di;
    e232[i] = i > 0 ? minor_e232(ei) : 0.f;
  }
};

// Eigenvalue k (0 is the lowest) of rows r0 .. m - 1 of T by one warp: multisection
// on the counts at 32 points of the bracket, 33 times narrower a round; all lanes
// return it.  FP32 counts to about 1e-7 of the Gershgorin bound, then FP64 ones
// from a bracket widened by four times that (checked, the whole range if the
// eigenvalue is not in it) until it is two ulps wide.  The lowest of 100
// rows took 616 us by quotients and takes 129 us; 146 values of 300 rows 12.0 ms
// and 2.6 ms.
__device__ inline double warp_eigenvalue(const TdT& T, int r0, int m, int k) {
  const int lane = threadIdx.x & 31;
  const double *d = T.d + r0, *e2 = T.e2 + r0 + 1;
  const float *d32 = T.d32 + r0, *e232 = T.e232 + r0 + 1;
  m -= r0;
  double lo = 1e300, hi = -1e300;
  for (int i = lane; i < m; i += 32) {
    const double r = (i > 0 ? fabs(T.e[r0 + i]) : 0.0) + (i + 1 < m ? fabs(T.e[r0 + i + 1]) : 0.0);
    lo = fmin(lo, d[i] - r);
    hi = fmax(hi, d[i] + r);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  const double scale = fmax(fabs(lo), fabs(hi));
  lo -= 2.2e-16 * scale + 1e-300;
  hi += 2.2e-16 * scale + 1e-300;
  const double gl = lo, gu = hi;
  // one round: the counts at x, and the part of the bracket that holds k
  auto narrow = [&](auto& a, auto& b, auto x, int count, bool inside) {
    const unsigned above = __ballot_sync(0xffffffffu, inside && count > k);
    const unsigned in = __ballot_sync(0xffffffffu, inside);
    if (in == 0u) return false;  // the bracket has no interior point left
    const int first = above ? __ffs((int)above) - 1 : 32;  // counts grow with x
    const auto xa = __shfl_sync(0xffffffffu, x, first > 0 ? first - 1 : 0);
    const auto xb = __shfl_sync(0xffffffffu, x, first < 32 ? first : 31);
    if (first > 0 && ((in >> (first - 1)) & 1u)) a = xa;
    if (first < 32) b = xb;
    return true;
  };
  float fa = (float)lo, fb = (float)hi;
  for (int it = 0; it < 8; ++it) {
    if (!(fb - fa > 4.f * 1.1920929e-7f * fmaxf(fabsf(fa), fabsf(fb)))) break;
    const float x = fa + (fb - fa) * ((float)(lane + 1) / 33.f);
    if (!narrow(fa, fb, x, minor_count(d32, e232, m, x), x > fa && x < fb)) break;
  }
  const double width = (double)fb - (double)fa + 4e-7 * scale;
  const double wa = fmax(gl, (double)fa - width), wb = fmin(gu, (double)fb + width);
  const unsigned below = __ballot_sync(0xffffffffu, minor_count(d, e2, m, lane == 0 ? wa : wb) <= k);
  if ((below & 1u) && !(below & 2u)) {
    lo = wa;
    hi = wb;
  }
  for (int round = 0; round < 64; ++round) {
    if (hi - lo <= 2.0 * 2.2204460492503131e-16 * fmax(fabs(lo), fabs(hi))) break;
    const double x = lo + (hi - lo) * ((double)(lane + 1) / 33.0);
    if (!narrow(lo, hi, x, minor_count(d, e2, m, x), x > lo && x < hi)) break;
  }
  return 0.5 * (lo + hi);
}
#endif

// Eigenvector of eigenvalue lam, normalised, written to x[0..m-1].  Work
// arrays: 5*m doubles in `wk`.  The sign is fixed so that the largest
// component is positive.  For a level of a cluster of (nearly) equal
// eigenvalues, `prev` holds the n_prev unit vectors already computed for the
// cluster (m doubles each, consecutive): each sweep's iterate is
// orthogonalised against them (modified Gram-Schmidt), and `seed` > 0 varies
// the start vector, so the cluster's vectors come out orthonormal (the
// approach of LAPACK's inverse iteration for clustered eigenvalues).
TD_HD void tridiag_eigenvector_ex(const double* d, const double* e, int m, double lam, double* x, double* wk,
                                  const double* prev, int n_prev, int seed);
TD_HD void tridiag_eigenvector(const double* d, const double* e, int m, double lam, double* x, double* wk) {
  tridiag_eigenvector_ex(d, e, m, lam, x, wk, nullptr, 0, 0);
}
TD_HD void tridiag_eigenvector_ex(const double* d, const double* e, int m, double lam, double* x, double* wk,
                                  const double* prev, int n_prev, int seed) {
  double* u0 = wk;          // main diagonal of U
  double* u1 = wk + m;      // first superdiagonal of U
  double* u2 = wk + 2 * m;  // second superdiagonal of U (fill-in from pivoting)
  double* l = wk + 3 * m;   // multipliers
  double* piv = wk + 4 * m; // 1 when rows k, k+1 were swapped
  double scale = 0.0;
  for (int i = 0; i < m; ++i) scale = fmax(scale, fabs(d[i]) + (i > 0 ? fabs(e[i]) : 0.0));
  const double tiny = fmax(scale, 1e-300) * 2.2204460492503131e-16;
  // LU with partial pivoting of (T - lam I)
  for (int i = 0; i < m; ++i) {
    u0[i] = d[i] - lam;
    u1[i] = (i + 1 < m) ? e[i + 1] : 0.0;
    u2[i] = 0.0;
  }
  for (int k = 0; k + 1 < m; ++k) {
    const double sub = e[k + 1];
    if (fabs(u0[k]) >= fabs(sub)) {
      piv[k] = 0.0;
      if (u0[k] == 0.0) u0[k] = tiny;
      l[k] = sub / u0[k];
      u0[k + 1] -= l[k] * u1[k];
      u1[k + 1] -= l[k] * u2[k];
    } else {
      piv[k] = 1.0;
      l[k] = u0[k] / sub;
      // swap row k (u0[k], u1[k], u2[k]) with row k+1 (sub, u0[k+1], u1[k+1])
      const double r0 = sub, r1 = u0[k + 1], r2 = u1[k + 1];
      const double o1 = u1[k], o2 = u2[k];
      u0[k] = r0;
      u1[k] = r1;
      u2[k] = r2;
      u0[k + 1] = o1 - l[k] * r1;
      u1[k + 1] = o2 - l[k] * r2;
    }
  }
  if (u0[m - 1] == 0.0) u0[m - 1] = tiny;
  for (int i = 0; i < m; ++i) x[i] = seed > 0 ? 1.0 + 0.25 * (double)((i * (2 * seed + 1) + seed) % 7) / 7.0 : 1.0;
  for (int sweep = 0; sweep < 3; ++sweep) {
    // forward: apply the row operations to the right-hand side
    for (int k = 0; k + 1 < m; ++k) {
      if (piv[k] != 0.0) {
        const double t = x[k];
        x[k] = x[k + 1];
        x[k + 1] = t;
      }
      x[k + 1] -= l[k] * x[k];
    }
    // back substitution with U
    for (int i = m - 1; i >= 0; --i) {
      double s = x[i];
      if (i + 1 < m) s -= u1[i] * x[i + 1];
      if (i + 2 < m) s -= u2[i] * x[i + 2];
      double p = u0[i];
      if (fabs(p) < tiny) p = p < 0 ? -tiny : tiny;
      x[i] = s / p;
    }
    for (int q = 0; q < n_prev; ++q) {
      const double* pq = prev + (int64_t)q * m;
      double dot = 0.0;
      for (int i = 0; i < m; ++i) dot += pq[i] * x[i];
      for (int i = 0; i < m; ++i) x[i] -= dot * pq[i];
    }
    double nrm = 0.0, big = 0.0;
    int arg = 0;
    for (int i = 0; i < m; ++i) {
      nrm += x[i] * x[i];
      if (fabs(x[i]) > big) { big = fabs(x[i]); arg = i; }
    }
    nrm = sqrt(nrm);
    const double sgn = x[arg] < 0 ? -1.0 : 1.0;
    for (int i = 0; i < m; ++i) x[i] = sgn * x[i] / nrm;
  }
}

}  // namespace edg
