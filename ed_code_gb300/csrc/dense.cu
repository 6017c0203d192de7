// The reference's dense small-sector path on the device: exact_evecs
// (lanczos.cpp:81-131) on the matrix makeH builds (H_v.cpp:21-190), used by
// sector_lanczos for n_p <= 10000 (Lanczos_sector.cpp:105-120).
//
//   1. H assembled in one kernel from the stored rows: per nonzero
//      norm_i * value * norm_inv_j (the same matrix elements the stored-row
//      H*v uses), Ezz_i on the diagonal; without stored rows, column j is
//      H e_j from the matrix-free kernel.  Only the upper triangle is used,
//      as zheev('V','U') does (Matrix_Functions.cpp:39-40).
//   2. Householder reduction to a real symmetric tridiagonal T = Q^H H Q
//      (Golub and Van Loan, "Matrix Computations", sec. 8.3.1, for complex
//      Hermitian matrices: H_k = I - tau_k v_k v_k^H with a complex tau_k
//      that makes the sub-diagonal real).  Step k: the reflector of column k,
//      p = tau A22 v, w = p - (tau/2)(p^H v) v, and the rank-2 update
//      A22 -= v w^H + w v^H, in two kernels on the lower triangle: one brings
//      column k up to date and takes its reflector, the other applies the
//      previous step's update and multiplies by the new v in one pass.
//   3. All n eigenvalues of T, eight lanes each: multisection on Sturm counts
//      (the signs of the leading minors) in FP32 to about 1e-7 of |T|, then in
//      FP64 from there; GB300 runs FP64 at 1/64 of its FP32 rate.
//   4. The wanted eigenvectors: inverse iteration on T (tridiag.cuh;
//      orthogonalised within clusters of equal eigenvalues), then x = Q y by
//      applying the reflectors from the last to the first.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <string>
#include <vector>

#include "../../include/edgpu.h"
#include "blas1.cuh"
#include "csr_row.cuh"
#include "edg_sector.cuh"
#include "tridiag.cuh"

namespace edg {

int fail(int code, const std::string& msg);
int cuda_fail(cudaError_t e, const char* what);

namespace {

constexpr int kDenseThreads = 256;

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cconjmul(double2 a, double2 b) {  // conj(a) * b
  return make_double2(a.x * b.x + a.y * b.y, a.x * b.y - a.y * b.x);
}

// H[j*n + i] += H_ij from the stored rows: a thread per row, a warp per slice
// (csr_row.cuh)
__global__ void k_dense_rows(const uint64_t* __restrict__ row_ptr, const uint32_t* __restrict__ col,
                             const uint16_t* __restrict__ vid, int cb, const double2* __restrict__ vtab,
                             const double* __restrict__ ezz, const uint8_t* __restrict__ lid,
                             const double* __restrict__ nrm, const double* __restrict__ nrm_inv, int64_t n,
                             double2* __restrict__ H) {
  const uint32_t lt = (1u << (threadIdx.x & 31)) - 1u;
  for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < n; base += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = base + threadIdx.x;
    const Slice s = slice_at(row_ptr, i, n);
    const double ni = i < n ? nrm[lid[i]] : 0.0;
    uint64_t at = s.base;
    for (int k = 0; k < s.mx; ++k) {
      const uint32_t m = __ballot_sync(0xffffffffu, s.len > k);
      if (s.len > k) {
        const uint64_t t = at + __popc(m & lt);
        const uint32_t e = col[t];
        const uint32_t j = vid ? e : e & ((1u << cb) - 1u);
        const double2 c = vtab[vid ? (uint32_t)vid[t] : e >> cb];
        const double sc = nrm_inv ? ni * nrm_inv[lid[j]] : ni;  // nullptr: in the values
        double2* h = H + (int64_t)j * n + i;
        h->x += c.x * sc;
        h->y += c.y * sc;
      }
      at += __popc(m);
    }
    if (i < n) H[i * n + i].x += ezz[i];
  }
}

__global__ void k_unit_col(double2* e, int64_t n, int64_t j) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    e[i] = make_double2(i == j ? 1.0 : 0.0, 0.0);
}

// A Hermitian from its upper triangle: A_rc = conj(A_cr) for r > c, real diagonal
__global__ void k_herm_upper(double2* __restrict__ A, int64_t n) {
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, c = blockIdx.y;
  if (r >= n) return;
  if (r > c) {
    const double2 u = A[r * n + c];  // (c, r), c < r: upper
    A[c * n + r] = make_double2(u.x, -u.y);
  } else if (r == c) {
    A[c * n + c].y = 0.0;
  }
}

__device__ double block_sum(double x, double* sh) {
  sh[threadIdx.x] = x;
  __syncthreads();
  for (int h = blockDim.x / 2; h > 0; h >>= 1) {
    if ((int)threadIdx.x < h) sh[threadIdx.x] += sh[threadIdx.x + h];
    __syncthreads();
  }
  const double r = sh[0];
  __syncthreads();
  return r;
}

// The reduction's state beside A (n x n, column-major, lower triangle): v_k is
// stored in column k below the diagonal, as the back-transformation wants it.
// What a step leaves for the next is kept twice, by the parity of k.
constexpr int kTile = 32, kTileThreads = 128;
struct Hh {
  double2* A;
  int64_t n;
  int nb;         // blocks of kTile rows
  double *d, *e;
  double2* tau;
  double2* x;     // [2][n]: column k, up to date, before its scaling: v = x inv, v_{k+1} = 1
  double2* inv;   // [2]
  double2* y;     // [2][n]: A22 v
  double2* D;     // per block of rows: sum conj(y) v
  double2* K;     // [2]: -|tau|^2/2 v^H A v: w = tau y + K v
  double2* part;  // nb x n: the tiles' shares of y
  double* norms;  // the reflector's CTAs' shares of |x|^2
  int* cnt;       // nb + 1 tickets, zero between launches
};

// The sum of x over a CTA of kTileThreads, in every thread: shuffles and one
// round through shared memory.
__device__ __forceinline__ double tile_sum(double x) {
  __shared__ double sh[kTileThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = x;
  __syncthreads();
  double s = sh[0];
#pragma unroll
  for (int w = 1; w < kTileThreads / 32; ++w) s += sh[w];
  return s;
}

// true in the CTA that takes the last of `total` tickets (no CTA waits)
__device__ __forceinline__ bool hh_last(int* cnt, int total) {
  __shared__ int last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(cnt, 1) == total - 1;
    if (last) *cnt = 0;
  }
  __syncthreads();
  const bool r = last != 0;
  if (r) __threadfence();
  __syncthreads();
  return r;
}

__device__ __forceinline__ double2 ldcg2(const double2* p) { return __ldcg(p); }

// a - v conj(w_j) - w conj(v_j)
__device__ __forceinline__ double2 rank2(double2 a, double2 v, double2 w, double2 vj, double2 wj) {
  a.x = fma(-v.x, wj.x, fma(-v.y, wj.y, fma(-w.x, vj.x, fma(-w.y, vj.y, a.x))));
  a.y = fma(-v.y, wj.x, fma(v.x, wj.y, fma(-w.y, vj.x, fma(w.x, vj.y, a.y))));
  return a;
}

// Step k, first kernel: column k with step k-1's update, x = A[k+1.., k] -> its
// reflector v = (1, x_1/(alpha - beta), ...): d[k], e[k] = beta, tau[k].  A CTA
// per 128 rows; the last one finishes the norm and the scalars.
__global__ void __launch_bounds__(kTileThreads) k_hh_column(Hh H, int64_t k) {
  const int64_t n = H.n;
  const int p = (int)(k & 1), lane = threadIdx.x & 31;
  double2 Kc = make_double2(0.0, 0.0), t = make_double2(0.0, 0.0), wk = Kc;
  const double2* vo = H.A + (k - 1) * n;  // v_{k-1}: 1 at row k
  const double2* yo = H.y + (1 - p) * n;
  if (k > 0) {  // w_{k-1} = t y + K v, K from the blocks' shares in block order
    __shared__ double2 sK;
    if (threadIdx.x < 32) {
      double a = 0, b = 0;
      for (int r = (int)(k / kTile) + lane; r < H.nb; r += 32) {
        const double2 q = H.D[r];
        a += q.x;
        b += q.y;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, o);
        b += __shfl_down_sync(0xffffffffu, b, o);
      }
      if (lane == 0) {
        const double2 tt = H.tau[k - 1];
        const double h = -0.5 * (tt.x * tt.x + tt.y * tt.y);
        sK = make_double2(h * a, h * b);
        if (blockIdx.x == 0) H.K[1 - p] = sK;
      }
    }
    __syncthreads();
    Kc = sK;
    t = H.tau[k - 1];
    wk = cmul(t, yo[k]);
    wk.x += Kc.x;
    wk.y += Kc.y;
  }
  const int64_t i = k + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  double s = 0.0;
  if (i < n) {
    double2 a = H.A[k * n + i];
    if (k > 0) {
      const double2 v = i == k ? make_double2(1.0, 0.0) : vo[i];
      double2 w = cmul(t, yo[i]);
      const double2 kv = cmul(Kc, v);
      w.x += kv.x;
      w.y += kv.y;
      a = rank2(a, v, w, make_double2(1.0, 0.0), wk);
    }
    if (i == k) H.d[k] = a.x;
    else H.x[p * n + i] = a;
    if (i > k + 1) s = a.x * a.x + a.y * a.y;
  }
  if (k + 1 >= n) return;
  s = tile_sum(s);
  if (threadIdx.x == 0) H.norms[blockIdx.x] = s;
  if (!hh_last(H.cnt + H.nb, gridDim.x)) return;
  s = 0.0;
  for (int q = threadIdx.x; q < (int)gridDim.x; q += blockDim.x) s += __ldcg(H.norms + q);
  s = tile_sum(s);
  if (threadIdx.x < 4) {  // the four quotients side by side: a division is a long chain
    const double2 alpha = ldcg2(H.x + p * n + k + 1);
    double beta = alpha.x, quot = threadIdx.x == 2 ? 1.0 : 0.0;
    if (s != 0.0 || alpha.y != 0.0) {
      beta = -copysign(sqrt(alpha.x * alpha.x + alpha.y * alpha.y + s), alpha.x);
      const double zr = alpha.x - beta, zi = alpha.y, z2 = zr * zr + zi * zi;
      const double num = threadIdx.x == 0 ? beta - alpha.x : threadIdx.x == 1 ? -alpha.y : threadIdx.x == 2 ? zr : -zi;
      quot = num / (threadIdx.x < 2 ? beta : z2);
    }
    double* to = reinterpret_cast<double*>(threadIdx.x < 2 ? H.tau + k : H.inv + p);
    to[threadIdx.x & 1] = quot;
    if (threadIdx.x == 0) H.e[k] = beta;
  }
}

// Step k, second kernel: A22 (rows and columns > k) with step k-1's update, and
// y = A22 v_k from its lower triangle: a CTA per 32 x 32 tile on or below the
// diagonal, a lane per row, eight columns a warp.  An element off the diagonal
// serves y_i and y_j; the eight columns' shares of y_j over the lanes are closed
// by an exchange that halves them (16 additions instead of 80).  The tiles'
// shares are summed in block order by the last tile of each block of rows, with
// sum conj(y) v.  Bound by FP64 issue (16 clocks a warp instruction): 18
// instructions an element of half the matrix, where separate update (12) and
// product (4) kernels took 16 of all of it, and passed over it three times.
// 2,700 states: the first column took 331 us in four kernels and takes 152 us in
// two (FP64 pipe 79 % busy while an SM has tiles), the whole spectrum 369 ms and
// 185 ms.
__global__ void __launch_bounds__(kTileThreads) k_hh_tile(Hh H, int64_t k, int b0) {
  __shared__ double2 vn[2][kTile], vo[2][kTile], wo[2][kTile];  // rows' and columns' blocks
  __shared__ double2 ysum[kTileThreads / 32][kTile];
  const int64_t n = H.n;
  const int p = (int)(k & 1), lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  // tile (bi, bj), b0 <= bj <= bi: index = r (r + 1) / 2 + c
  const int idx = blockIdx.x;
  int r = (int)((sqrtf(8.f * (float)idx + 1.f) - 1.f) * 0.5f);
  while ((r + 1) * (r + 2) / 2 <= idx) ++r;
  while (r * (r + 1) / 2 > idx) --r;
  const int bi = b0 + r, bj = b0 + idx - r * (r + 1) / 2;
  const int64_t i = (int64_t)bi * kTile + lane, j0 = (int64_t)bj * kTile + 8 * wid;
  double2 a[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {  // in flight during the vectors' preparation
    const int64_t j = j0 + q;
    a[q] = make_double2(0.0, 0.0);
    if (j > k && i >= j && i < n) a[q] = H.A[j * n + i];
  }
  if (threadIdx.x < 2 * kTile) {
    const int side = threadIdx.x >> 5;
    const int64_t m = (int64_t)(side ? bj : bi) * kTile + lane;
    double2 f = make_double2(0.0, 0.0), b = f, c = f;
    if (m > k && m < n) {
      f = m == k + 1 ? make_double2(1.0, 0.0) : cmul(H.x[p * n + m], H.inv[p]);
      if (bi == bj && side == 0) H.A[k * n + m] = f;
      if (k > 0) {
        b = H.A[(k - 1) * n + m];
        c = cmul(H.tau[k - 1], H.y[(1 - p) * n + m]);
        const double2 kv = cmul(H.K[1 - p], b);
        c.x += kv.x;
        c.y += kv.y;
      }
    }
    vn[side][lane] = f;
    vo[side][lane] = b;
    wo[side][lane] = c;
  }
  __syncthreads();
  const double2 vi = vn[0][lane], oi = vo[0][lane], wi = wo[0][lane];
  double yr = 0.0, yi = 0.0, c[16];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int64_t j = j0 + q;
    const int jl = 8 * wid + q;
    const bool in = j > k && i >= j && i < n;
    if (k > 0) {
      a[q] = rank2(a[q], oi, wi, vo[1][jl], wo[1][jl]);
      if (i == j) a[q].y = 0.0;
      if (in) H.A[j * n + i] = a[q];
    }
    if (!in) a[q] = make_double2(0.0, 0.0);
    const double2 vj = vn[1][jl];
    yr = fma(a[q].x, vj.x, fma(-a[q].y, vj.y, yr));
    yi = fma(a[q].x, vj.y, fma(a[q].y, vj.x, yi));
    const double2 z = i == j ? make_double2(0.0, 0.0) : a[q];
    c[2 * q] = fma(z.x, vi.x, z.y * vi.y);
    c[2 * q + 1] = fma(z.x, vi.y, -(z.y * vi.x));
  }
#pragma unroll
  for (int o = 16, w = 8; o >= 2; o >>= 1, w >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (j < w) c[j] = (up ? c[w + j] : c[j]) + __shfl_xor_sync(0xffffffffu, up ? c[j] : c[w + j], o);
  }
  c[0] += __shfl_xor_sync(0xffffffffu, c[0], 1);  // value lane >> 1 of the 16
  ysum[wid][lane] = make_double2(yr, yi);
  __shared__ double cs[kTile][2];
  if ((lane & 1) == 0) cs[8 * wid + (lane >> 2)][(lane >> 1) & 1] = c[0];
  __syncthreads();
  if (wid == 0) {
    double2 z = ysum[0][lane];
#pragma unroll
    for (int q = 1; q < kTileThreads / 32; ++q) {
      z.x += ysum[q][lane].x;
      z.y += ysum[q][lane].y;
    }
    if (bi == bj) {
      z.x += cs[lane][0];
      z.y += cs[lane][1];
    }
    if (i < n) H.part[(int64_t)bj * n + i] = z;
  } else if (wid == 1 && bi != bj) {
    H.part[(int64_t)bi * n + (int64_t)bj * kTile + lane] = make_double2(cs[lane][0], cs[lane][1]);
  }
  // the last tile of a block of rows closes its y
  for (int side = 0; side < (bi == bj ? 1 : 2); ++side) {
    const int blk = side ? bj : bi;
    if (!hh_last(H.cnt + blk, H.nb - b0)) continue;
    const int64_t row = (int64_t)blk * kTile + lane;
    double2 z = make_double2(0.0, 0.0);
    if (row < n)
      for (int q = b0 + wid; q < H.nb; q += kTileThreads / 32) {
        const double2 f = ldcg2(H.part + (int64_t)q * n + row);
        z.x += f.x;
        z.y += f.y;
      }
    __syncthreads();
    ysum[wid][lane] = z;
    __syncthreads();
    if (wid == 0) {
#pragma unroll
      for (int q = 1; q < kTileThreads / 32; ++q) {
        z.x += ysum[q][lane].x;
        z.y += ysum[q][lane].y;
      }
      if (row < n) H.y[p * n + row] = z;
      double2 g = cconjmul(z, vn[side][lane]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        g.x += __shfl_down_sync(0xffffffffu, g.x, o);
        g.y += __shfl_down_sync(0xffffffffu, g.y, o);
      }
      if (lane == 0) H.D[blk] = g;
    }
  }
}

// ---- eigenvalues of T: d[0..n-1], off-diagonal e[0..n-2] (row i to i+1) ----

__global__ void k_tri_prep(const double* __restrict__ d, const double* __restrict__ e, int n, float* __restrict__ d32,
                           float* __restrict__ e232, double* __restrict__ e2) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    d32[i] = (float)d[i];
    if (i + 1 < n) {
      e2[i] = minor_e2(e[i]);
      e232[i] = minor_e232(e[i]);
    }
  }
}

// One round of multisection for eigenvalue k in (lo, hi] by a group of eight
// lanes: the counts at eight interior points, and the ninth of the bracket that
// holds it.  All lanes of the warp take part.
template <typename R, class Count>
__device__ __forceinline__ void narrow(R& lo, R& hi, int k, bool run, Count count) {
  const int sub = threadIdx.x & 7, at = threadIdx.x & 24;
  const R x = lo + (hi - lo) * ((R)(sub + 1) / (R)9);
  const unsigned above = (__ballot_sync(0xffffffffu, count(x) > k) >> at) & 0xFFu;
  const int first = above ? __ffs((int)above) - 1 : 8;  // counts grow with x
  const R a = __shfl_sync(0xffffffffu, x, at + (first > 0 ? first - 1 : 0));
  const R b = __shfl_sync(0xffffffffu, x, at + (first < 8 ? first : 7));
  if (!run) return;
  if (first > 0) lo = a;
  if (first < 8) hi = b;
}

// Eigenvalue k of T by a group of eight lanes; bounds [gl, gu] enclose the
// spectrum.  FP32 counts to about 1e-7 of |T|, then FP64 counts from a bracket
// widened by four times that (checked; the whole range if the eigenvalue is not
// in it) to half an ulp of |T|: ten rounds of three FP64 instructions a row of
// T, four warps an SM.  Newton's method on the determinant took six passes of
// twice the instructions and left multiple roots to 31 bisections by one lane,
// which made it 43 ms at 2,700 states; this takes 5.8 ms.
__global__ void __launch_bounds__(32) k_tri_all(const double* __restrict__ d, const double* __restrict__ e2,
                                                const float* __restrict__ d32, const float* __restrict__ e232, int n,
                                                double gl, double gu, double tnorm, double* __restrict__ out) {
  const int k = min(n - 1, (int)((blockIdx.x * 32 + threadIdx.x) >> 3));
  auto c32 = [&](float x) { return minor_count(d32, e232, n, x); };
  auto c64 = [&](double x) { return minor_count(d, e2, n, x); };
  float lo = (float)gl, hi = (float)gu;
  for (int it = 0; it < 16; ++it) {
    const bool run = hi - lo > 4.f * 1.1920929e-7f * fmaxf(fabsf(lo), fabsf(hi));
    if (!__any_sync(0xffffffffu, run)) break;
    narrow(lo, hi, k, run, c32);
  }
  const double width = (double)hi - (double)lo + 4e-7 * tnorm;
  double a = (double)lo - width, b = (double)hi + width;
  // lane 0 of a group looks at a, the others at b
  const int sub = threadIdx.x & 7;
  const bool below = c64(sub == 0 ? a : b) <= k;
  const unsigned m = __ballot_sync(0xffffffffu, below) >> (threadIdx.x & 24);
  if (!(m & 1u)) a = gl;
  if (m & 2u) b = gu;
  const double tol = 1.110223024625157e-16 * tnorm;
  for (int it = 0; it < 24; ++it) {
    const double x = a + (b - a) * (1.0 / 9.0);
    const bool run = b - a > tol && x > a && x < b;
    if (!__any_sync(0xffffffffu, run)) break;
    narrow(a, b, k, run, c64);
  }
  if (sub == 0) out[k] = 0.5 * (a + b);
}

// eigenvectors of T for lam[0..nv-1] (ascending), one thread in sequence:
// levels within 1e-9 |T| of each other are a cluster, orthogonalised
__global__ void k_tri_vectors(const double* __restrict__ d, const double* __restrict__ eoff, int n,
                              const double* __restrict__ lam, int nv, double tnorm, double* __restrict__ y,
                              double* __restrict__ wk) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  int c0 = 0;  // first level of the current cluster
  for (int q = 0; q < nv; ++q) {
    if (q > 0 && fabs(lam[q] - lam[q - 1]) > 1e-9 * fmax(tnorm, 1.0)) c0 = q;
    tridiag_eigenvector_ex(d, eoff, n, lam[q], y + (int64_t)q * n, wk, y + (int64_t)c0 * n, q - c0, q - c0);
  }
}

// x = Q y for nv vectors (one CTA each): Q = H_0 ... H_{n-2}, applied from the
// last reflector to the first; y real (n doubles), x complex
__global__ void __launch_bounds__(kDenseThreads) k_backtransform(const double2* __restrict__ A, int64_t n,
                                                                 const double2* __restrict__ tau,
                                                                 const double* __restrict__ y,
                                                                 double2* __restrict__ X) {
  __shared__ double sh[kDenseThreads];
  double2* x = X + (int64_t)blockIdx.x * n;
  const double* yq = y + (int64_t)blockIdx.x * n;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) x[i] = make_double2(yq[i], 0.0);
  __syncthreads();
  for (int64_t k = n - 2; k >= 0; --k) {
    const double2 t = tau[k];
    if (t.x == 0.0 && t.y == 0.0) continue;
    const int64_t m = n - k - 1;
    const double2* v = A + k * n + (k + 1);
    double2* z = x + (k + 1);
    double sr = 0.0, si = 0.0;
    for (int64_t i = threadIdx.x; i < m; i += blockDim.x) {
      const double2 q = cconjmul(v[i], z[i]);
      sr += q.x;
      si += q.y;
    }
    sr = block_sum(sr, sh);
    si = block_sum(si, sh);
    const double2 c = cmul(t, make_double2(sr, si));
    for (int64_t i = threadIdx.x; i < m; i += blockDim.x) {
      const double2 u = cmul(c, v[i]);
      z[i].x -= u.x;
      z[i].y -= u.y;
    }
    __syncthreads();
  }
}

int grid1(int64_t n) { return (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 152 * 16)); }

}  // namespace

int solve_dense_device(Sector& S, double* eigs, int64_t cap, int64_t* n_out, double* evecs, int64_t evecs_cap,
                       edg_solver_stats* stats) {
  const int64_t n = S.P.n_p;
  if (cap < n) return fail(EDG_ERR_INVALID, "dense path returns all n_p eigenvalues: eigs_capacity too small");
  if (n > 46340) return fail(EDG_ERR_UNSUPPORTED, "dense path: sector too large");
  const int64_t nv = (evecs && evecs_cap > 0) ? std::min<int64_t>(evecs_cap, n) : 0;
  cudaStream_t st = S.stream;
  double2 *H = nullptr, *tau = nullptr, *pw = nullptr, *X = nullptr, *part = nullptr;
  double *d = nullptr, *e = nullptr, *e2 = nullptr, *lam = nullptr, *y = nullptr, *wk = nullptr;
  float* f32 = nullptr;
  int* hcnt = nullptr;
  const int nb = (int)((n + kTile - 1) / kTile);
  // pw: x, y (two each), D, inv, K, norms
  const size_t pw_n = (size_t)(4 * n + nb + 4 + (n + kTileThreads) / kTileThreads);
  auto cleanup = [&]() {
    void* p[] = {H, tau, pw, X, part, hcnt, d, e, e2, lam, y, wk, f32};
    for (void* q : p)
      if (q) cudaFree(q);
  };
  cudaError_t ce = cudaMalloc(&H, sizeof(double2) * n * n);
  if (ce == cudaSuccess) ce = cudaMalloc(&tau, sizeof(double2) * n);
  if (ce == cudaSuccess) ce = cudaMalloc(&pw, sizeof(double2) * pw_n);
  if (ce == cudaSuccess) ce = cudaMalloc(&part, sizeof(double2) * (size_t)nb * n);
  if (ce == cudaSuccess) ce = cudaMalloc(&hcnt, sizeof(int) * (nb + 1));
  if (ce == cudaSuccess) ce = cudaMalloc(&d, sizeof(double) * n);
  if (ce == cudaSuccess) ce = cudaMalloc(&e, sizeof(double) * n);
  if (ce == cudaSuccess) ce = cudaMalloc(&e2, sizeof(double) * n);
  if (ce == cudaSuccess) ce = cudaMalloc(&lam, sizeof(double) * n);
  if (ce == cudaSuccess) ce = cudaMalloc(&f32, sizeof(float) * 2 * n);
  if (ce == cudaSuccess && nv > 0) ce = cudaMalloc(&X, sizeof(double2) * n * nv);
  if (ce == cudaSuccess && nv > 0) ce = cudaMalloc(&y, sizeof(double) * n * nv);
  if (ce == cudaSuccess && nv > 0) ce = cudaMalloc(&wk, sizeof(double) * 5 * n);
  if (ce != cudaSuccess) {
    cleanup();
    return fail(EDG_ERR_NOMEM, "dense path: out of device memory");
  }
  using clk = std::chrono::steady_clock;
  const auto t0 = clk::now();
  // 1. H
  cudaMemsetAsync(H, 0, sizeof(double2) * n * n, st);
  int64_t hv_calls = 0;
  if (S.col) {
    const double* nrm = reinterpret_cast<const double*>(reinterpret_cast<const char*>(S.dP) +
                                                        offsetof(SectorParams, nrm));
    const double* nrm_inv = reinterpret_cast<const double*>(reinterpret_cast<const char*>(S.dP) +
                                                            offsetof(SectorParams, nrm_inv));
    k_dense_rows<<<grid1(n), 256, 0, st>>>(S.row_ptr, S.col, S.vid, S.pack_cb, S.rtab64, S.ezz, S.lid, nrm,
                                           S.folded ? nullptr : nrm_inv,
                                           n, H);
  } else {
    for (int64_t j = 0; j < n && ce == cudaSuccess; ++j) {
      k_unit_col<<<grid1(n), 256, 0, st>>>(pw, n, j);
      ce = launch_hv(S, pw, H + j * n, true, st);
      ++hv_calls;
    }
  }
  if (ce == cudaSuccess) ce = cudaGetLastError();
  if (ce != cudaSuccess) {
    cleanup();
    return cuda_fail(ce, "dense path: assembling H");
  }
  const auto t1 = clk::now();
  // 2. Householder tridiagonalisation
  k_herm_upper<<<dim3((unsigned)((n + 255) / 256), (unsigned)n), 256, 0, st>>>(H, n);
  cudaMemsetAsync(hcnt, 0, sizeof(int) * (nb + 1), st);
  Hh h{H, n, nb, d, e, tau, pw, nullptr, pw + 2 * n, nullptr, nullptr, part, nullptr, hcnt};
  h.D = pw + 4 * n;
  h.inv = h.D + nb;
  h.K = h.inv + 2;
  h.norms = reinterpret_cast<double*>(h.K + 2);
  for (int64_t k = 0; k < n; ++k) {
    k_hh_column<<<(unsigned)((n - k + kTileThreads - 1) / kTileThreads), kTileThreads, 0, st>>>(h, k);
    if (k + 1 == n) break;
    const int b0 = (int)((k + 1) / kTile);
    const int64_t m = nb - b0;
    k_hh_tile<<<(unsigned)(m * (m + 1) / 2), kTileThreads, 0, st>>>(h, k, b0);
  }
  // 3. eigenvalues: Gershgorin bounds of T on the host (2n doubles)
  std::vector<double> dh(n), eh(n, 0.0);
  cudaMemcpyAsync(dh.data(), d, sizeof(double) * n, cudaMemcpyDeviceToHost, st);
  if (n > 1) cudaMemcpyAsync(eh.data(), e, sizeof(double) * (n - 1), cudaMemcpyDeviceToHost, st);
  if ((ce = cudaStreamSynchronize(st)) != cudaSuccess) {
    cleanup();
    return cuda_fail(ce, "dense path: tridiagonalisation");
  }
  double gl = dh[0], gu = dh[0], tnorm = 0.0;
  for (int64_t i = 0; i < n; ++i) {
    const double r = (i > 0 ? std::fabs(eh[i - 1]) : 0.0) + (i + 1 < n ? std::fabs(eh[i]) : 0.0);
    gl = std::min(gl, dh[i] - r);
    gu = std::max(gu, dh[i] + r);
    tnorm = std::max(tnorm, std::fabs(dh[i]) + r);
  }
  const double pad = 1e-6 * std::max(tnorm, 1.0);
  gl -= pad;
  gu += pad;
  k_tri_prep<<<grid1(n), 256, 0, st>>>(d, e, (int)n, f32, f32 + n, e2);
  k_tri_all<<<(unsigned)((n + 3) / 4), 32, 0, st>>>(d, e2, f32, f32 + n, (int)n, gl, gu, tnorm, lam);
  // 4. eigenvectors
  if (nv > 0) {
    // off-diagonal in the tridiag.cuh convention: eoff[i] couples rows i-1 and i
    double* eoff = e2;  // e2 is no longer needed once the eigenvalues are in
    cudaMemsetAsync(eoff, 0, sizeof(double), st);
    if (n > 1) cudaMemcpyAsync(eoff + 1, e, sizeof(double) * (n - 1), cudaMemcpyDeviceToDevice, st);
    k_tri_vectors<<<1, 1, 0, st>>>(d, eoff, (int)n, lam, (int)nv, tnorm, y, wk);
    k_backtransform<<<(unsigned)nv, kDenseThreads, 0, st>>>(H, n, tau, y, X);
  }
  std::vector<double> out(n);
  cudaMemcpyAsync(out.data(), lam, sizeof(double) * n, cudaMemcpyDeviceToHost, st);
  if (nv > 0) cudaMemcpyAsync(evecs, X, sizeof(double2) * n * nv, cudaMemcpyDeviceToHost, st);
  ce = cudaStreamSynchronize(st);
  if (ce == cudaSuccess) ce = cudaGetLastError();
  cleanup();
  if (ce != cudaSuccess) return cuda_fail(ce, "dense path");
  // the k-th eigenvalue is at index k; neighbours within rounding may come out
  // in either order
  std::sort(out.begin(), out.end());
  for (int64_t i = 0; i < n; ++i) eigs[i] = out[i];
  *n_out = n;
  if (stats) {
    stats->path = 1;
    stats->hv_calls = hv_calls;
    stats->hv_seconds = std::chrono::duration<double>(t1 - t0).count();
    stats->ortho_seconds = 0.0;
    stats->total_seconds = std::chrono::duration<double>(clk::now() - t0).count();
  }
  return EDG_OK;
}

}  // namespace edg
