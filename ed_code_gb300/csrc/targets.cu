// Stored targets: the orbit search of H*v done once per sector, the result
// kept in HBM as compressed sparse rows.
//
// For row i, every anti-aligned flip group g whose flipped state has an
// allowed representative j contributes one stored entry: the column j and
// the value id remap[(off[g] + variant) * n_cls + cls], where `variant` packs
// bit a of the state and the bits z of the group's chirality terms (the
// inputs of the coefficient, H_v.cpp:232-303) and `cls` is the phase class of
// the translation to the representative.  The value table
// vtab[id] = coefficient(g, variant) * phase(cls) is built on the host from
// the same term lists and deduplicated (remap).  An entry is one u32 with the
// id above the column when both fit (4 bytes), else a u32 column and a u16
// id (6 bytes).  Rows also keep their diagonal Ezz.
//
// H*v is then a sparse matrix-vector product with a value dictionary, a warp
// per slice of 32 rows (csr_row.cuh, hv_rows.cuh):
//     w_i = norm_i * sum_t vtab[vid_t] * u[col_t] + Ezz_i * v_i,
//     u_j = v_j / norm_j (a streaming pass before the row loop), or, with folded
// rows (build_targets), u = v and a vtab that includes 1 / norm_j.
// This stores the Hamiltonian's structure (4 bytes per nonzero, 56 GB for the
// 36-site Sz=0, k=0 sector) instead of searching orbits every H*v; the matrix-free
// kernels (hv.cu) remain for sectors whose entries do not fit.  The reference
// has the same trade as an option of its own (sHv on an sMatrix, H_v.cpp:3-19).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <complex>
#include <cstddef>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <utility>
#include <vector>

#include "csr_row.cuh"
#include "hv_common.cuh"
#include "hv_rows.cuh"
#include "row_walk.cuh"

namespace edg {

namespace {

constexpr int kPassThreads = 128;
constexpr int kPassTurns = 16;  // 48: 0.1 ms of 10.6 more

// Pass 1 (count) and pass 2 (fill) share this walk over the rows' targets: a
// thread owns a row and all of them go through the flip groups together, those
// of high sites first (`order`).
// Neighbouring rows are neighbouring representatives, equal in their high
// sites: a group of high sites is anti-aligned in the whole warp or in none of
// it, its search takes the same turns in
// every lane, and its rank records and remap entries come from neighbouring
// addresses.  Counting takes this walk only where k_tgt_count cannot; it needs
// no rank for a target that is alone in its orbit search (one candidate
// translate): its stabiliser is trivial, so it is allowed.  The fill pass writes
// each entry's value id as remap[(pair variant) x class], the index into the
// deduplicated value table (value_tables), packed above the column when cb > 0
// (csr_row.cuh).
//
// The pass is bound by integer issue (ALU pipe 77 %, 22 lanes of a warp active),
// not by memory.  With a warp per row and a lane per pair it took 22.8 ms on the
// 18.8-million-state 8x4 triangular sector; a lane per row on 32-bit states took
// 12.4 ms, kPassTurns times the resident CTAs instead of one turn of them 10.1 ms
// (rows differ in their searches, and the last CTAs ran alone for a third of the
// time), and group fields read where they stand, without loops over the two
// chirality sites or checks that a search on rows cannot fail, 9.6 ms.  Filling
// idle lanes was slower (10.7 ms): queues in shared memory for the targets that
// are their own representatives and for the others, so that each was taken by 32
// lanes at a time, cost more instructions than the idle lanes.
template <int kOrb, bool kFill>
__global__ void __launch_bounds__(kPassThreads) k_tgt_pass(SectorView V, int cb, int slots_at,
                                                           double* __restrict__ ezz, uint64_t* row_ptr,
                                                           uint32_t* __restrict__ col, uint16_t* __restrict__ vid) {
  __shared__ SectorParams P;
  extern __shared__ __align__(16) uint8_t sm[];
  for (int i = threadIdx.x; i < (int)(sizeof(SectorParams) / 8); i += blockDim.x)
    reinterpret_cast<uint64_t*>(&P)[i] = reinterpret_cast<const uint64_t*>(V.params)[i];
  __syncthreads();
  const PassSmem H = stage_pass<kOrb>(V, P, sm);
  __syncthreads();
  using St = typename OrbRows<kOrb>::T::State;
  const int ng = P.n_groups;
  const int64_t n_p = P.n_p, stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < n_p; base += stride) {
    const int64_t i = base + threadIdx.x;
    const bool live = i < n_p;
    const St s = live ? (St)V.reps[i] : 0;  // no pair is anti-aligned past the end
    uint64_t facs = 0, pos = 0;
    uint32_t cnt = 0;
    uint32_t len = 0;
    uint2* slot = reinterpret_cast<uint2*>(sm + slots_at) + (threadIdx.x >> 5) * ng;
    if (kFill) {
      // where the slice's slots start, and which rows have them (csr_row.cuh)
      const Slice sl = slice_at(row_ptr, i, n_p);
      len = (uint32_t)sl.len;
      uint32_t at = 0;
      __syncwarp();
      for (int k = 0; k < sl.mx; ++k) {
        const uint32_t m = __ballot_sync(0xffffffffu, sl.len > k);
        if ((threadIdx.x & 31) == 0) slot[k] = make_uint2(at, m);
        at += __popc(m);
      }
      __syncwarp();
      pos = sl.base;
    }
    RowStart<kOrb> row;
    row.set(s, P, H);
    for (int g = 0; g < ng; ++g) {
      const PassGroup& gr = H.groups[g];
      const St pm = (St)gr.mask, both = s & pm;
      const bool anti = both != 0 && both != pm;
      if (!anti) continue;
      if (!kFill) facs += gr.facadd;
      bool known;
      const Orbit o = target_orbit<kOrb, !kFill>((St)(s ^ pm), gr, row, P, H, V.n_chunks, known);
      if (!kFill) {
        if (known || position(o, V, P) >= 0) ++cnt;
        continue;
      }
      const int64_t j = kOrb >= kOrbPacked ? position_of(o.rep, V, P) : position(o, V, P);
      if (j < 0) continue;
      const uint32_t id = value_id(s, gr, o.g, V, P) * P.n_stab + P.stab_idx[o.stab];
      const uint2 sk = slot[cnt++];
      const uint64_t p = pos + sk.x + __popc(sk.y & ((1u << (threadIdx.x & 31)) - 1u));
      if (cb) {
        col[p] = (uint32_t)j | (id << cb);
      } else {
        col[p] = (uint32_t)j;
        vid[p] = (uint16_t)id;
      }
    }
    if (kFill)  // a slot left over would be a hole that the rows gather through
      for (; cnt < len; ++cnt) {
        const uint2 sk = slot[cnt];
        const uint64_t p = pos + sk.x + __popc(sk.y & ((1u << (threadIdx.x & 31)) - 1u));
        col[p] = (uint32_t)i;
        if (!cb) vid[p] = 0;
      }
    if (!kFill && live) {
      row_ptr[i] = cnt;
      ezz[i] = row_ezz(s, facs, P, H);
    }
  }
}

// The count on a packed torus.  A target without a stabiliser is allowed, so a
// row's entries are its anti-aligned pairs, less the few targets of risky rows
// (row_walk.cuh) that have one and no allowed representative.  That takes six
// instructions a pair where a search for every target took about 90 (5.7 ms for
// the 18.8 million rows of the 8x4 triangular sector, bound by integer issue);
// here 0.68 ms.
template <typename St>
struct __align__(16) CountGroup {
  uint64_t facadd;
  St mask;
};

// Has the target of an anti-aligned group no allowed representative?
template <typename St>
__device__ __noinline__ bool refused_target(St s, int at, uint32_t risk, const PrimeShifts& G, const SectorView& V,
                                            const SectorParams& P, const PassSmem& H, const St* moved) {
  return symmetric_target(s, at, risk, G, P, moved) &&
         position(orbit_torus(s ^ (St)H.groups[at].mask, P, H.nk, H.rots), V, P) < 0;
}

template <int kOrb>
__global__ void __launch_bounds__(kPassThreads) k_tgt_count(SectorView V, PrimeShifts shifts, int moved_at,
                                                            double* __restrict__ ezz, uint64_t* __restrict__ counts) {
  using St = typename OrbRows<kOrb>::T::State;
  __shared__ SectorParams P;
  __shared__ PrimeShifts G;
  extern __shared__ __align__(16) uint8_t sm[];
  for (int i = threadIdx.x; i < (int)(sizeof(SectorParams) / 8); i += blockDim.x)
    reinterpret_cast<uint64_t*>(&P)[i] = reinterpret_cast<const uint64_t*>(V.params)[i];
  if (threadIdx.x == 0) G = shifts;
  __syncthreads();
  const PassSmem H = stage_pass<kOrb>(V, P, sm);
  __syncthreads();
  const int ng = P.n_groups;
  CountGroup<St>* groups = reinterpret_cast<CountGroup<St>*>(sm + moved_at);
  St* moved = reinterpret_cast<St*>(groups + ng);
  for (int at = threadIdx.x; at < ng; at += blockDim.x) groups[at] = {H.groups[at].facadd, (St)H.groups[at].mask};
  stage_moved(G, P, H, moved);
  __syncthreads();
  const int64_t n_p = P.n_p, stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_p; i += stride) {
    const St s = (St)V.reps[i];
    uint64_t facs = 0;
    uint32_t cnt = 0;
#pragma unroll 4
    for (int g = 0; g < ng; ++g) {
      const St pm = groups[g].mask, both = s & pm;
      if (both != 0 && both != pm) {
        ++cnt;
        facs += groups[g].facadd;
      }
    }
    if (const uint32_t risk = risky_shifts(s, G, P))
      for (int g = 0; g < ng; ++g) {
        const St both = s & groups[g].mask;
        if (both != 0 && both != groups[g].mask && refused_target(s, g, risk, G, V, P, H, moved)) --cnt;
      }
    counts[i] = cnt;
    ezz[i] = row_ezz(s, facs, P, H);
  }
}

// 64-bit exclusive scan of the counts in row_ptr[0..n-1], in place (row_ptr[n] = total)
constexpr int kScan = 256, kScanPer = 16, kChunk = kScan * kScanPer;

__device__ __forceinline__ unsigned long long block_scan64(unsigned long long x, unsigned long long* tot) {
  __shared__ unsigned long long ws[kScan / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  unsigned long long inc = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  if (lane == 31) ws[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    const unsigned long long v = lane < kScan / 32 ? ws[lane] : 0ull;
    unsigned long long vi = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, vi, o);
      if (lane >= o) vi += y;
    }
    if (lane < kScan / 32) ws[lane] = vi - v;
    if (lane == kScan / 32 - 1) *tot = vi;
  }
  __syncthreads();
  const unsigned long long r = inc - x + ws[wid];
  __syncthreads();
  return r;
}

__global__ void __launch_bounds__(kScan) k_scan64_chunks(const uint64_t* __restrict__ in, int64_t n,
                                                          unsigned long long* __restrict__ sums) {
  const int64_t b = (int64_t)blockIdx.x * kChunk + (int64_t)threadIdx.x * kScanPer;
  unsigned long long s = 0;
  for (int k = 0; k < kScanPer; ++k)
    if (b + k < n) s += in[b + k];
  __shared__ unsigned long long tot;
  block_scan64(s, &tot);
  if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(kScan) k_scan64_sums(unsigned long long* __restrict__ sums, int64_t n,
                                                        unsigned long long* __restrict__ total) {
  __shared__ unsigned long long tot;
  unsigned long long carry = 0;
  for (int64_t b0 = 0; b0 < n; b0 += kScan) {
    const int64_t i = b0 + threadIdx.x;
    const unsigned long long x = i < n ? sums[i] : 0ull;
    const unsigned long long e = block_scan64(x, &tot);
    if (i < n) sums[i] = carry + e;
    __syncthreads();
    carry += tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = carry;
}

__global__ void __launch_bounds__(kScan) k_scan64_apply(uint64_t* io, int64_t n,
                                                         const unsigned long long* __restrict__ offs,
                                                         const unsigned long long* __restrict__ total) {
  const int64_t b = (int64_t)blockIdx.x * kChunk + (int64_t)threadIdx.x * kScanPer;
  unsigned long long s = 0;
  for (int k = 0; k < kScanPer; ++k)
    if (b + k < n) s += io[b + k];
  __shared__ unsigned long long tot;
  unsigned long long run = block_scan64(s, &tot) + offs[blockIdx.x];
  for (int k = 0; k < kScanPer; ++k)
    if (b + k < n) {
      const uint64_t x = io[b + k];
      io[b + k] = run;
      run += x;
    }
  if (blockIdx.x == 0 && threadIdx.x == 0) io[n] = *total;
}

// u_j = v_j / norm_j
template <typename Real>
__global__ void k_u_scale(const typename CT2<Real>::T* __restrict__ v, const uint8_t* __restrict__ lid,
                          const double* __restrict__ nrm_inv_tab, int64_t n, typename CT2<Real>::T* __restrict__ u) {
  __shared__ Real tab[65];
  for (int k = threadIdx.x; k < 65; k += blockDim.x) tab[k] = (Real)nrm_inv_tab[k];
  __syncthreads();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    typename CT2<Real>::T x = v[i];
    const Real s = tab[lid[i]];
    x.x *= s;
    x.y *= s;
    u[i] = x;
  }
}

// The same u, for a v that the device reads in place (page-locked host memory
// mapped into its address space), plus a device copy vd of v for the rows'
// diagonal term: one pass over the host link, four loads in flight per
// thread, instead of a copy-engine copy followed by the u pass.  u gets the
// bits k_u_scale gives it.
// u may be nullptr (rows that gather v itself).
template <typename Real>
__global__ void k_u_scale_in(const typename CT2<Real>::T* __restrict__ v, const uint8_t* __restrict__ lid,
                             const double* __restrict__ nrm_inv_tab, int64_t n, typename CT2<Real>::T* __restrict__ vd,
                             typename CT2<Real>::T* __restrict__ u) {
  using CT = typename CT2<Real>::T;
  __shared__ Real tab[65];
  for (int k = threadIdx.x; k < 65; k += blockDim.x) tab[k] = (Real)nrm_inv_tab[k];
  __syncthreads();
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (; i + 3 * stride < n; i += 4 * stride) {
    CT x[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) x[k] = v[i + k * stride];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int64_t r = i + k * stride;
      vd[r] = x[k];
      if (!u) continue;
      const Real s = tab[lid[r]];
      x[k].x *= s;
      x[k].y *= s;
      u[r] = x[k];
    }
  }
  for (; i < n; i += stride) {
    CT x = v[i];
    vd[i] = x;
    if (!u) continue;
    const Real s = tab[lid[i]];
    x.x *= s;
    x.y *= s;
    u[i] = x;
  }
}

// Grid of a grid-stride kernel: `turns` times the CTAs that fit on every SM at
// once, no more than the work needs.
template <typename K>
int grid_for(K kernel, size_t smem, int64_t work, int threads, int turns) {
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
  if (per_sm < 1) per_sm = 1;
  const int64_t want = (work + threads - 1) / threads;
  return (int)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)sms * per_sm * turns));
}

// The row kernel's tuned choices as template arguments: entries of a row in
// flight (csr_lpr / 2: 4, 8 or 16; at most 8 in FP64, whose entries are twice
// as large), cache policy, entry format, pipelining.  A value table too large
// for shared memory is read through L1 with 8 entries in flight.
template <typename Real, int kPol, int kFmt>
cudaError_t launch_rows_f(const Sector& S, const void* v, const void* u, void* w, int64_t r0, int64_t r1,
                          cudaStream_t st) {
  constexpr int kMost = sizeof(Real) == 4 ? 16 : 8;
  if (sizeof(typename CT2<Real>::T) * S.n_rvals > 96 * 1024)
    return launch_rows_k<Real, 1, false, kPol, kFmt, 8, 8, false>(S, v, u, w, r0, r1, st);
  if (S.csr_pipe) switch (S.csr_lpr) {
      case 8: return launch_rows_k<Real, 1, true, kPol, kFmt, 4, 4, true>(S, v, u, w, r0, r1, st);
      case 16: return launch_rows_k<Real, 1, true, kPol, kFmt, 8, 8, true>(S, v, u, w, r0, r1, st);
      default: return launch_rows_k<Real, 1, true, kPol, kFmt, kMost, kMost, true>(S, v, u, w, r0, r1, st);
    }
  switch (S.csr_lpr) {
    case 8: return launch_rows_k<Real, 1, true, kPol, kFmt, 4, 4, false>(S, v, u, w, r0, r1, st);
    case 16: return launch_rows_k<Real, 1, true, kPol, kFmt, 8, 8, false>(S, v, u, w, r0, r1, st);
    default: return launch_rows_k<Real, 1, true, kPol, kFmt, kMost, kMost, false>(S, v, u, w, r0, r1, st);
  }
}

template <typename Real>
cudaError_t launch_rows_t(const Sector& S, const void* v, const void* u, void* w, int64_t r0, int64_t r1,
                          cudaStream_t st) {
  if (S.pack_cb)
    return S.csr_pol == 2 ? launch_rows_f<Real, 2, kPacked>(S, v, u, w, r0, r1, st)
                          : launch_rows_f<Real, 1, kPacked>(S, v, u, w, r0, r1, st);
  return S.csr_pol == 2 ? launch_rows_f<Real, 2, kSplit>(S, v, u, w, r0, r1, st)
                        : launch_rows_f<Real, 1, kSplit>(S, v, u, w, r0, r1, st);
}

int64_t gcd64(int64_t a, int64_t b) {
  while (b) {
    const int64_t t = a % b;
    a = b;
    b = t;
  }
  return a < 0 ? -a : a;
}

}  // namespace

void free_targets(Sector& S) {
  void* ptrs[] = {S.row_ptr, S.col, S.vid, S.ezz, S.row_values, S.ubuf.ptr};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  S.row_ptr = nullptr;
  S.col = nullptr;
  S.vid = nullptr;
  S.pack_cb = 0;
  S.ezz = nullptr;
  S.row_values = nullptr;
  S.rtab64 = nullptr;
  S.rtab32 = nullptr;
  S.n_rvals = 0;
  S.folded = false;
  S.ubuf = DeviceBuffer{};
  S.P.n_targets = 0;
  S.device_bytes -= S.targets_bytes;
  S.targets_bytes = 0;
}

// Value tables of a sector: for every flip group and variant (bit a of the
// state, the bits z of its chirality terms) and phase class of a translation,
// the id of coefficient x phase among the distinct values (compared by bits;
// with uniform couplings a handful).  Sets P.n_cls and P.g2cls.
int value_tables(SectorParams& P, const std::vector<TermGroup>& groups, const std::vector<ChTerm>& ch,
                 ValueTables& T) {
  if (P.n_groups > kMaxRowSlots) {
    T.why = "stored targets need at most 256 flip groups";
    return EDG_ERR_UNSUPPORTED;
  }
  // phase classes: translation (a, b, c) has phase index
  // (kx a L2 L3 + ky b L1 L3 + kz c L1 L2) mod G, G = L1 L2 L3 (c = 0 in 2-D)
  const int G = P.L1 * P.L2 * P.L3;
  const int64_t d = gcd64(gcd64(gcd64((int64_t)P.kx * P.L2 * P.L3, (int64_t)P.ky * P.L1 * P.L3),
                                (int64_t)P.kz * P.L1 * P.L2), G);
  const int n_cls = (int)(G / (d ? d : G));
  std::vector<std::complex<double>> cph(n_cls);
  std::vector<char> seen(n_cls, 0);
  for (int c3 = 0; c3 < P.L3; ++c3)
    for (int b = 0; b < P.L2; ++b)
      for (int a = 0; a < P.L1; ++a) {
        const int g = a + P.L1 * b + P.L1 * P.L2 * c3;
        const int64_t m = ((int64_t)P.kx * a * P.L2 * P.L3 + (int64_t)P.ky * b * P.L1 * P.L3 +
                           (int64_t)P.kz * c3 * P.L1 * P.L2) % G;
        const int c = (int)(m / (d ? d : G));
        P.g2cls[g] = (uint8_t)c;
        if (!seen[c]) {  // the first translation of a class gives its phase value
          seen[c] = 1;
          cph[c] = std::complex<double>(P.ph_re[g], P.ph_im[g]);
        }
      }
  P.n_cls = n_cls;
  int64_t n_var = 0;
  std::vector<uint16_t> voff(P.n_groups);
  for (int g = 0; g < P.n_groups; ++g) {
    const int nch = groups[g].ch_end - groups[g].ch_begin;
    if (nch > kMaxChPerGroup) {
      T.why = "stored targets: more than 4 chirality terms on one pair";
      return EDG_ERR_UNSUPPORTED;
    }
    if (n_var > 65535) break;
    voff[g] = (uint16_t)n_var;
    n_var += 2 << nch;
  }
  if (n_var * n_cls > 65536) {
    T.why = "stored targets: more than 65536 distinct values";
    return EDG_ERR_UNSUPPORTED;
  }
  // distinct coefficients first, then their products with the phases
  using Key = std::pair<uint64_t, uint64_t>;
  auto key_of = [](std::complex<double> z) {
    const double re = z.real(), im = z.imag();
    Key k;
    std::memcpy(&k.first, &re, 8);
    std::memcpy(&k.second, &im, 8);
    return k;
  };
  std::map<Key, int> coefs;
  std::map<Key, uint16_t> values;
  std::vector<std::vector<uint16_t>> ids;  // of a coefficient, by class
  T.remap.resize(n_var * n_cls);
  for (int g = 0; g < P.n_groups; ++g) {
    const TermGroup& gr = groups[g];
    const int nch = gr.ch_end - gr.ch_begin;
    for (int variant = 0; variant < (2 << nch); ++variant) {
      const int cs = variant & 1;
      std::complex<double> c(gr.Bre[cs], gr.Bim[cs]);
      for (int q = 0; q < nch; ++q) {
        const ChTerm& t = ch[gr.ch_begin + q];
        const double sg = ((variant >> (q + 1)) & 1) ? 1.0 : -1.0;
        c += sg * std::complex<double>(t.Are[cs], t.Aim[cs]);
      }
      const auto at = coefs.emplace(key_of(c), (int)ids.size());
      if (at.second) {
        ids.emplace_back(n_cls);
        for (int cl = 0; cl < n_cls; ++cl) {
          const std::complex<double> val = c * cph[cl];
          const auto v = values.emplace(key_of(val), (uint16_t)T.v64.size());
          if (v.second) {
            T.v64.push_back(make_double2(val.real(), val.imag()));
            T.v32.push_back(make_float2((float)val.real(), (float)val.imag()));
          }
          ids.back()[cl] = v.first->second;
        }
      }
      std::copy(ids[at.first->second].begin(), ids[at.first->second].end(),
                T.remap.begin() + (size_t)(voff[g] + variant) * n_cls);
    }
  }
  // The rows take the groups of high sites first: consecutive representatives
  // differ in their low sites, so a pair of high sites is anti-aligned in all
  // rows of a warp or in none, and its targets in neighbouring rows are
  // neighbours.
  std::vector<uint16_t> order(P.n_groups);
  for (int g = 0; g < P.n_groups; ++g) order[g] = (uint16_t)g;
  std::stable_sort(order.begin(), order.end(), [&](int p, int q) {
    return groups[p].a != groups[q].a ? groups[p].a > groups[q].a : groups[p].b > groups[q].b;
  });
  T.voff.swap(voff);
  T.order.swap(order);
  return EDG_OK;
}

// Returns EDG_OK, or a reason (EDG_ERR_NOMEM / EDG_ERR_UNSUPPORTED) with the
// sector left on the matrix-free kernels.
int build_targets(Sector& S, int64_t max_bytes, std::string& err) {
  SectorParams& P = S.P;
  if (S.col) return EDG_OK;
  if (P.use_chch) {
    err = "stored targets do not cover ChCh terms";
    return EDG_ERR_UNSUPPORTED;
  }
  if (!S.n_vals) {
    err = S.values_err;
    return EDG_ERR_UNSUPPORTED;
  }
  // Packed entries when the value ids and the columns fit one u32 together:
  // vb bits of value id above cb = 32 - vb column bits, n_p < 2^cb.
  // EDG_ROW_FORMAT=split keeps the two arrays (for comparisons).
  auto pack_bits = [&](int64_t values) {
    int vb = 1;
    while (((int64_t)1 << vb) < values) ++vb;
    return vb < 32 && P.n_p < (int64_t(1) << (32 - vb)) ? 32 - vb : 0;
  };
  // Folded rows: the values include the target's 1/norm, one value per distinct
  // stabiliser count, and the rows gather v itself: no pass over v, no u.  Unless
  // that makes the entries six bytes (36 sites: 2^4 values at most beside
  // the columns) or the table large: the pass is 1 % of those sectors' H v, while
  // on a small sector it is one launch of two (16 sites, with fewer queries a launch: 11.7 -> 7.5 us).
  const int n_stab = std::max(1, __builtin_popcountll(S.lids));
  const int64_t n_fold = (int64_t)S.n_vals * n_stab;
  S.folded = n_fold <= 4096 && (pack_bits(n_fold) || !pack_bits(S.n_vals));
  S.n_rvals = S.folded ? (int)n_fold : S.n_vals;
  P.n_stab = S.folded ? n_stab : 1;
  std::memset(P.stab_idx, 0, sizeof P.stab_idx);
  const char* fmt_env = std::getenv("EDG_ROW_FORMAT");
  const bool want_split = fmt_env && std::strcmp(fmt_env, "split") == 0;
  S.pack_cb = want_split ? 0 : pack_bits(S.n_rvals);
  const double entry_bytes = S.pack_cb ? 4.0 : 6.0;
  size_t fold_bytes = 0;
  if (S.folded) {
    std::vector<uint8_t> both(24 * n_fold);
    double2* r64 = reinterpret_cast<double2*>(both.data());
    float2* r32 = reinterpret_cast<float2*>(both.data() + 16 * n_fold);
    int at = 0;
    for (int l = 1; l <= 64; ++l) {
      if (!((S.lids >> (l - 1)) & 1ull)) continue;
      P.stab_idx[l] = (uint8_t)at;
      for (int v = 0; v < S.n_vals; ++v) {
        const double2 x = make_double2(S.values_host[v].x * P.nrm_inv[l], S.values_host[v].y * P.nrm_inv[l]);
        r64[(size_t)v * n_stab + at] = x;
        r32[(size_t)v * n_stab + at] = make_float2((float)x.x, (float)x.y);
      }
      ++at;
    }
    fold_bytes = both.size();
    cudaError_t ce = cudaMalloc(&S.row_values, fold_bytes);
    if (ce == cudaSuccess) ce = cudaMemcpy(S.row_values, both.data(), fold_bytes, cudaMemcpyHostToDevice);
    if (ce != cudaSuccess) {
      cudaGetLastError();
      free_targets(S);
      err = "stored targets: out of device memory for the value table";
      return EDG_ERR_NOMEM;
    }
    S.rtab64 = static_cast<double2*>(S.row_values);
    S.rtab32 = reinterpret_cast<float2*>(S.rtab64 + n_fold);
  } else {
    S.rtab64 = S.vtab64;
    S.rtab32 = S.vtab32;
  }

  cudaStream_t st = S.stream;
  const int64_t n = P.n_p;
  unsigned long long *sums = nullptr, *tot = nullptr;
  const int64_t n_chunks = (n + kChunk - 1) / kChunk;
  cudaError_t e = cudaMemcpy(S.dP, &P, sizeof(P), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMalloc(&sums, sizeof(unsigned long long) * (n_chunks + 1));
  if (e == cudaSuccess) tot = sums + n_chunks;
  if (e == cudaSuccess) e = cudaMalloc(&S.row_ptr, sizeof(uint64_t) * (n + 1));
  if (e == cudaSuccess) e = cudaMalloc(&S.ezz, sizeof(double) * n);
  auto cleanup = [&]() { cudaFree(sums); };
  if (e != cudaSuccess) {
    cleanup();
    free_targets(S);
    err = "stored targets: out of device memory for the row data";
    return EDG_ERR_NOMEM;
  }
  const int orb = orb_of(P);
  const size_t terms = align16(pass_smem_bytes(P, orb, S.V.row_bits, S.V.n_chunks, S.V.n_perm));
  auto pass = [&](auto kern, size_t smem) {
    kern<<<grid_for(kern, smem, n, kPassThreads, kPassTurns), kPassThreads, smem, st>>>(
        S.V, S.pack_cb, (int)terms, S.ezz, S.row_ptr, S.col, S.vid);
  };
  const PrimeShifts G = prime_shifts(P);
  auto count = [&](auto kern, size_t state) {
    const size_t smem = terms + P.n_groups * (16 + 8 + state * G.n);
    kern<<<grid_for(kern, smem, n, kPassThreads, kPassTurns), kPassThreads, smem, st>>>(S.V, G, (int)terms, S.ezz,
                                                                                            S.row_ptr);
  };
  if (orb == kOrbPacked) count(k_tgt_count<kOrbPacked>, 4);
  else if (orb == kOrbPacked32) count(k_tgt_count<kOrbPacked32>, 4);
  else if (orb == kOrbPacked64) count(k_tgt_count<kOrbPacked64>, 8);
  else if (orb == kOrbTorus) pass(k_tgt_pass<kOrbTorus, false>, terms);
  else pass(k_tgt_pass<kOrbWalk, false>, terms);
  k_scan64_chunks<<<(unsigned)n_chunks, kScan, 0, st>>>(S.row_ptr, n, sums);
  k_scan64_sums<<<1, kScan, 0, st>>>(sums, n_chunks, tot);
  k_scan64_apply<<<(unsigned)n_chunks, kScan, 0, st>>>(S.row_ptr, n, sums, tot);
  unsigned long long nnz = 0;
  e = cudaMemcpyAsync(&nnz, tot, sizeof(nnz), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  size_t free_b = 0, total_b = 0;
  cudaMemGetInfo(&free_b, &total_b);
  const double need = entry_bytes * (double)nnz + 16.0 * (double)n;
  if (e != cudaSuccess || need > (double)max_bytes || need > 0.9 * (double)free_b) {
    cleanup();
    free_targets(S);
    err = e != cudaSuccess ? std::string("stored targets: ") + cudaGetErrorString(e)
                           : "stored targets do not fit in the allowed device memory";
    return e != cudaSuccess ? EDG_ERR_CUDA : EDG_ERR_NOMEM;
  }
  e = cudaMalloc(&S.col, sizeof(uint32_t) * std::max<unsigned long long>(1, nnz));
  if (e == cudaSuccess && !S.pack_cb) e = cudaMalloc(&S.vid, sizeof(uint16_t) * std::max<unsigned long long>(1, nnz));
  if (e == cudaSuccess && !S.folded) e = cudaMalloc(&S.ubuf.ptr, (size_t)(16 * n));
  if (e != cudaSuccess) {
    cleanup();
    free_targets(S);
    err = "stored targets: out of device memory";
    return EDG_ERR_NOMEM;
  }
  S.ubuf.bytes = S.folded ? 0 : (size_t)(16 * n);
  const size_t fill = terms + kPassThreads / 32 * sizeof(uint2) * P.n_groups;
  if (orb == kOrbPacked) pass(k_tgt_pass<kOrbPacked, true>, fill);
  else if (orb == kOrbPacked32) pass(k_tgt_pass<kOrbPacked32, true>, fill);
  else if (orb == kOrbPacked64) pass(k_tgt_pass<kOrbPacked64, true>, fill);
  else if (orb == kOrbTorus) pass(k_tgt_pass<kOrbTorus, true>, fill);
  else pass(k_tgt_pass<kOrbWalk, true>, fill);
  e = cudaStreamSynchronize(st);
  cleanup();
  if (e != cudaSuccess) {
    free_targets(S);
    err = std::string("stored targets: ") + cudaGetErrorString(e);
    return EDG_ERR_CUDA;
  }
  P.n_targets = (int64_t)nnz;
  S.targets_bytes = (S.pack_cb ? 4 : 6) * nnz + 8 * (n + 1) + 8 * n + S.ubuf.bytes + fold_bytes;
  S.device_bytes += S.targets_bytes;
  e = cudaMemcpy(S.dP, &P, sizeof(P), cudaMemcpyHostToDevice);
  return e == cudaSuccess ? EDG_OK : EDG_ERR_CUDA;
}

// Entries in flight (lanes per row / 2), cache policy, CTAs per SM and
// pipelining.  lpr in {8, 16, 32} fixes the first; 0 times all of them.  First
// every (lanes, pipelining 0/1, CTA cap in {as many as fit, 4, 3, 2, 1}) with
// cache policy 1, the faster one at 24 to 36 sites (392 us against 482 us at 30
// sites, 54.8 ms against 61.8 ms at 36), then the best of those with policy 2.
// Each combination runs twice (FP32; once on sectors whose launch takes over
// 5 ms) after one warm-up launch, and the fastest is kept.  The CTA cap matters
// because the gathers reuse u through L2: fewer rows in flight keep their
// targets' window of u smaller.  ms_out[k] receives the best time of lane
// count 8, 16, 32 (-1 when not timed).
int tune_rows(Sector& S, int lpr, int* chosen, double* ms_out) {
  if (!S.col) {
    if (chosen) *chosen = 0;
    return EDG_OK;  // matrix-free sectors have nothing to tune
  }
  if (lpr != 0 && lpr != 8 && lpr != 16 && lpr != 32) return EDG_ERR_INVALID;
  const int64_t n = S.P.n_p;
  float2 *v = nullptr, *w = nullptr;
  if (cudaMalloc(&v, sizeof(float2) * n) != cudaSuccess || cudaMalloc(&w, sizeof(float2) * n) != cudaSuccess) {
    cudaFree(v);
    return EDG_ERR_NOMEM;
  }
  cudaStream_t st = S.stream;
  cudaMemsetAsync(v, 0, sizeof(float2) * n, st);
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  bool warm = false;
  int reps = 2;  // one launch per trial once a launch takes over 5 ms
  auto time_it = [&]() {
    if (!warm) launch_hv_stored(S, v, w, false, st);
    warm = true;
    cudaEventRecord(e0, st);
    for (int r = 0; r < reps; ++r) launch_hv_stored(S, v, w, false, st);
    cudaEventRecord(e1, st);
    cudaEventSynchronize(e1);
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    ms /= reps;
    if (ms > 5.f) reps = 1;
    return ms;
  };
  const int cand[3] = {8, 16, 32};
  const int caps[5] = {0, 4, 3, 2, 1};
  int best = 8, best_cps = 0, best_pipe = 1;
  float best_ms = 1e30f;
  for (int k = 0; k < 3; ++k) {
    if (ms_out) ms_out[k] = -1;
    if (lpr != 0 && cand[k] != lpr) continue;
    for (int pipe = 0; pipe < 2; ++pipe) {
      for (int c = 0; c < 5; ++c) {
        S.csr_lpr = cand[k];
        S.csr_pol = 1;
        S.csr_cps = caps[c];
        S.csr_pipe = pipe;
        const float ms = time_it();
        if (ms_out && (ms_out[k] < 0 || ms < ms_out[k])) ms_out[k] = ms;
        if (ms < best_ms) {
          best_ms = ms;
          best = cand[k];
          best_cps = caps[c];
          best_pipe = pipe;
        }
      }
    }
  }
  S.csr_lpr = best;
  S.csr_cps = best_cps;
  S.csr_pipe = best_pipe;
  S.csr_pol = 2;
  const float ms2 = time_it();
  const int k = best == 8 ? 0 : best == 16 ? 1 : 2;
  if (ms_out && ms2 < ms_out[k]) ms_out[k] = ms2;
  if (ms2 >= best_ms) S.csr_pol = 1;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(v);
  cudaFree(w);
  if (chosen) *chosen = best;
  return cudaGetLastError() == cudaSuccess ? EDG_OK : EDG_ERR_CUDA;
}

cudaError_t launch_u(const Sector& S, const void* v, void* u, bool fp64, cudaStream_t st) {
  const int64_t n = S.P.n_p;
  const int grid = (int)std::min<int64_t>((n + 255) / 256, 152 * 32);
  const double* nrm_inv = params_field(S, offsetof(SectorParams, nrm_inv));
  if (fp64)
    k_u_scale<double><<<grid, 256, 0, st>>>(static_cast<const double2*>(v), S.lid, nrm_inv, n, static_cast<double2*>(u));
  else
    k_u_scale<float><<<grid, 256, 0, st>>>(static_cast<const float2*>(v), S.lid, nrm_inv, n, static_cast<float2*>(u));
  return cudaGetLastError();
}

cudaError_t launch_hv_rows(const Sector& S, const void* v, const void* u, void* w, bool fp64, int64_t r0, int64_t r1,
                           cudaStream_t st) {
  return fp64 ? launch_rows_t<double>(S, v, u, w, r0, r1, st) : launch_rows_t<float>(S, v, u, w, r0, r1, st);
}

cudaError_t launch_u_in(const Sector& S, const void* v_src, void* v_dst, bool fp64, cudaStream_t st) {
  const int64_t n = S.P.n_p;
  const int grid = (int)std::min<int64_t>((n + 255) / 256, 152 * 16);
  const double* nrm_inv = params_field(S, offsetof(SectorParams, nrm_inv));
  if (fp64)
    k_u_scale_in<double><<<grid, 256, 0, st>>>(static_cast<const double2*>(v_src), S.lid, nrm_inv, n,
                                               static_cast<double2*>(v_dst), static_cast<double2*>(S.ubuf.ptr));
  else
    k_u_scale_in<float><<<grid, 256, 0, st>>>(static_cast<const float2*>(v_src), S.lid, nrm_inv, n,
                                              static_cast<float2*>(v_dst), static_cast<float2*>(S.ubuf.ptr));
  return cudaGetLastError();
}

cudaError_t launch_hv_stored(const Sector& S, const void* v, void* w, bool fp64, cudaStream_t st) {
  if (S.folded) return launch_hv_rows(S, v, v, w, fp64, 0, S.P.n_p, st);
  const cudaError_t e = launch_u(S, v, S.ubuf.ptr, fp64, st);
  return e == cudaSuccess ? launch_hv_rows(S, v, S.ubuf.ptr, w, fp64, 0, S.P.n_p, st) : e;
}

}  // namespace edg
