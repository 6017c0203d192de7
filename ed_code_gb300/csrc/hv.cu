// Matrix-free H*v in the momentum basis: the role of sHv (H_v.cpp:192-357).
//
// k_hv_free takes every Hamiltonian whose values fit the value tables
// (targets.cu): a thread per row walks the flip groups as the stored rows'
// build does (row_walk.cuh), leaves what it finds in shared memory and sums it
// as the stored rows are summed (csr_row.cuh).  k_hv takes the rest: ChCh terms
// and couplings of many values.
//
// k_hv: one thread owns one basis row i (coalesced loads of reps/lid/v and a
// coalesced store of w).  Per row:
//   * the anti-aligned flip groups are found 64 at a time as a bit mask
//     (groups merge every bond and chirality term that flips the same pair);
//   * each one is flipped with one XOR, its representative and translation
//     come from the orbit search (row-rotation candidates on row-major tori,
//     the reference's walk otherwise), its position j from the value-indexed
//     rank records, its phase and norm ratio from shared-memory tables;
//   * w_i = sum_targets c(s)*phase*norm_i/norm_j*v_j + Ezz(s)*v_i, with
//     Ezz(s) = sum_bonds lambda*J/4 - 2*sum_{anti-aligned} lambda*J/4.
// ChCh bowtie terms (H_v.cpp:305-353) run as a separate per-row loop, only
// when |ChCh| > 1e-16 as in the reference.
//
// The grid is persistent (a fixed number of CTAs per SM striding over rows),
// so the per-CTA shared-memory staging of the term tables is paid once per
// CTA, not once per 256 rows.
#include <cuda_runtime.h>

#include <algorithm>

#include "csr_row.cuh"
#include "hv_common.cuh"
#include "launch.cuh"
#include "row_walk.cuh"

namespace edg {

namespace {


template <typename Real, bool kTorus, bool kChCh>
__global__ void __launch_bounds__(kHvThreads, 4) k_hv(SectorView V, const typename C2<Real>::T* __restrict__ v,
                                                   typename C2<Real>::T* __restrict__ w) {
  using CT = typename C2<Real>::T;
  __shared__ SectorParams P;
  extern __shared__ __align__(16) uint8_t sm[];
  for (int i = threadIdx.x; i < (int)(sizeof(SectorParams) / 8); i += blockDim.x)
    reinterpret_cast<uint64_t*>(&P)[i] = reinterpret_cast<const uint64_t*>(V.params)[i];
  __syncthreads();
  const HvSmem<Real> H = stage_hv<Real, kTorus>(V, P, sm);
  __syncthreads();

  const int64_t n_p = P.n_p;
  const int ng = P.n_groups;
  const bool use_ch = P.use_ch != 0;
  const Real total_fac = (Real)P.total_fac;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_p; i += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t s = __ldg(reinterpret_cast<const unsigned long long*>(V.reps) + i);
    const int li = __ldg(V.lid + i);
    const CT vi = v[i];
    const Real norm_i = H.nrm[li];
    Real accr = 0, acci = 0, anti = 0;
    RowInfo ri{0, false};
    if (kTorus) ri = torus_row_info(s, P, H);
    const int top = P.L2 - 1;
    const uint64_t rmask = (1ull << P.L1) - 1ull;
    for (int g0 = 0; g0 < ng; g0 += 64) {
      const int gn = min(64, ng - g0);
      uint64_t am = 0;
      for (int k = 0; k < gn; ++k) {
        const uint64_t m = H.groups[g0 + k].mask;
        am |= (uint64_t)(popc64(s & m) == 1) << k;
      }
      while (am) {
        const int g = g0 + ffs64(am);
        am &= am - 1;
        const SmemGroup<Real>& gr = H.groups[g];
        anti += gr.fac;
        const int cs = (int)((s >> gr.a) & 1u);
        Real cr = gr.Bre[cs], ci = gr.Bim[cs];
        if (use_ch) {
          for (int m = gr.ch_begin; m < gr.ch_end; ++m) {
            const SmemCh<Real>& c = H.ch[m];
            const Real sg = ((s >> c.z) & 1u) ? Real(1) : Real(-1);
            cr += sg * c.Are[cs];
            ci += sg * c.Aim[cs];
          }
        }
        const uint64_t t = s ^ gr.mask;
        Orbit o;
        bool fast = false;
        if (kTorus && ri.uniq && gr.ya != top && gr.yb != top) {
          const int na = H.nk[(int)((t >> (P.L1 * gr.ya)) & rmask)];
          const int nb = H.nk[(int)((t >> (P.L1 * gr.yb)) & rmask)];
          if (na > ri.mstar && nb > ri.mstar) {
            o.rep = t;
            o.g = 0;
            o.stab = 1;
            fast = true;
          }
        }
        if (!fast) o = search<Real, kTorus>(t, P, H, V.n_chunks);
        const int64_t j = position(o, V, P);
        if (j >= 0) {
          const Real sc = norm_i * H.nrm_inv[o.stab];
          const Real pr = H.ph_re[o.g], pi = H.ph_im[o.g];
          const Real er = (cr * pr - ci * pi) * sc;
          const Real ei = (cr * pi + ci * pr) * sc;
          const CT vj = v[j];
          accr += er * vj.x - ei * vj.y;
          acci += er * vj.y + ei * vj.x;
        }
      }
    }
    if (kChCh) {
      // ChCh (H_v.cpp:305-353): two successive pair flips, term by term.
      const Real chch = (Real)(P.ChCh * 0.25 * 0.25);
      for (int k = 0; k < P.n_bowties; ++k) {
        const Bowtie b = V.bows[k];
        const int tx = (int)((s >> b.x) & 1u), ty = (int)((s >> b.y) & 1u);
        if (tx == ty) continue;
        // ch_sgn1 = (ty ? i : -i), negated when bit z of the flipped state is 0
        Real s1 = ty ? Real(1) : Real(-1);
        const uint64_t tmp = s ^ ((1ull << b.x) | (1ull << b.y));
        if (!((tmp >> b.z) & 1u)) s1 = -s1;
        const int tp = (int)((tmp >> b.p) & 1u), tq = (int)((tmp >> b.q) & 1u);
        if (tp == tq) continue;
        Real s2 = tq ? Real(1) : Real(-1);
        const uint64_t tmp2 = tmp ^ ((1ull << b.p) | (1ull << b.q));
        if (!((tmp2 >> b.r) & 1u)) s2 = -s2;
        Orbit o;
        const int64_t j = locate<Real, kTorus>(tmp2, V, P, H, o);
        if (j >= 0) {
          // (i s1)(i s2) = -s1 s2
          const Real sc = -chch * s1 * s2 * norm_i * H.nrm_inv[o.stab];
          const Real er = H.ph_re[o.g] * sc, ei = H.ph_im[o.g] * sc;
          const CT vj = v[j];
          accr += er * vj.x - ei * vj.y;
          acci += er * vj.y + ei * vj.x;
        }
      }
    }
    const Real ezz = total_fac - Real(2) * anti;
    CT out;
    out.x = accr + ezz * vi.x;
    out.y = acci + ezz * vi.y;
    w[i] = out;
  }
}

// The matrix-free H*v over the value tables.  The warps of a CTA each take 32
// neighbouring rows; the lanes go through the flip groups together, and a
// target found goes into the lane's next slot of the warp's queue in shared
// memory (column and value id).  When a lane's queue is full, or the groups are
// through, the warp sums the slots as it would stored ones.  So the search runs
// on rows that take the same turns, the gathers of several targets are in
// flight together, and a target costs four FP64 multiply-adds (two when real)
// instead of 16 FP64 instructions for its coefficient, phase, norm and product,
// which was what bound it (FP64 pipe 83 % busy): 2,484 us -> 1,026 us at 28 sites in
// FP64.  The gathered entries would need v / norm; with trivial stabilisers the
// norms are one factor of the row, and the few targets with others are added
// apart.
constexpr int kFreeThreads = 128, kQueue = 16;

// (r, i) += c x sc; a call, so that its FP64 instructions are not predicated
// into every turn of the walk
template <typename Real, typename CT>
__device__ __noinline__ void add_rest(CT c, CT x, Real sc, Real& r, Real& i) {
  r += (c.x * x.x - c.y * x.y) * sc;
  i += (c.x * x.y + c.y * x.x) * sc;
}

template <typename Real>
size_t free_smem_bytes(const Sector& S, int orb) {
  return align16(pass_smem_bytes(S.P, orb, S.V.row_bits, S.V.n_chunks, S.V.n_perm)) +
         sizeof(typename CT2<Real>::T) * S.n_vals;
}

template <typename Real, int kOrb>
__global__ void __launch_bounds__(kFreeThreads) k_hv_free(SectorView V, const typename CT2<Real>::T* __restrict__ vtab,
                                                          int n_vals, int table_at, int wps,
                                                          const typename CT2<Real>::T* __restrict__ v,
                                                          typename CT2<Real>::T* __restrict__ w) {
  using CT = typename CT2<Real>::T;
  __shared__ SectorParams P;
  __shared__ Real nrm[65], nrm_inv[65];
  __shared__ uint32_t q_col[kFreeThreads / 32][kQueue][32];
  __shared__ uint16_t q_id[kFreeThreads / 32][kQueue][32];
  __shared__ Real part_sum[kFreeThreads / 32][2][32];
  __shared__ uint64_t part_facs[kFreeThreads / 32][32];
  extern __shared__ __align__(16) uint8_t sm[];
  for (int i = threadIdx.x; i < (int)(sizeof(SectorParams) / 8); i += blockDim.x)
    reinterpret_cast<uint64_t*>(&P)[i] = reinterpret_cast<const uint64_t*>(V.params)[i];
  __syncthreads();
  const PassSmem H = stage_pass<kOrb>(V, P, sm);
  CT* tab = reinterpret_cast<CT*>(sm + table_at);
  for (int k = threadIdx.x; k < n_vals; k += blockDim.x) tab[k] = vtab[k];
  for (int k = threadIdx.x; k < 65; k += blockDim.x) {
    nrm[k] = (Real)P.nrm[k];
    nrm_inv[k] = (Real)P.nrm_inv[k];
  }
  __syncthreads();
  using St = typename OrbRows<kOrb>::T::State;
  const int ng = P.n_groups, lane = threadIdx.x & 31;
  auto& qc = q_col[threadIdx.x >> 5];
  auto& qi = q_id[threadIdx.x >> 5];
  const uint64_t pl = l2_evict_last();
  const RowsView<Real> R{nullptr, nullptr, nullptr, tab, v, 0};
  // wps warps share a slice of 32 rows, with every wps-th group each
  const int64_t n_p = P.n_p;
  const int wid = threadIdx.x >> 5, part = wid % wps, per_cta = kFreeThreads / 32 / wps;
  for (int64_t s0 = (int64_t)blockIdx.x * per_cta; s0 * 32 < n_p; s0 += (int64_t)gridDim.x * per_cta) {
    const int64_t i = (s0 + wid / wps) * 32 + lane;
    const bool live = i < n_p;
    const St s = live ? (St)V.reps[i] : 0;  // no pair is anti-aligned past the end
    CT vi;
    vi.x = vi.y = 0;
    int li = 1;
    if (live) {
      vi = v[i];
      li = V.lid[i];
    }
    Real acc[partial_sums<Real>()][2];
#pragma unroll
    for (int a = 0; a < partial_sums<Real>(); ++a) acc[a][0] = acc[a][1] = 0;
    Real rest_r = 0, rest_i = 0;  // targets with a stabiliser, by norm_1 / norm_j
    uint64_t facs = 0;
    int cnt = 0;
    RowStart<kOrb> row;
    row.set(s, P, H);
    auto flush = [&]() {
      const int mx = (int)__reduce_max_sync(0xffffffffu, (unsigned)cnt);
      __syncwarp();
      for (int k = 0; k < mx; k += 4) {
        uint32_t e[4], act = 0;
        uint16_t h[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const bool has = k + q < cnt;
          e[q] = has ? qc[k + q][lane] : 0u;
          h[q] = has ? qi[k + q][lane] : (uint16_t)0;
          act |= has ? 1u << q : 0u;
        }
        take_slots<Real, 1, kSplit, 4, 4>(R, e, h, act, 0xFFFFFFFFu, false, pl, acc);
      }
      __syncwarp();
      cnt = 0;
    };
    for (int g = part; g < ng; g += wps) {
      const PassGroup& gr = H.groups[g];
      const St pm = (St)gr.mask, both = s & pm;
      const bool anti = both != 0 && both != pm;
      if (anti) {
        facs += gr.facadd;
        bool known;
        const Orbit o = target_orbit<kOrb, false>((St)(s ^ pm), gr, row, P, H, V.n_chunks, known);
        const int64_t j = kOrb >= kOrbPacked ? position_of(o.rep, V, P) : position(o, V, P);
        if (j >= 0) {
          const uint32_t id = value_id(s, gr, o.g, V, P);
          if (o.stab == 1) {
            qc[cnt][lane] = (uint32_t)j;
            qi[cnt][lane] = (uint16_t)id;
            ++cnt;
          } else {
            add_rest(tab[id], v[j], nrm_inv[o.stab] * nrm[1], rest_r, rest_i);
          }
        }
      }
      if (__any_sync(0xffffffffu, cnt == kQueue)) flush();
    }
    flush();
    Real sum[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      constexpr int kAcc = partial_sums<Real>();
#pragma unroll
      for (int a = 0; a < kAcc / 2; ++a) acc[a][j] += acc[a + kAcc / 2][j];
      sum[j] = kAcc == 2 ? acc[0][j] : acc[0][j] + acc[1 % kAcc][j];
    }
    sum[0] += rest_r;
    sum[1] += rest_i;
    if (wps > 1) {
      part_sum[wid][0][lane] = sum[0];
      part_sum[wid][1][lane] = sum[1];
      part_facs[wid][lane] = facs;
      __syncthreads();
      if (part == 0)
        for (int q = 1; q < wps; ++q) {
          sum[0] += part_sum[wid + q][0][lane];
          sum[1] += part_sum[wid + q][1][lane];
          facs += part_facs[wid + q][lane];
        }
      __syncthreads();
    }
    if (part == 0 && live) {
      const Real f = nrm[li] * nrm_inv[1];
      w[i] = row_out(sum[0], sum[1], f, (Real)row_ezz(s, facs, P, H), vi);
    }
  }
}

template <bool kTorus>
__global__ void __launch_bounds__(kHvThreads) k_count_offdiag(SectorView V, unsigned long long* __restrict__ nnz) {
  __shared__ SectorParams P;
  extern __shared__ __align__(16) uint8_t sm[];
  for (int i = threadIdx.x; i < (int)(sizeof(SectorParams) / 8); i += blockDim.x)
    reinterpret_cast<uint64_t*>(&P)[i] = reinterpret_cast<const uint64_t*>(V.params)[i];
  __syncthreads();
  const HvSmem<float> H = stage_hv<float, kTorus>(V, P, sm);
  __syncthreads();
  unsigned long long cnt = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < P.n_p; i += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t s = V.reps[i];
    for (int g = 0; g < P.n_groups; ++g) {
      const uint64_t m = H.groups[g].mask;
      if (popc64(s & m) != 1) continue;
      Orbit o;
      if (locate<float, kTorus>(s ^ m, V, P, H, o) >= 0) ++cnt;
    }
  }
  for (int o = 16; o > 0; o >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(nnz, cnt);
}

template <typename K>
int persistent_grid(K kernel, size_t smem, int64_t rows) {
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kHvThreads, smem);
  if (per_sm < 1) per_sm = 1;
  int64_t want = (rows + kHvThreads - 1) / kHvThreads;
  return (int)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)sms * per_sm));
}

template <typename Real, bool kTorus, bool kChCh>
cudaError_t launch_t(const Sector& S, const void* v, void* w, cudaStream_t st) {
  using CT = typename C2<Real>::T;
  const size_t smem = hv_smem_bytes<Real>(S.P.n_groups, S.P.n_ch, kTorus, S.V.row_bits, S.V.n_chunks, S.V.n_perm);
  auto kern = k_hv<Real, kTorus, kChCh>;
  const int grid = persistent_grid(kern, smem, S.P.n_p);
  kern<<<grid, kHvThreads, smem, st>>>(S.V, reinterpret_cast<const CT*>(v), reinterpret_cast<CT*>(w));
  return cudaGetLastError();
}

template <typename Real, int kOrb>
cudaError_t launch_free(const Sector& S, int orb, const void* v, void* w, cudaStream_t st) {
  using CT = typename CT2<Real>::T;
  const size_t at = align16(pass_smem_bytes(S.P, orb, S.V.row_bits, S.V.n_chunks, S.V.n_perm));
  const size_t smem = free_smem_bytes<Real>(S, orb);
  auto kern = k_hv_free<Real, kOrb>;
  // Up to 1.6e5 rows there are too few warps to hide the chain of searches: 822
  // rows took 37 us with a warp a slice and take 17 us, 9,250 rows 73 and 28 us,
  // 112,632 rows 109 and 88 us (FP32).
  const int wps = S.P.n_p < (int64_t)152 * 32 * 32 ? kFreeThreads / 32 : 1;
  // shared memory: at most the walk's tables (48 KB of permutations), 256 groups,
  // 1,024 chirality sites and 2,048 values
  const Resident r = resident((const void*)kern, kFreeThreads, smem, 128 * 1024);
  const int64_t want = (S.P.n_p * wps + kFreeThreads - 1) / kFreeThreads;
  // Up to 16 turns of the CTAs that fit at once: rows differ in their searches, and
  // one turn ends in a tail (FP32 at 28, 30 and 36 sites 831 -> 774 us, 3.74 ->
  // 3.16 ms, 270 -> 231 ms; FP64 at 36 sites 284 -> 262 ms).  A CTA keeps one and a
  // half sets of rows on average, for staging the tables is a cost of its own (one set
  // each: 24 sites 73 -> 78 us in FP32, 28 sites 1,037 -> 1,056 us in FP64).
  const int64_t once = (int64_t)r.sms * r.per_sm;
  const int64_t turns = std::max<int64_t>(1, std::min<int64_t>(16, 2 * want / (3 * once)));
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(want, once * turns));
  const CT* tab = reinterpret_cast<const CT*>(sizeof(Real) == 8 ? (const void*)S.vtab64 : (const void*)S.vtab32);
  kern<<<grid, kFreeThreads, smem, st>>>(S.V, tab, S.n_vals, (int)at, wps, reinterpret_cast<const CT*>(v),
                                         reinterpret_cast<CT*>(w));
  return cudaGetLastError();
}

template <typename Real>
cudaError_t launch_free_t(const Sector& S, const void* v, void* w, cudaStream_t st) {
  const int orb = orb_of(S.P);
  switch (orb) {
    case kOrbPacked: return launch_free<Real, kOrbPacked>(S, orb, v, w, st);
    case kOrbPacked32: return launch_free<Real, kOrbPacked32>(S, orb, v, w, st);
    case kOrbPacked64: return launch_free<Real, kOrbPacked64>(S, orb, v, w, st);
    case kOrbTorus: return launch_free<Real, kOrbTorus>(S, orb, v, w, st);
    default: return launch_free<Real, kOrbWalk>(S, orb, v, w, st);
  }
}

}  // namespace

cudaError_t launch_hv(const Sector& S, const void* v, void* w, bool fp64, cudaStream_t st) {
  if (S.col) return launch_hv_stored(S, v, w, fp64, st);
  return launch_hv_generic(S, v, w, fp64, st);
}

cudaError_t launch_hv_generic(const Sector& S, const void* v, void* w, bool fp64, cudaStream_t st) {
  const bool torus = S.P.torus != 0, chch = S.P.use_chch != 0;
  // the table beside the queues in shared memory: up to 2,048 FP64 values
  if (!chch && S.n_vals > 0 && S.n_vals <= 2048)
    return fp64 ? launch_free_t<double>(S, v, w, st) : launch_free_t<float>(S, v, w, st);
  if (fp64) {
    if (torus) return chch ? launch_t<double, true, true>(S, v, w, st) : launch_t<double, true, false>(S, v, w, st);
    return chch ? launch_t<double, false, true>(S, v, w, st) : launch_t<double, false, false>(S, v, w, st);
  }
  if (torus) return chch ? launch_t<float, true, true>(S, v, w, st) : launch_t<float, true, false>(S, v, w, st);
  return chch ? launch_t<float, false, true>(S, v, w, st) : launch_t<float, false, false>(S, v, w, st);
}

cudaError_t count_offdiag(const Sector& S, unsigned long long* nnz_dev, cudaStream_t st) {
  const bool torus = S.P.torus != 0;
  const size_t smem = hv_smem_bytes<float>(S.P.n_groups, S.P.n_ch, torus, S.V.row_bits, S.V.n_chunks, S.V.n_perm);
  cudaMemsetAsync(nnz_dev, 0, sizeof(unsigned long long), st);
  if (torus) {
    const int grid = persistent_grid(k_count_offdiag<true>, smem, S.P.n_p);
    k_count_offdiag<true><<<grid, kHvThreads, smem, st>>>(S.V, nnz_dev);
  } else {
    const int grid = persistent_grid(k_count_offdiag<false>, smem, S.P.n_p);
    k_count_offdiag<false><<<grid, kHvThreads, smem, st>>>(S.V, nnz_dev);
  }
  return cudaGetLastError();
}

}  // namespace edg
