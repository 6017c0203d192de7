// A thread's walk over its row's targets, shared by the build of the stored
// rows (targets.cu) and the matrix-free H*v (hv.cu): the flip groups staged in
// shared memory and the orbit search of a flipped state.
#pragma once
#include <cuda_runtime.h>

#include "hv_common.cuh"

namespace edg {
namespace {

constexpr int kMaxRowSlots = 256;  // a row has at most one target per flip group
constexpr int kMaxChPerGroup = 4;

// A flip group as the kernels stage it: what a row needs to find out
// whether the pair is anti-aligned, and where its sites sit on a packed torus.
struct PassGroup {
  uint64_t mask;
  uint64_t facadd;        // 1 << 16 * fid: counts the row's anti-aligned pairs by diagonal part
  double fac;
  uint16_t off;           // first value variant
  int8_t a, n_ch;
  int8_t sa, sb, ba, bb;  // packed torus: bit offset of each site's row in the state, of its byte
  int8_t top;             // packed torus: the pair touches the top row
  int8_t z[kMaxChPerGroup], pad[3];  // chirality sites
};

// Which orbit search the kernels use: the reference's walk, the row-rotation
// search, or the row-rotation search on packed rows (row length and row count
// up to 8) with 32-bit states and minima, 32-bit states, or 64-bit ones.
constexpr int kOrbWalk = 0, kOrbTorus = 1, kOrbPacked = 2, kOrbPacked32 = 3, kOrbPacked64 = 4;
template <int kOrb>
struct OrbRows {
  using T = PackedRows<uint64_t, uint64_t>;
};
template <>
struct OrbRows<kOrbPacked> {
  using T = PackedRows<uint32_t, uint32_t>;
};
template <>
struct OrbRows<kOrbPacked32> {
  using T = PackedRows<uint32_t, uint64_t>;
};
int orb_of(const SectorParams& P) {
  if (!P.torus) return kOrbWalk;
  if (P.L1 > 8 || P.L2 > 8) return kOrbTorus;
  return P.n_sites > 32 ? kOrbPacked64 : P.L2 <= 4 ? kOrbPacked : kOrbPacked32;
}

struct PassSmem {
  PassGroup* groups;
  const uint8_t* nk;
  const uint16_t* rots;
  const uint64_t *p1, *p2, *p3;
};

size_t pass_smem_bytes(const SectorParams& P, int orb, int row_bits, int n_chunks, int n_perm) {
  size_t b = align16(sizeof(PassGroup) * P.n_groups);
  if (orb == kOrbWalk) return b + (size_t)n_perm * n_chunks * 256 * sizeof(uint64_t);
  return b + align16((size_t)3 << row_bits);
}

template <int kOrb>
__device__ PassSmem stage_pass(const SectorView& V, const SectorParams& P, uint8_t* sm) {
  PassSmem H{};
  size_t off = 0;
  H.groups = reinterpret_cast<PassGroup*>(sm);
  off += align16(sizeof(PassGroup) * P.n_groups);
  for (int at = threadIdx.x; at < P.n_groups; at += blockDim.x) {
    const int g = V.order[at];
    const TermGroup src = V.groups[g];
    PassGroup d{};
    d.mask = src.mask;
    d.facadd = P.n_facs <= kMaxFacs ? 1ull << (16 * src.fid) : 0;
    d.fac = src.fac;
    d.off = V.voff[g];
    d.a = (int8_t)src.a;
    d.n_ch = (int8_t)(src.ch_end - src.ch_begin);
    for (int m = src.ch_begin, b = 0; m < src.ch_end && b < kMaxChPerGroup; ++m, ++b) d.z[b] = (int8_t)V.ch[m].z;
    if (kOrb >= kOrbPacked) {
      const int ya = src.a / P.L1, yb = src.b / P.L1;
      d.sa = (int8_t)(P.L1 * ya);
      d.sb = (int8_t)(P.L1 * yb);
      d.ba = (int8_t)(8 * ya);
      d.bb = (int8_t)(8 * yb);
      d.top = ya == P.L2 - 1 || yb == P.L2 - 1;
    }
    H.groups[at] = d;
  }
  if (kOrb == kOrbWalk) {
    const int n = V.n_perm * V.n_chunks * 256;
    uint64_t* p = reinterpret_cast<uint64_t*>(sm + off);
    for (int i = threadIdx.x; i < n; i += blockDim.x) p[i] = V.perms[i];
    H.p1 = p;
    H.p2 = p + V.n_chunks * 256;
    H.p3 = p + 2 * V.n_chunks * 256;
  } else {
    const int n = 1 << V.row_bits;
    uint16_t* rots = reinterpret_cast<uint16_t*>(sm + off);
    uint8_t* nk = sm + off + 2 * n;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      rots[i] = V.rots[i];
      nk[i] = V.nk[i];
    }
    H.rots = rots;
    H.nk = nk;
  }
  return H;
}

// What a row's searches start from.  On a packed torus: s is a representative,
// so its top row is at its rotation minimum and no row has a smaller one; when
// it is the only row that reaches it and is aperiodic (uniq), a flip that leaves
// it alone and gives no other row a minimum <= mstar is its own representative
// with stabiliser 1.
template <int kOrb>
struct RowStart {
  using R = typename OrbRows<kOrb>::T;
  typename R::Bytes kb, valid;
  int mstar;
  bool uniq;
  __device__ __forceinline__ void set(typename R::State s, const SectorParams& P, const PassSmem& H) {
    kb = 0;
    valid = 0;
    mstar = 0;
    uniq = false;
    if (kOrb >= kOrbPacked) {
      valid = R::valid(P);
      kb = R::pack(s, P, H.nk);
      typename R::Bytes hit;
      mstar = R::min_rows(kb, valid, hit);
      const typename R::State rmask = ((typename R::State)1 << P.L1) - 1;
      uniq = R::single(hit) && H.rots[(int)((s >> (P.L1 * (P.L2 - 1))) & rmask)] == 1u;
    }
  }
};

// The orbit of t = s with group gr flipped.  kCount: only whether t has an
// allowed representative is wanted; known is set (and the orbit left out) when
// it is alone in its search -- one candidate translate, so a trivial stabiliser,
// which is allowed at every momentum.
template <int kOrb, bool kCount>
__device__ __forceinline__ Orbit target_orbit(typename OrbRows<kOrb>::T::State t, const PassGroup& gr,
                                              const RowStart<kOrb>& row, const SectorParams& P, const PassSmem& H,
                                              int n_chunks, bool& known) {
  using R = typename OrbRows<kOrb>::T;
  known = false;
  if (kOrb >= kOrbPacked) {
    const typename R::State rmask = ((typename R::State)1 << P.L1) - 1;
    const int na = H.nk[(int)((t >> gr.sa) & rmask)], nb = H.nk[(int)((t >> gr.sb) & rmask)];
    if (row.uniq && !gr.top && na > row.mstar && nb > row.mstar) {
      known = true;
      return Orbit{(uint64_t)t, 0, 1};
    }
    typename R::Bytes hit;
    R::min_rows(R::set(R::set(row.kb, gr.ba, na), gr.bb, nb), row.valid, hit);
    if (kCount && R::single(hit)) {
      const uint32_t rs = H.rots[(int)((t >> (P.L1 * R::row_of(hit))) & rmask)];
      known = (rs & (rs - 1)) == 0;
      if (known) return Orbit{0, 0, 1};
    }
    return R::search(t, hit, P, H.rots);
  }
  if (kOrb == kOrbTorus) return orbit_torus(t, P, H.nk, H.rots);
  return orbit_walk(t, P, H.p1, H.p2, H.p3, n_chunks);
}

// Targets with a stabiliser, on a packed torus.  Such a target is left alone by
// one of the translations of prime order (at most 8 up to those that generate
// the same subgroup; 8x4 has 3).  For a translation T and the pair's mask m,
// T(s ^ m) = s ^ m just when s ^ T s = m ^ T m, a word of at most 4 bits: a row
// whose s ^ T s has more bits than that under every T (all but 1 in 150 at 8x4)
// has no such target, and all its targets are allowed, at every momentum.
struct PrimeShifts {
  int n;
  int8_t x[8], y[8];
};

PrimeShifts prime_shifts(const SectorParams& P) {
  PrimeShifts R{};
  for (int y = 0; y < P.L2; ++y)
    for (int x = 0; x < P.L1; ++x) {
      int order = 1;
      while (order * x % P.L1 || order * y % P.L2) ++order;
      bool first = order > 1;  // of prime order, and the first of its subgroup
      for (int q = 2; q < order; ++q)
        first = first && order % q && (q * y % P.L2) * P.L1 + q * x % P.L1 > y * P.L1 + x;
      if (!first || R.n == 8) continue;
      R.x[R.n] = (int8_t)x;
      R.y[R.n++] = (int8_t)y;
    }
  return R;
}

template <typename St>
__device__ __forceinline__ St shifted(St t, const PrimeShifts& G, int g, const SectorParams& P) {
  const uint64_t u = torus_rotate_rows((uint64_t)t, P.L1 * G.y[g], P.n_sites, P.full_mask);
  return (St)torus_rotate_within(u, G.x[g], P.L1, P);
}

// m ^ T m of every translation and group (moved[g * n_groups + group])
template <typename St>
__device__ __forceinline__ void stage_moved(const PrimeShifts& G, const SectorParams& P, const PassSmem& H, St* moved) {
  for (int k = threadIdx.x; k < P.n_groups * G.n; k += blockDim.x) {
    const St m = (St)H.groups[k % P.n_groups].mask;
    moved[k] = m ^ shifted(m, G, k / P.n_groups, P);
  }
}

// the translations that may leave a target of s alone, as bits
template <typename St>
__device__ __forceinline__ uint32_t risky_shifts(St s, const PrimeShifts& G, const SectorParams& P) {
  uint32_t risk = 0;
  for (int g = 0; g < G.n; ++g) risk |= popc64(s ^ shifted(s, G, g, P)) <= 4 ? 1u << g : 0u;
  return risk;
}

// has the target of an anti-aligned group a stabiliser?
template <typename St>
__device__ __noinline__ bool symmetric_target(St s, int at, uint32_t risk, const PrimeShifts& G, const SectorParams& P,
                                              const St* moved) {
  for (; risk; risk &= risk - 1) {
    const int g = __ffs((int)risk) - 1;
    if (moved[g * P.n_groups + at] == (s ^ shifted(s, G, g, P))) return true;
  }
  return false;
}

// The value id of a target: bit a of the state and the bits z of the group's
// chirality terms, and the phase class of the translation (value_tables).
template <typename St>
__device__ __forceinline__ uint32_t value_id(St s, const PassGroup& gr, int g, const SectorView& V,
                                             const SectorParams& P) {
  int variant = (int)((s >> gr.a) & 1u);
  const int n = gr.n_ch;
  if (n == 2) {  // an inner bond of a torus of triangles: no loop
    variant |= (int)((s >> gr.z[0]) & 1u) << 1 | (int)((s >> gr.z[1]) & 1u) << 2;
  } else {
    for (int b = 0; b < n; ++b) variant |= (int)((s >> gr.z[b]) & 1u) << (b + 1);
  }
  return __ldg(V.remap + (gr.off + variant) * P.n_cls + P.g2cls[g]);
}

// Ezz of a row from its counted diagonal parts or, with more couplings than
// there are counters, summed in a loop of its own: an FP64 instruction in the
// walk would take its 16 clocks for every group, predicated off or not.
template <typename St>
__device__ __noinline__ double row_ezz(St s, uint64_t facs, const SectorParams& P, const PassSmem& H) {
  double fac = 0.0;
  if (P.n_facs <= kMaxFacs) {
    for (int k = 0; k < P.n_facs; ++k) fac += P.facs[k] * (double)((facs >> (16 * k)) & 0xFFFFu);
  } else {
    for (int g = 0; g < P.n_groups; ++g) {
      const St pm = (St)H.groups[g].mask, both = s & pm;
      if (both != 0 && both != pm) fac += H.groups[g].fac;
    }
  }
  return P.total_fac - 2.0 * fac;  // sum_bonds lJ/4 - 2 sum_anti lJ/4
}

}  // namespace
}  // namespace edg
