// Device helpers shared by the Hamiltonian and PT2 kernels: connection-group targets and the
// FC term sums that give Hamiltonian elements.
#pragma once

#include "ops.h"

namespace vhci {

// Sum of a group's terms for ket key k: each term is fc * prod_j T[pw_j][q(mode_j)][dl_j], multiplied
// left to right and summed in table order (the reference's AnharmPot product and Vij sum order).
// Products and sums use explicit round-to-nearest operations so no multiply-add is contracted:
// the results are the same bits as the reference's separate multiplies and adds.
template <int W>
__device__ __forceinline__ double group_value(const ConnDev& cd, int tb, int te,
                                              const uint64_t (&k)[W], const KeyLayout& L) {
  const int qs = L.qmax + 1;
  double v = 0.0;
  for (int t = tb; t < te; ++t) {
    const TermDev tm = cd.terms[t];
    double tv = tm.fc;
    for (int j = 0; j < tm.nk; ++j) {
      const int q = key_q<W>(k, tm.mode[j], L.mpw, L.bits);
      tv = __dmul_rn(tv, __ldg(cd.T + ((int64_t)tm.pw[j] * qs + q) * 13 + tm.dl[j] + 6));
    }
    v = __dadd_rn(v, tv);
  }
  return v;
}

// Diagonal element: harmonic energy (Ham.cpp:211-220 operation order) plus the Delta = 0 terms
// in table order (quartic then sextic); equals the reference's fl(E_i + V_ii).
template <int W>
__device__ __forceinline__ double diag_value(const ConnDev& cd, const uint64_t (&k)[W],
                                             const KeyLayout& L) {
  double e = 0.0;
  for (int m = 0; m < cd.nm; ++m) {
    double ej = 0.5;
    ej = __dadd_rn(ej, (double)key_q<W>(k, m, L.mpw, L.bits));
    ej = __dmul_rn(ej, __ldg(cd.freq + m));
    e = __dadd_rn(e, ej);
  }
  const int qs = L.qmax + 1;
  double v = 0.0;
  for (int t = 0; t < cd.ndterms; ++t) {
    const TermDev tm = cd.dterms[t];
    double tv = tm.fc;
    for (int j = 0; j < tm.nk; ++j) {
      const int q = key_q<W>(k, tm.mode[j], L.mpw, L.bits);
      tv = __dmul_rn(tv, __ldg(cd.T + ((int64_t)tm.pw[j] * qs + q) * 13 + 6));
    }
    v = __dadd_rn(v, tv);
  }
  return __dadd_rn(e, v);
}

// Whether a state k can move by group g: every changed mode stays within [0, qmax] (a state outside
// cannot be in a basis stored with this layout).
template <int W>
__device__ __forceinline__ bool group_applies(const GroupDev& g, const uint64_t (&k)[W],
                                              const KeyLayout& L) {
  for (int c = 0; c < g.nchg; ++c) {
    const int q = key_q<W>(k, g.mode[c], L.mpw, L.bits) + g.delta[c];
    if (q < 0 || q > L.qmax) return false;
  }
  return true;
}

// ---- lowered-mode index: visit only the groups a state can move by --------------------------

// Binomial coefficients C(a, r) for a <= 32, r <= 6 at [a * kBinomR + r]; each block copies them to
// shared memory with fill_binom (followed by __syncthreads).
constexpr int kBinomA = 33, kBinomR = 7, kBinomElems = kBinomA * kBinomR;

struct BinomTable {
  uint32_t c[kBinomElems];
};
constexpr BinomTable make_binom() {
  BinomTable t{};
  for (int a = 0; a < kBinomA; ++a)
    for (int r = 0; r < kBinomR; ++r) {
      uint64_t v = 1;  // C(a, i) after step i; exact at every step
      for (int i = 0; i < r; ++i) v = v * (uint64_t)(a > i ? a - i : 0) / (uint64_t)(i + 1);
      t.c[a * kBinomR + r] = (uint32_t)v;
    }
  return t;
}
static __device__ const BinomTable d_binom = make_binom();

__device__ __forceinline__ void fill_binom(uint32_t* binom) {
  for (int t = threadIdx.x; t < kBinomElems; t += blockDim.x) binom[t] = d_binom.c[t];
}

// Segment of the groups lowering the mode set `key` (lowered_key layout): first group, count.
__device__ __forceinline__ void seg_find(const ConnDev& cd, uint64_t key, int& first, int& count) {
  uint32_t h = (uint32_t)mix64(key) & cd.lmask;
  for (uint32_t probe = 0; probe <= cd.lmask; ++probe) {  // load <= 1/2: ends at an empty slot
    const uint64_t k = __ldg(cd.lkey + h);
    if (k == key) {
      first = __ldg(cd.lseg + 2 * h);
      count = __ldg(cd.lseg + 2 * h + 1);
      return;
    }
    if (k == 0) return;
    h = (h + 1) & cd.lmask;
  }
}

// ---- the connection walk ---------------------------------------------------------------------

// Probes in flight per lane, and the ring of possible hits they feed (31 waiting + 32 kWalkIlp new).
constexpr int kWalkIlp = 2;
constexpr unsigned kWalkRing = 128;
constexpr int kWalkThreads = 128, kWalkWarps = kWalkThreads / 32;

struct WalkScratch {        // one per warp, in shared memory
  uint2 ring[kWalkRing];    // (index found, group)
  int2 seg[32];             // segments of a batch: end in the flattened list, group - position
  uint8_t exc[128];         // excited modes of the state
};

// Calls hit(j, u) for the states of `tab` that state k is connected to, in warp-uniform rounds: in
// every call each lane holds one connected state (its index j in the table, its group u) or j = -1;
// the states come in a fixed order (by lane within a call), so count and fill passes agree.
//
// A group lowering a mode that is not excited in k cannot apply, so with the lowered-mode index only
// the segments of the subsets of k's excited modes (sizes 0..maxl, r-major then colexicographic
// order) are visited; without it, or when the subsets outnumber half the groups, every group is.
// Most visits miss (3,600 groups a state for 350 connected ones on a 15-mode basis, 12,300 for 93 on
// a 48-mode one), so a visit is kept short: the hash of the target is the state's linear hash plus
// the group's constant, one 32-byte sector of slots is compared by fingerprint, and whatever matches
// goes into a ring.  The target key, the bounds of its quanta and the caller's work are done for 32
// ring entries at a time with every lane busy.  (The bounds come last because they rarely fail on a
// match: a target outside them wraps into other modes' fields and is almost never a basis key.)
// Bound by the L1 tag stage (one scattered sector a visit) and the L2 latency behind it.  Measured,
// count pass: 200,000 states of 48 modes 132 -> 13.3 ms (2.5e9 visits), 150,001 of 15 modes 18.3 ->
// 3.2 ms, against visits that checked the bounds first and probed one slot at a time; two probes in
// flight per lane beat four (13.3 : 15.7 ms, fewer registers), one 32-byte load beats a 16-byte one
// over two slots (14.8 ms) or two of them over four (19.2 ms, four in flight).
template <int W, class Hit>
__device__ __forceinline__ void walk_connections(const ConnDev& cd, const HashView& tab,
                                                 const uint64_t (&k)[W], const KeyLayout& L,
                                                 WalkScratch& ws, const uint32_t* binom, Hit&& hit) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const uint64_t hk = hash_lin<W>(k);
  unsigned head = 0, tail = 0;  // ring positions, the same in every lane

  // hands on ring entries, 32 at a time (`all`: the rest too)
  auto drain = [&](bool all) {
    __syncwarp();
    while (tail - head >= 32 || (all && tail != head)) {
      const unsigned have = min(32u, tail - head);
      int64_t j = -1;
      uint32_t u = 0;
      if (lane < have) {
        const uint2 r = ws.ring[(head + lane) % kWalkRing];
        u = r.y;
        uint64_t t[W];
#pragma unroll
        for (int w = 0; w < W; ++w) t[w] = k[w] + (uint64_t)__ldg(cd.wdelta + (int64_t)u * W + w);
        // another key of the same fingerprint (about one visit in 2^31): look the target up in full
        j = key_eq<W>(tab.keys, r.x, t) ? (int64_t)r.x : hash_find<W>(tab, t, key_hash<W>(t));
        if (j >= 0 && !group_applies<W>(cd.groups[u], k, L)) j = -1;
      }
      hit(j, u);
      head += have;
    }
    __syncwarp();
  };
  // visits the flattened list of the segments in ws.seg
  auto visit = [&](int total) {
    int at = 0;
    int2 sg = ws.seg[0];
    for (int f0 = 0; f0 < total; f0 += 32 * kWalkIlp) {
      uint32_t u[kWalkIlp];
      uint64_t h[kWalkIlp], s[kWalkIlp];
      ulonglong2 a[kWalkIlp], b[kWalkIlp];
#pragma unroll
      for (int t = 0; t < kWalkIlp; ++t) {
        const int f = f0 + 32 * t + lane;
        h[t] = 0;
        u[t] = kNoIndex;
        if (f < total) {
          while (f >= sg.x) sg = ws.seg[++at];
          u[t] = (uint32_t)(f + sg.y);
          h[t] = __ldg(cd.hdelta + u[t]);
        }
      }
#pragma unroll
      for (int t = 0; t < kWalkIlp; ++t) {
        h[t] = hash_final(hk + h[t]);
        s[t] = hash_home(h[t], tab.mask);
        if (u[t] != kNoIndex) load_slots(tab.slots + s[t], a[t], b[t]);
        else a[t] = b[t] = make_ulonglong2(kEmptySlot, kEmptySlot);
      }
#pragma unroll
      for (int t = 0; t < kWalkIlp; ++t) {
        const uint32_t fp = hash_fp(h[t]);
        SlotHit r = match_slots(a[t], b[t], fp);
        for (uint64_t it = 0; r.more && it <= tab.mask; it += 4) {
          s[t] = (s[t] + 4) & tab.mask;
          ulonglong2 c, d;
          load_slots(tab.slots + s[t], c, d);
          r = match_slots(c, d, fp);
        }
        const bool on = r.idx != kNoIndex;
        const unsigned m = __ballot_sync(full, on);
        if (on) ws.ring[(tail + __popc(m & lanemask_lt())) % kWalkRing] = make_uint2(r.idx, u[t]);
        tail += __popc(m);
      }
      if (tail - head >= 32) drain(false);
    }
  };

  int e = 0;
  int nsub = -1;
  __syncwarp();  // the previous state's readers of the scratch are done
  if (cd.maxl >= 0) {
    for (int m0 = 0; m0 < cd.nm; m0 += 32) {
      const int m = m0 + lane;
      const bool x = m < cd.nm && key_q<W>(k, m, L.mpw, L.bits) > 0;
      const unsigned b = __ballot_sync(full, x);
      if (x) ws.exc[e + __popc(b & lanemask_lt())] = (uint8_t)m;
      e += __popc(b);
    }
    __syncwarp();
    if (e < kBinomA) {
      int64_t ns = 0;
      for (int r = 0; r <= cd.maxl && r <= e; ++r) ns += binom[e * kBinomR + r];
      if (ns <= cd.ngroups / 2) nsub = (int)ns;
    }
  }
  if (nsub < 0) {
    if (lane == 0) ws.seg[0] = make_int2((int)cd.ngroups, 0);
    __syncwarp();
    visit((int)cd.ngroups);
  }
  for (int s0 = 0; s0 < nsub; s0 += 32) {
    const int s = s0 + lane;
    int first = 0, cnt = 0;
    if (s < nsub) {
      int r = 0;
      uint32_t rem = (uint32_t)s;
      while (rem >= binom[e * kBinomR + r]) rem -= binom[e * kBinomR + r++];
      uint64_t key = (uint64_t)(r + 1);
      int hi = e;  // element i = largest c < hi with C(c, i) <= rem (combinatorial number system)
      for (int i = r; i >= 1; --i) {
        int c = hi - 1;
        while (binom[c * kBinomR + i] > rem) --c;
        rem -= binom[c * kBinomR + i];
        key |= (uint64_t)(ws.exc[c] + 1) << (3 + 7 * (i - 1));
        hi = c;
      }
      seg_find(cd, key, first, cnt);
    }
    int incl = cnt;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(full, incl, d);
      if (lane >= d) incl += v;
    }
    const int total = __shfl_sync(full, incl, 31);
    const unsigned some = __ballot_sync(full, cnt > 0);
    if (cnt > 0) ws.seg[__popc(some & lanemask_lt())] = make_int2(incl, first - (incl - cnt));
    __syncwarp();
    visit(total);
    __syncwarp();
  }
  drain(true);
}

// ---- staged connections ----------------------------------------------------------------------
// The count pass can keep what it finds, so that the fill need not walk again: batches of up to 32
// (state index, group) pairs in any order, each with its row and the row's entries before it.
// Unused places of a batch hold kNoIndex.  A batch beyond the capacity is only counted.
// Called by the whole warp with the hits of one walk round (j < 0: none in this lane).
__device__ __forceinline__ void stage_hits(const StageView& st, uint32_t row, uint32_t off, int64_t j,
                                           uint32_t u) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned m = __ballot_sync(full, j >= 0);
  if (m == 0) return;
  unsigned long long b = 0;
  if (lane == 0) b = atomicAdd(st.cursor, 1ull);
  b = __shfl_sync(full, b, 0);
  if ((int64_t)b >= st.cap) return;
  if (lane == 0) st.batch[b] = make_uint2(row, off);
  const unsigned below = j >= 0 ? m : ~m;
  const int at = __popc(below & lanemask_lt()) + (j >= 0 ? 0 : __popc(m));
  st.pair[b * 32 + at] = make_uint2(j >= 0 ? (uint32_t)j : kNoIndex, u);
}

}  // namespace vhci
